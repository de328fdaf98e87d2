// Checks of the sharing rule (csrc/sm_share.h); prints the first that fails.
#include <cstdio>
#include <thread>
#include <vector>

#include "../../gpu_cdt_refine_b200/csrc/sm_share.h"

using gqm_share::Ticket;
#define CHECK(x)                                 \
  do {                                           \
    if (!(x)) {                                  \
      printf("line %d: %s\n", __LINE__, #x);     \
      return 1;                                  \
    }                                            \
  } while (0)

int main() {
  {  // alone: what it asks for, again and again, and after others have ended
    Ticket a;
    a.open(0, 1000, 1.0);
    CHECK(a.take(148, 148) == 148 && a.take(148, 148) == 148 && a.take(16, 148) == 16);
    {
      Ticket b, other;
      b.open(0, 1000, 1.0);
      other.open(1, 5, 1.0);  // another device's calls do not count
      CHECK(b.take(148, 148) == 132);  // beside 16 held
      CHECK(a.take(148, 148) == 74);   // its half, although b holds more
      CHECK(b.take(148, 148) == 74);
      CHECK(other.take(148, 148) == 148);
    }
    CHECK(a.take(148, 148) == 148);
  }
  {  // registered together: parts by size, which fit together whoever starts first
    for (int first = 0; first < 3; ++first) {
      Ticket t[3];
      const double size[3] = {800000, 40000, 10000};
      for (int k = 0; k < 3; ++k) t[k].open(0, size[k], 1.0);
      int sum = 0, n[3];
      for (int k = 0; k < 3; ++k) sum += n[(first + k) % 3] = t[(first + k) % 3].take(148, 148);
      CHECK(sum <= 148 && n[0] >= 139 && n[1] >= 6 && n[2] >= 1);
      t[0].close();
      CHECK(t[1].take(148, 148) >= 118);  // four fifths
    }
  }
  {  // never none, and a launch that has ended leaves its blocks
    std::vector<Ticket> t(500);
    for (Ticket &x : t) x.open(2, 7, 1.0);
    for (Ticket &x : t) CHECK(x.take(148, 148) == 1);
    for (Ticket &x : t) x.give();
    Ticket late;
    late.open(2, 1e9, 1.0);
    CHECK(late.take(148, 148) == 147);
  }
  {  // half as busy, half as much kept for it
    Ticket a, b;
    a.open(0, 100, 0.5);
    b.open(0, 100, 0.5);
    CHECK(a.take(148, 148) == 111 && b.take(148, 148) == 74);
  }
  {  // threads: nothing is left behind
    std::vector<std::thread> pool;
    for (int k = 0; k < 8; ++k)
      pool.emplace_back([k] {
        for (int i = 0; i < 20000; ++i) {
          Ticket t;
          t.open(3, 1.0 + k * 0.1, 1.0);
          t.take(148, 148);
          if (i & 1) t.give();
        }
      });
    for (auto &t : pool) t.join();
    CHECK(gqm_share::g_devices[3].blocks == 0 && gqm_share::g_devices[3].calls == 0);
    CHECK(gqm_share::g_devices[3].size == 0.0 && gqm_share::g_devices[3].waiting == 0.0);
  }
  puts("ok");
  return 0;
}
