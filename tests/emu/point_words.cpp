// The last point of a context's buffers is deleted, for capacities of every
// remainder to a word; built with -fsanitize=address, which ends the program
// where a byte outside an allocation is touched.
#include "../../gpu_cdt_refine_b200/csrc/refine.cu"

int main() {
  for (long n = 5; n < 13; ++n) {
    gqm::Refiner r;
    if (r.setup(0) != GQM_OK || r.alloc_points(n) != GQM_OK || r.alloc_points(n + 9) != GQM_OK) return 2;
    const long last = n + 8;
    r.M.ps[last] = 0;
    gqm::delete_point(r.M, (int)last);
    if (r.M.ps[last] != gqm::PS_DELETED || r.M.ps[last - 1] != gqm::PS_DELETED) return 3;
  }
  return 0;
}
