// Batched refinement of many independent domains in one persistent launch, and
// the refinement of one domain in one launch.
//
// Each team of thread blocks is a complete refiner for one domain at a time
// (engine.cuh).  Teams take domains from a queue ordered largest first (one
// atomic counter), so the whole batch, including every domain's round loop and
// flip-flop loop, is decided on the device: no host round trip and no launch
// per step.
//
// A domain's result is the one the single-domain path returns for it: the
// same steps run in the same order on the same slot discipline.  Each team
// owns one scratch arena sized for the largest domain of the batch; a domain
// whose mesh would outgrow its arena stops with GQM_ERR_ARENA and is refined
// again by the single-domain path on the host side of the call.
#define GQM_CTA_MODE 1
#define gqm gqm_cta
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <queue>
#include <thread>
#include <vector>

#include "host_copy.h"

#include "../../include/gqm_refine.h"
#include "engine.cuh"

namespace gqm {

// ---------------------------------------------------------------------------
// One domain of a batch, in device memory.  The host fills the inputs, the
// options and the output pointers; the block that refines the domain fills
// the results.
// ---------------------------------------------------------------------------
struct Job {
  const double2 *pts;
  const int *tri, *nbr;
  const int2 *seg;
  int np, nt, ns;
  int offcenter, offconstant, mode, pred, placement;
  MlpDev mlp;  // GQM_PLACE_LEARNED: the network on the device
  double theta, max_area;
  long long max_rounds;
  // outputs: each finished domain takes its space from one shared region
  // (bump allocation), so the region holds exactly the batch's results
  char *obase;
  unsigned long long *oused;
  unsigned long long ocap;
  unsigned long long ooff;  // offset of this domain's output block
  // results
  int status, out_np, out_nt, out_ns, rounds;
  long long flip_steps, steiner, midpoints, bad_total, exact_fallbacks, learned_candidates, learned_used;
  double goodcos2;
};

// Arena sizes of one domain: room for four more point blocks and five more
// triangle blocks of growth, and for eight subsegments per input segment plus
// one per two input points.
__host__ __device__ inline Caps caps_of(int np, int nt, int ns) {
  Caps c;
  c.pointblock = (int)(np * 0.5);
  c.triblock = 2 * c.pointblock;
#ifdef GQM_TEST_TIGHT_BUFFERS
  // test builds: arenas with no room to grow, so that domains overflow and
  // take the single-domain path
  c.pphys = np + c.pointblock;
  c.tphys = nt + c.triblock;
#else
  c.pphys = np + 5 * c.pointblock;
  c.tphys = nt + 6 * c.triblock;
#endif
  c.sphys = 8L * ns + np / 2 + 1024;
  c.cav_cap = c.tphys / 4 + 64;
  c.hsz = 1;
  while (c.hsz < 2L * ns + 16) c.hsz <<= 1;
  return c;
}

// Walks the arena layout: with base == 0 it only measures (host), otherwise it
// assigns every pointer of S (device).  Every array starts on 256 bytes.
struct Cursor {
  char *base;
  size_t off;
  template <class T>
  __host__ __device__ T *take(long n) {
    off = (off + 255) & ~(size_t)255;
    T *p = reinterpret_cast<T *>(reinterpret_cast<uintptr_t>(base) + off);
    off += sizeof(T) * (size_t)(n > 0 ? n : 1);
    return p;
  }
};
__host__ __device__ inline void carve(Cursor &a, Scratch &S, const Caps &c) {
  const long P = c.pphys, T = c.tphys, Sg = c.sphys;
  Mesh &M = S.M;
  M.pts = a.take<double2>(P);
  M.ps = a.take<uint8_t>(P);
  M.pred = a.take<uint8_t>(P);
  S.emptyp = a.take<int>(P);
  S.pnew = a.take<int>(P);
  S.tail = a.take<int>(P > T ? P : T);
  M.tv = a.take<int4>(T);
  M.tn = a.take<int4>(T);
  M.tsg = a.take<int4>(T);
  M.tst = a.take<uint8_t>(T);
  M.tflip = a.take<uint8_t>(T);
  M.tfo = a.take<uint8_t>(T);
  M.tmark = a.take<int>(T);
  M.fstamp = a.take<int>(T);
  S.emptyt = a.take<int>(T);
  S.bad = a.take<int>(T);
  S.imark = a.take<int>(T);
  S.ilist = a.take<int>(T);
  S.sinks = a.take<int>(T);
  S.wl = a.take<int>(T);
  S.newidx = a.take<int>(T);
  M.fmark = a.take<unsigned long long>(T);
  M.emap = a.take<int4>(T);
  S.fl.q0 = a.take<int>(T);
  S.fl.q1 = a.take<int>(T);
  S.fl.rec = a.take<int4>(T);
  S.fl.red = a.take<int>(2 * T);
  S.fl.late = a.take<int4>(2 * Sg);
  winner_carve(S.fl, a.take<unsigned>((long)winner_words(T)), T);
  S.center = a.take<double2>(T);
  M.s2t = a.take<s2t_t>(Sg);
  M.s2seg = a.take<int>(Sg);
  M.enc = a.take<int>(Sg);
  S.enclist = a.take<int>(Sg);
  S.encl2 = a.take<int>(Sg);
  S.smark = a.take<int>(Sg);
  S.mids = a.take<int>(Sg);
  S.snap = a.take<int>(Sg);
  S.cav = a.take<int>((long)kCavityCap * c.cav_cap);
  S.cavn = a.take<int>(c.cav_cap);
  S.hkeys = a.take<unsigned long long>(c.hsz);
  S.hvals = a.take<int>(c.hsz);
  S.s2ti = a.take<int>(c.hsz);
}
// Output block of one finished domain: points, triangles, neighbours,
// segments, point and triangle status bytes, each on 16 bytes.
struct OutLayout {
  unsigned long long pts, tri, nbr, seg, ps, ts, bytes;
};
__host__ __device__ inline unsigned long long up16(unsigned long long x) { return (x + 15) & ~15ull; }
__host__ __device__ inline OutLayout out_layout(long np, long nt, long ns) {
  OutLayout L;
  L.pts = 0;
  L.tri = L.pts + up16(16ull * np);
  L.nbr = L.tri + up16(12ull * nt);
  L.seg = L.nbr + up16(12ull * nt);
  L.ps = L.seg + up16(8ull * ns);
  L.ts = L.ps + up16((unsigned long long)np);
  L.bytes = L.ts + up16((unsigned long long)nt);
  return L;
}
inline size_t arena_bytes(const Caps &c) {
  Cursor a{nullptr, 0};
  Scratch S;
  carve(a, S, c);
  return (a.off + 255) & ~(size_t)255;
}

// One domain of a batch: the refinement, then its output block.
template <int PRED>
__device__ int run_job(Engine<PRED> &R, Job &J) {
  BlockState &sh = R.sh;
  TeamState &ts = R.ts;
  GridTeam &T = R.T;
  Scratch &S = sh.S;
  R.c = caps_of(J.np, J.nt, J.ns);
  if (threadIdx.x == 0) {
    S.M.segs = J.seg;
    S.M.err = &ts.err;
    S.fl.c = &ts.fc;
  }
  if (R.lead()) {
    ts.err = 0;
    for (int i = 0; i < 6; ++i) ts.ctr[i] = 0;
    ts.fc.gen = 0;
    ts.fc.epoch = 0;
    ctl_reset(&ts.fc, 64 * J.max_rounds, &ts.err, true);
  }
  // stamps and claims start afresh for every domain
  __syncthreads();
  R.fill(S.M.fstamp, R.c.tphys, 0);
  R.fill(S.M.fmark, R.c.tphys, ~0ull);
  R.fill(S.M.emap, R.c.tphys, make_int4(0, 0, 0, 0));
  TSYNC();
  double gc = 0.0;
  int rc = R.refine(J, J.theta, &gc);
  if (R.lead()) J.goodcos2 = gc;
  int out_np = 0, out_nt = 0;
  if (rc == GQM_OK) rc = R.compact_output(&out_np, &out_nt);
  if (rc == GQM_ERR_TOPOLOGY) return rc;
  if (const int e = R.read_err()) rc = rc ? rc : e;
  if (rc == GQM_OK) {
    const OutLayout L = out_layout(out_np, out_nt, R.last_subseg);
    if (R.lead()) {
      const unsigned long long off = atomicAdd(J.oused, (unsigned long long)L.bytes);
      ts.part[0][0] = off + L.bytes <= J.ocap ? 0 : GQM_ERR_ARENA;
      J.ooff = off;
    }
    TSYNC();
    rc = vload(&ts.part[0][0]);
    if (rc == GQM_OK) {
      char *o = J.obase + *(volatile unsigned long long *)&J.ooff;
      k_emit_output(S.M, out_nt, R.last_subseg, reinterpret_cast<int *>(o + L.tri), reinterpret_cast<int *>(o + L.nbr),
                    reinterpret_cast<int *>(o + L.seg), reinterpret_cast<uint8_t *>(o + L.ts), &ts.fc);
      k_emit_pstatus(S.M, out_np, reinterpret_cast<uint8_t *>(o + L.ps));
      double2 *op = reinterpret_cast<double2 *>(o + L.pts);
      for (int i = T.tid(); i < out_np; i += T.size()) op[i] = S.M.pts[i];
    }
    TSYNC();
  }
  if (R.lead()) {
    J.out_np = out_np;
    J.out_nt = out_nt;
    J.out_ns = R.last_subseg;
    J.rounds = R.rounds;
    J.bad_total = R.bad_total;
    J.flip_steps = ts.fc.steps;
    J.steiner = (long long)ts.ctr[0];
    J.midpoints = (long long)ts.ctr[1];
    J.exact_fallbacks = (long long)ts.ctr[2];
    J.learned_candidates = (long long)ts.ctr[4];
    J.learned_used = (long long)ts.ctr[5];
  }
  return rc;
}

// The persistent batch kernel: teams of nb consecutive blocks, each taking the
// next domain (largest first) until the queue is empty, refining it in its own
// arena.  A team of one block keeps its state in shared memory.
template <int PRED>
__device__ __forceinline__ void batch_body(Job *jobs, const int *order, int njobs, int *next, char *arenas,
                                           size_t arena_stride, TeamState *teams, int nb, BlockState &sh,
                                           TeamState &own) {
  const int team = (int)blockIdx.x / nb;
  TeamState &ts = nb == 1 ? own : teams[team];
  if (threadIdx.x == 0) {
    gqm_team_rank = (int)blockIdx.x % nb;
    gqm_team_blocks = nb;
  }
  __syncthreads();
  char *arena = arenas + (size_t)team * arena_stride;
  Engine<PRED> R{sh, ts, GridTeam{&ts.bar, nb, gqm_team_rank, 0ull, &ts.err}, nullptr, nullptr,
                 kTeamSmallLimit};
  for (;;) {
    if (R.lead()) ts.job = atomicAdd(next, 1);
    if (!R.T.sync()) return;
    const int k = vload(&ts.job);
    if (!R.T.sync()) return;
    if (k >= njobs) break;
    Job &J = jobs[order[k]];
    if (threadIdx.x == 0) {
      Cursor a{arena, 0};
      carve(a, sh.S, caps_of(J.np, J.nt, J.ns));
    }
    __syncthreads();
    const int rc = run_job(R, J);
    if (R.lead()) J.status = rc;
    if (!R.T.sync()) return;
  }
}
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_batch(Job *jobs, const int *order, int njobs, int *next, char *arenas, size_t arena_stride, TeamState *teams,
            int nb, int pred) {
  __shared__ BlockState sh;
  __shared__ TeamState own;
  if (pred)
    batch_body<1>(jobs, order, njobs, next, arenas, arena_stride, teams, nb, sh, own);
  else
    batch_body<0>(jobs, order, njobs, next, arenas, arena_stride, teams, nb, sh, own);
}

// One domain in the single-domain engine's buffers, by the whole grid.
template <int PRED>
__global__ void __launch_bounds__(512, 1)
    k_refine_one(Scratch S, Caps c, EngineRun *run, TeamState *ts, int small_limit, KTimer *ktm, KTimer *stm) {
  __shared__ BlockState sh;
  const int nb = (int)gridDim.x;
  if (threadIdx.x == 0) {
    gqm_team_rank = (int)blockIdx.x;
    gqm_team_blocks = nb;
    sh.S = S;
    sh.S.M.segs = run->seg;
    sh.S.M.err = &ts->err;
  }
  __syncthreads();
  Engine<PRED> R{sh, *ts, GridTeam{&ts->bar, nb, (int)blockIdx.x, 0ull, &ts->err}, ktm, stm, small_limit, c};
  double gc = 0.0;
  int out_np = 0, out_nt = 0;
  int rc = R.refine(*run, run->theta, &gc);
  if (rc == GQM_OK) rc = R.compact_output(&out_np, &out_nt);
  if (rc != GQM_ERR_TOPOLOGY)
    if (const int e = R.read_err()) rc = rc ? rc : e;
  if (R.lead()) {
    run->status = rc;
    run->need_grow = R.need_grow;
    run->out_np = out_np;
    run->out_nt = out_nt;
    run->out_ns = R.last_subseg;
    run->rounds = R.rounds;
    run->bad_total = R.bad_total;
    run->last_point = R.last_point;
    run->last_triangle = R.last_triangle;
    run->goodcos2 = gc;
    for (int i = 0; i < 6; ++i) run->ctr[i] = ts->ctr[i];
  }
}

}  // namespace gqm

// ===========================================================================
// Host side
// ===========================================================================
namespace gqm {
namespace {

typedef void (*BatchFn)(Job *, const int *, int, int *, char *, size_t, TeamState *, int, int);
struct Variant {
  int threads, minb;
  BatchFn fn;
};
// compiled (threads per block, blocks per SM) pairs; the autotuner picks one
const Variant kVariants[] = {{128, 4, k_batch<128, 4>}, {256, 1, k_batch<256, 1>}, {256, 2, k_batch<256, 2>},
                             {512, 1, k_batch<512, 1>}};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
// one 512-thread block per SM: the fastest on every batch measured (256
// domains 101 ms against 152, 181 and 355 ms for 256x1, 256x2 and 128x4, 700
// domains 117 ms against 171, 204 and 393 ms), and the one that forms teams
constexpr int kTeamVariant = 3;
constexpr int kDefaultVariant = kTeamVariant;

// Buffers kept per device between calls (grow only).
struct DevCache {
  std::mutex mu;
  bool init = false;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  char *d_in = nullptr, *d_out = nullptr, *d_arena = nullptr, *h_in = nullptr, *h_out = nullptr;
  char *d_teams = nullptr;
  size_t in_cap = 0, out_cap = 0, arena_cap = 0, h_in_cap = 0, h_out_cap = 0, teams_cap = 0;
  Job *d_jobs = nullptr;
  int *d_order = nullptr;
  int jobs_cap = 0;
  int *d_next = nullptr;
  unsigned long long *d_used = nullptr;
  int tuned = -1;  // autotuned variant, -1 until gqm_batch_autotune ran
  int sms = 148;
};
DevCache g_dev[16];

template <class T>
int grow_dev(T **p, size_t *cap, size_t need) {
  if (need <= *cap) return GQM_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  if (cudaMalloc((void **)p, need) != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return GQM_ERR_MEMORY;
  }
  *cap = need;
  return GQM_OK;
}
int grow_host(char **p, size_t *cap, size_t need) {
  if (need <= *cap) return GQM_OK;
  if (*p) cudaFreeHost(*p);
  *p = nullptr;
  *cap = 0;
  if (cudaMallocHost((void **)p, need) != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return GQM_ERR_MEMORY;
  }
  *cap = need;
  return GQM_OK;
}
size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

// f(k) for k in [0, n) on the host's cores (packing and unpacking of the
// domains' arrays are independent memcpy's)
template <class F>
void parallel_for(int n, F f) {
  int nt = (int)std::thread::hardware_concurrency();
  nt = std::max(1, std::min(nt, 32));
  if (n < 64 || nt == 1) {
    for (int k = 0; k < n; ++k) f(k);
    return;
  }
  std::vector<std::thread> pool;
  for (int t = 0; t < nt; ++t)
    pool.emplace_back([&, t] {
      for (int k = t; k < n; k += nt) f(k);
    });
  for (auto &th : pool) th.join();
}

int check_domain(const gqm_cdt_in *in, const gqm_options *opt) {
  if (!in || !opt) return GQM_ERR_ARGUMENT;
  if (in->numberofpoints < 3 || in->numberoftriangles < 1 || in->numberofsegments < 0) return GQM_ERR_ARGUMENT;
  if (!in->pointlist || !in->trianglelist || !in->neighborlist) return GQM_ERR_ARGUMENT;
  if (in->numberofsegments > 0 && !in->segmentlist) return GQM_ERR_ARGUMENT;
  if (!(opt->theta > 0.0 && opt->theta < 60.0)) return GQM_ERR_ARGUMENT;
  if (opt->placement != GQM_PLACE_PLAIN && (opt->placement != GQM_PLACE_LEARNED || !opt->mlp)) return GQM_ERR_ARGUMENT;
  if (!(opt->max_area >= 0.0)) return GQM_ERR_ARGUMENT;
  return GQM_OK;
}

double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// Blocks per team for a batch on `resident` blocks.  A team of one block keeps
// every block busy in a large batch, but a block works on its last, or largest,
// domain alone.  A domain of n points takes a team of nb blocks about
// L + P / nb: L = 1.35 log2(n) - 8.8 ms for the chain of its steps (at least
// 1 ms), whatever the team, and P = 0.75 ms per 1,000 points for the work in
// them (measured on an idle GPU: 49,497 points take 48.6, 32.7, 22.1, 16.8, 14.3
// and 13.1 ms with 1, 2, 4, 8, 16 and 32 blocks).  The team size is the one whose
// queue, largest domain first, ends soonest by that.  With all SMs busy the times
// are 1.6 to 2 times the rule's: it stands for the order of the team sizes, not
// for the time of a batch (256 domains of 200 to 50,000 points: 49 and 37 ms by
// the rule with one and two blocks, 100.2 and 65.6 ms measured).  Measured with
// one block per team and with the rule's choice: 16 domains 53.5 and 16.7 ms, 64
// domains 79.8 and 33.5 ms, 256 domains 100.2 and 65.6 ms; 700 domains 115.8 ms
// with one block, the rule's choice, and 144.3 ms with two.
constexpr int kTeamSizes[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48};
int blocks_per_team(const gqm_cdt_in *in, const std::vector<int> &ids, long resident) {
  std::vector<double> n;
  for (int d : ids) n.push_back((double)in[d].numberofpoints);
  std::sort(n.begin(), n.end(), std::greater<double>());
  int nb = 1;
  double best = 0.0;
  for (int k : kTeamSizes) {
    const size_t teams = std::min((size_t)(resident / k), n.size());
    if (teams < 1) break;
    std::priority_queue<double, std::vector<double>, std::greater<double>> ends;
    double last = 0.0;
    for (double x : n) {
      double at = 0.0;
      if (ends.size() == teams) {
        at = ends.top();
        ends.pop();
      }
      at += std::max(1.0, 1.35 * std::log2(x) - 8.8) + 0.75e-3 * x / k;
      ends.push(at);
      last = std::max(last, at);
    }
    if (k == 1 || last < best) {
      best = last;
      nb = k;
    }
  }
  return nb;
}

// One persistent batch over the domains `ids` (all with the same predicate
// mode) with kernel variant `var`.  Results of domains that finished land in
// out/stats; the status of each domain in status[d].
int run_batch(DevCache &C, const std::vector<int> &ids, const gqm_cdt_in *in, gqm_cdt_out *out,
              const gqm_options *opt, gqm_stats *stats, int var, double mem_fraction, int *status,
              gqm_batch_report *rep, bool keep_outputs) {
  const int n = (int)ids.size();
  if (n == 0) return GQM_OK;
  auto t0 = std::chrono::steady_clock::now();
  // sizes
  std::vector<size_t> in_off(n);
  size_t in_bytes = 0, arena = 0;
  unsigned long long out_bound = 0;
  for (int k = 0; k < n; ++k) {
    const gqm_cdt_in &d = in[ids[k]];
    in_off[k] = in_bytes;
    in_bytes += up256(16ull * d.numberofpoints) + 2 * up256(12ull * d.numberoftriangles) +
                up256(8ull * d.numberofsegments);
    const Caps c = caps_of(d.numberofpoints, d.numberoftriangles, d.numberofsegments);
    arena = std::max(arena, arena_bytes(c));
    out_bound += out_layout(c.pphys, c.tphys, c.sphys).bytes;
  }
  // grid: resident blocks of the variant, bounded by the domains and memory
  const Variant &V = kVariants[var];
  int per_sm = V.minb, nb = 1;
#ifndef GQM_HOST_EMU
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, V.fn, V.threads, 0) == cudaSuccess && occ > 0)
    per_sm = occ;
  else
    cudaGetLastError();
#endif
  const long resident = (long)C.sms * per_sm;
  if (var == kTeamVariant) nb = blocks_per_team(in, ids, resident);
  long grid = std::min<long>(resident / nb, n);  // teams
#ifndef GQM_HOST_EMU
  size_t freeb = 0, totb = 0;
  cudaMemGetInfo(&freeb, &totb);
  const size_t have = (size_t)(mem_fraction * (double)(freeb + C.in_cap + C.out_cap + C.arena_cap));
  const size_t fixed = up256(in_bytes) + up256(out_bound);
  if (fixed + arena > have) return GQM_ERR_MEMORY;
  grid = std::min<long>(grid, (long)((have - fixed) / arena));
#else
  (void)mem_fraction;
  grid = std::min(grid, std::max(1L, (long)GQM_EMU_BLOCKS / nb));
#endif
  if (grid < 1) return GQM_ERR_MEMORY;
  if (grow_dev(&C.d_in, &C.in_cap, in_bytes) || grow_dev(&C.d_out, &C.out_cap, out_bound) ||
      grow_dev(&C.d_arena, &C.arena_cap, arena * (size_t)grid) || grow_host(&C.h_in, &C.h_in_cap, in_bytes))
    return GQM_ERR_MEMORY;
  if (nb > 1 && (grow_dev(&C.d_teams, &C.teams_cap, sizeof(TeamState) * (size_t)grid) ||
                 cudaMemsetAsync(C.d_teams, 0, sizeof(TeamState) * (size_t)grid, C.st) != cudaSuccess))
    return GQM_ERR_MEMORY;
  if (n > C.jobs_cap) {
    if (C.d_jobs) cudaFree(C.d_jobs);
    if (C.d_order) cudaFree(C.d_order);
    C.d_jobs = nullptr;
    C.d_order = nullptr;
    C.jobs_cap = 0;
    if (cudaMalloc((void **)&C.d_jobs, sizeof(Job) * n) != cudaSuccess ||
        cudaMalloc((void **)&C.d_order, sizeof(int) * n) != cudaSuccess)
      return GQM_ERR_MEMORY;
    C.jobs_cap = n;
  }
  // inputs packed into pinned memory on the host's cores and uploaded in
  // pieces of 32 MB, the front while the back is packed
  std::vector<Job> jobs(n);
  {
    std::vector<HostCopy> parts;
    parts.reserve(4 * (size_t)n);
    for (int k = 0; k < n; ++k) {
      const gqm_cdt_in &D = in[ids[k]];
      char *h = C.h_in + in_off[k];
      const size_t bp = up256(16ull * D.numberofpoints), bt = up256(12ull * D.numberoftriangles);
      parts.push_back({h, D.pointlist, 16ull * D.numberofpoints});
      parts.push_back({h + bp, D.trianglelist, 12ull * D.numberoftriangles});
      parts.push_back({h + bp + bt, D.neighborlist, 12ull * D.numberoftriangles});
      if (D.numberofsegments) parts.push_back({h + bp + 2 * bt, D.segmentlist, 8ull * D.numberofsegments});
    }
    host_copy_streamed(parts, C.h_in, 32u << 20, [&](size_t off, size_t bytes) {
      cudaMemcpyAsync(C.d_in + off, C.h_in + off, bytes, cudaMemcpyHostToDevice, C.st);
    });
  }
  for (int k = 0; k < n; ++k) {
    const int d = ids[k];
    const gqm_cdt_in &D = in[d];
    char *g = C.d_in + in_off[k];
    const size_t bp = up256(16ull * D.numberofpoints), bt = up256(12ull * D.numberoftriangles);
    Job &J = jobs[k];
    memset(&J, 0, sizeof(J));
    J.pts = reinterpret_cast<const double2 *>(g);
    J.tri = reinterpret_cast<const int *>(g + bp);
    J.nbr = reinterpret_cast<const int *>(g + bp + bt);
    J.seg = reinterpret_cast<const int2 *>(g + bp + 2 * bt);
    J.np = D.numberofpoints;
    J.nt = D.numberoftriangles;
    J.ns = D.numberofsegments;
    const gqm_options &o = opt[d];
    J.theta = o.theta;
    J.max_area = o.max_area > 0.0 ? o.max_area : 0.0;
    J.mode = o.mode ? 1 : 0;
    J.pred = o.predicates ? 1 : 0;
    J.max_rounds = o.max_rounds > 0 ? o.max_rounds : 1000000;
    J.offcenter = 0;
    double offc = 0.0;
    if (o.insert_policy == GQM_OFFCENTER) {  // refine.cu:6555-6567, evaluated on the host as there
      J.offcenter = 1;
      const double cg = cos(o.theta * GQM_PI / 180);
      offc = 0.475 * sqrt((1.0 + cg) / (1.0 - cg));
    }
    J.offconstant = (int)offc;
    J.obase = C.d_out;
    J.oused = C.d_used;
    J.ocap = out_bound;
    J.status = GQM_ERR_CUDA;  // overwritten by the block that refines it
  }
  // networks of the learned placement: one device copy per distinct array
  std::vector<const float *> nets;
  for (int k = 0; k < n; ++k) {
    const gqm_options &o = opt[ids[k]];
    if (o.placement == GQM_PLACE_LEARNED && std::find(nets.begin(), nets.end(), o.mlp) == nets.end())
      nets.push_back(o.mlp);
  }
  char *dnet = nullptr;
  const size_t net_bytes = up256(sizeof(uint16_t) * kMlpW) + up256(sizeof(float) * kMlpB);
  if (!nets.empty()) {
    if (cudaMalloc((void **)&dnet, net_bytes * nets.size()) != cudaSuccess) return GQM_ERR_MEMORY;
    std::vector<char> h(net_bytes * nets.size());
    for (size_t i = 0; i < nets.size(); ++i)
      mlp_pack(nets[i], reinterpret_cast<uint16_t *>(h.data() + i * net_bytes),
               reinterpret_cast<float *>(h.data() + i * net_bytes + up256(sizeof(uint16_t) * kMlpW)));
    cudaMemcpy(dnet, h.data(), h.size(), cudaMemcpyHostToDevice);
  }
  for (int k = 0; k < n; ++k) {
    const gqm_options &o = opt[ids[k]];
    jobs[k].placement = o.placement == GQM_PLACE_LEARNED ? GQM_PLACE_LEARNED : GQM_PLACE_PLAIN;
    if (jobs[k].placement == GQM_PLACE_LEARNED) {
      const size_t i = (size_t)(std::find(nets.begin(), nets.end(), o.mlp) - nets.begin());
      char *base = dnet + i * net_bytes;
      jobs[k].mlp = mlp_dev(reinterpret_cast<uint16_t *>(base),
                            reinterpret_cast<float *>(base + up256(sizeof(uint16_t) * kMlpW)));
    }
  }
  // largest first
  std::vector<int> order(n);
  for (int k = 0; k < n; ++k) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return jobs[a].np > jobs[b].np; });
  cudaMemcpyAsync(C.d_jobs, jobs.data(), sizeof(Job) * n, cudaMemcpyHostToDevice, C.st);
  cudaMemcpyAsync(C.d_order, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice, C.st);
  cudaMemsetAsync(C.d_next, 0, sizeof(int), C.st);
  cudaMemsetAsync(C.d_used, 0, sizeof(unsigned long long), C.st);
  if (cudaStreamSynchronize(C.st) != cudaSuccess) return GQM_ERR_CUDA;
  const double h2d = ms_since(t0);
  // the persistent launch
  cudaEventRecord(C.e0, C.st);
  TeamState *teams = reinterpret_cast<TeamState *>(C.d_teams);
#ifdef GQM_HOST_EMU
  GQM_EMU_GRID((int)grid * nb,
               V.fn(C.d_jobs, C.d_order, n, C.d_next, C.d_arena, arena, teams, nb, jobs[0].pred));
#else
  {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // blocks of a team wait for one another
    at[0].val.cooperative = 1;
    cfg.gridDim = dim3((unsigned)(grid * nb));
    cfg.blockDim = dim3((unsigned)V.threads);
    cfg.stream = C.st;
    cfg.attrs = at;
    cfg.numAttrs = nb > 1 ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, V.fn, C.d_jobs, (const int *)C.d_order, n, C.d_next, C.d_arena, arena, teams, nb,
                           jobs[0].pred) != cudaSuccess) {
      if (dnet) cudaFree(dnet);
      return GQM_ERR_CUDA;
    }
  }
#endif
  cudaEventRecord(C.e1, C.st);
  if (cudaStreamSynchronize(C.st) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    if (dnet) cudaFree(dnet);
    return GQM_ERR_CUDA;
  }
  float kms = 0.0f;
  cudaEventElapsedTime(&kms, C.e0, C.e1);
  if (dnet) cudaFree(dnet);
  // results: the job table, then the used part of the output region
  auto t1 = std::chrono::steady_clock::now();
  unsigned long long used = 0;
  cudaMemcpy(jobs.data(), C.d_jobs, sizeof(Job) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(&used, C.d_used, sizeof(used), cudaMemcpyDeviceToHost);
  // a large output region is downloaded straight into a pinned block that the
  // domains' results share (released by the last gqm_free_result); a smaller
  // one through the staging buffer into malloc()ed arrays
  char *blk = nullptr;
  if (keep_outputs) {
    int nres = 0;
    for (int k = 0; k < n; ++k) nres += jobs[k].status == GQM_OK;
    blk = gqm_pinned_take((size_t)used, nres);
    if (blk) {
      if (cudaMemcpy(blk, C.d_out, (size_t)used, cudaMemcpyDeviceToHost) != cudaSuccess) {
        for (int k = 0; k < nres; ++k) gqm_pinned_give(blk);
        return GQM_ERR_CUDA;
      }
    } else {
      if (grow_host(&C.h_out, &C.h_out_cap, (size_t)used)) return GQM_ERR_MEMORY;
      if (used && cudaMemcpy(C.h_out, C.d_out, (size_t)used, cudaMemcpyDeviceToHost) != cudaSuccess)
        return GQM_ERR_CUDA;
    }
  }
  int alloc_fail = 0;
  for (int k = 0; k < n; ++k) {
    const int d = ids[k];
    const Job &J = jobs[k];
    status[d] = J.status;
    if (J.status != GQM_OK) continue;
    if (stats) {
      gqm_stats &s = stats[d];
      memset(&s, 0, sizeof(s));
      s.rounds = J.rounds;
      s.flip_steps = J.flip_steps;
      s.steiner_inserted = J.steiner;
      s.midpoints_inserted = J.midpoints;
      s.bad_total = J.bad_total;
      s.exact_fallbacks = J.exact_fallbacks;
      s.learned_candidates = J.learned_candidates;
      s.learned_used = J.learned_used;
      s.goodcos2 = J.goodcos2;
      s.kernel_launches = 1;
      s.device_ms = kms;
    }
    if (!keep_outputs) continue;
    gqm_cdt_out &R = out[d];
    R.numberofpoints = J.out_np;
    R.numberoftriangles = J.out_nt;
    R.numberofsegments = J.out_ns;
    if (blk) {
      const OutLayout L = out_layout(J.out_np, J.out_nt, J.out_ns);
      char *o = blk + J.ooff;
      R.pointlist = reinterpret_cast<double *>(o + L.pts);
      R.trianglelist = reinterpret_cast<int *>(o + L.tri);
      R.neighborlist = reinterpret_cast<int *>(o + L.nbr);
      R.segmentlist = reinterpret_cast<int *>(o + L.seg);
      R.pstatus = reinterpret_cast<unsigned char *>(o + L.ps);
      R.tstatus = reinterpret_cast<unsigned char *>(o + L.ts);
      continue;
    }
    R.pointlist = (double *)malloc(16ull * J.out_np + 16);
    R.trianglelist = (int *)malloc(12ull * J.out_nt + 16);
    R.neighborlist = (int *)malloc(12ull * J.out_nt + 16);
    R.segmentlist = (int *)malloc(8ull * J.out_ns + 16);
    R.pstatus = (unsigned char *)malloc((size_t)J.out_np + 16);
    R.tstatus = (unsigned char *)malloc((size_t)J.out_nt + 16);
    if (!R.pointlist || !R.trianglelist || !R.neighborlist || !R.segmentlist || !R.pstatus || !R.tstatus)
      alloc_fail = 1;
  }
  if (alloc_fail) return GQM_ERR_MEMORY;  // the caller releases every out[]
  if (keep_outputs && !blk)
    parallel_for(n, [&](int k) {
      const Job &J = jobs[k];
      if (J.status != GQM_OK) return;
      const OutLayout L = out_layout(J.out_np, J.out_nt, J.out_ns);
      const char *o = C.h_out + J.ooff;
      gqm_cdt_out &R = out[ids[k]];
      memcpy(R.pointlist, o + L.pts, 16ull * J.out_np);
      memcpy(R.trianglelist, o + L.tri, 12ull * J.out_nt);
      memcpy(R.neighborlist, o + L.nbr, 12ull * J.out_nt);
      memcpy(R.segmentlist, o + L.seg, 8ull * J.out_ns);
      memcpy(R.pstatus, o + L.ps, (size_t)J.out_np);
      memcpy(R.tstatus, o + L.ts, (size_t)J.out_nt);
    });
  if (rep) {
    rep->grid = (int)(grid * nb);
    rep->threads_per_block = V.threads;
    rep->blocks_per_sm = V.minb;
    rep->arena_bytes = (long long)arena;
    rep->kernel_ms += kms;
    rep->h2d_ms += h2d;
    rep->d2h_ms += ms_since(t1);
  }
  return GQM_OK;
}

int setup_dev(DevCache &C, int device) {
  if (cudaSetDevice(device) != cudaSuccess) return GQM_ERR_NO_DEVICE;
  if (C.init) return GQM_OK;
  if (cudaStreamCreateWithFlags(&C.st, cudaStreamNonBlocking) != cudaSuccess) return GQM_ERR_CUDA;
  if (cudaEventCreate(&C.e0) != cudaSuccess || cudaEventCreate(&C.e1) != cudaSuccess) return GQM_ERR_CUDA;
  if (cudaMalloc((void **)&C.d_next, sizeof(int)) != cudaSuccess ||
      cudaMalloc((void **)&C.d_used, sizeof(unsigned long long)) != cudaSuccess)
    return GQM_ERR_MEMORY;
#ifndef GQM_HOST_EMU
  cudaDeviceGetAttribute(&C.sms, cudaDevAttrMultiProcessorCount, device);
#else
  C.sms = GQM_EMU_BLOCKS;
#endif
  C.init = true;
  return GQM_OK;
}

int variant_of(const DevCache &C, const gqm_batch_options *b) {
  if (b && b->threads_per_block > 0) {
    for (int v = 0; v < kNumVariants; ++v)
      if (kVariants[v].threads == b->threads_per_block &&
          (b->blocks_per_sm <= 0 || kVariants[v].minb == b->blocks_per_sm))
        return v;
    return -1;
  }
  return C.tuned >= 0 ? C.tuned : kDefaultVariant;
}

// The whole call on one device: validation, the persistent launches (one per
// predicate mode present), then the single-domain path for domains that
// outgrew their arena.
int batch_call(int nd, const gqm_cdt_in *in, gqm_cdt_out *out, const gqm_options *opt, gqm_stats *stats,
               const gqm_batch_options *bopt, gqm_batch_report *rep, int *failed, int force_var, bool keep) {
  auto t0 = std::chrono::steady_clock::now();
  if (failed) *failed = -1;
  if (nd < 0 || (nd > 0 && (!in || !opt || (keep && !out)))) return GQM_ERR_ARGUMENT;
  if (rep) memset(rep, 0, sizeof(*rep));
  if (keep)
    for (int i = 0; i < nd; ++i) memset(&out[i], 0, sizeof(gqm_cdt_out));
  if (nd == 0) return GQM_OK;
  const int device = opt[0].device;
  if (device < 0 || device >= 16) return GQM_ERR_NO_DEVICE;
  for (int i = 0; i < nd; ++i) {
    int rc = check_domain(&in[i], &opt[i]);
    if (rc == GQM_OK && opt[i].device != device) rc = GQM_ERR_ARGUMENT;
    if (rc) {
      if (failed) *failed = i;
      return rc;
    }
  }
  DevCache &C = g_dev[device];
  std::lock_guard<std::mutex> lock(C.mu);
  int rc = setup_dev(C, device);
  if (rc) return rc;
  const int var = force_var >= 0 ? force_var : variant_of(C, bopt);
  if (var < 0) return GQM_ERR_ARGUMENT;
  const double frac = (bopt && bopt->memory_fraction > 0.0) ? bopt->memory_fraction : 0.8;
  std::vector<int> status(nd, GQM_ERR_CUDA);
  for (int pred = 0; pred < 2; ++pred) {
    std::vector<int> ids;
    for (int i = 0; i < nd; ++i)
      if ((opt[i].predicates ? 1 : 0) == pred) ids.push_back(i);
    rc = run_batch(C, ids, in, out, opt, stats, var, frac, status.data(), rep, keep);
    if (rc) {
      if (keep)
        for (int j = 0; j < nd; ++j) gqm_free_result(&out[j]);
      return rc;
    }
  }
  // domains that outgrew their arena: the single-domain path
  for (int i = 0; i < nd; ++i) {
    if (status[i] != GQM_ERR_ARENA) continue;
    if (rep) rep->fallbacks++;
    if (!keep) {
      status[i] = GQM_OK;
      continue;
    }
    gqm_stats st;
    status[i] = gqm_refine(&in[i], &out[i], &opt[i], &st);
    if (status[i] == GQM_OK && stats) stats[i] = st;
  }
  for (int i = 0; i < nd; ++i)
    if (status[i] != GQM_OK) {
      if (failed) *failed = i;
      if (keep)
        for (int j = 0; j < nd; ++j) gqm_free_result(&out[j]);
      return status[i];
    }
  if (rep) rep->total_ms = ms_since(t0);
  return GQM_OK;
}

}  // namespace
}  // namespace gqm

// The refinement of one domain on the single-domain engine's buffers (refine.cu)
// by one cooperative launch of `blocks` blocks.  scratch, caps, run and state
// are the caller's Scratch, Caps, device EngineRun and device TeamState (the
// same layouts in both compilations).
int gqm_refine_one_launch(const void *scratch, size_t scratch_bytes, const void *caps, void *run, void *state, int pred,
                          int blocks, int small_limit, void *ktimer, void *stimer, cudaStream_t st) {
  using namespace gqm;
  if (scratch_bytes != sizeof(Scratch)) return GQM_ERR_ARGUMENT;
  Scratch S;
  Caps c;
  memcpy(&S, scratch, sizeof(S));
  memcpy(&c, caps, sizeof(c));
  EngineRun *r = static_cast<EngineRun *>(run);
  TeamState *ts = static_cast<TeamState *>(state);
  KTimer *kt = static_cast<KTimer *>(ktimer), *stm = static_cast<KTimer *>(stimer);
#ifdef GQM_HOST_EMU
  (void)blocks;
  (void)st;
  GQM_EMU_GRID(blocks, (pred ? k_refine_one<1> : k_refine_one<0>)(S, c, r, ts, small_limit, kt, stm));
  return GQM_OK;
#else
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(512);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = pred ? cudaLaunchKernelEx(&cfg, k_refine_one<1>, S, c, r, ts, small_limit, kt, stm)
                             : cudaLaunchKernelEx(&cfg, k_refine_one<0>, S, c, r, ts, small_limit, kt, stm);
  return e == cudaSuccess ? GQM_OK : GQM_ERR_CUDA;
#endif
}
// The incircle expansion-fallback counter of this translation unit's kernels
// (see gqm_fallbacks_cluster in flipcl.cu).
int gqm_fallbacks_cta(unsigned long long *sum, int reset, cudaStream_t st) {
  unsigned long long v = 0;
#ifdef GQM_HOST_EMU
  (void)st;
  v = gqm::g_incircle_fallbacks;
  if (reset) gqm::g_incircle_fallbacks = 0;
#else
  if (sum && (cudaMemcpyFromSymbolAsync(&v, gqm::g_incircle_fallbacks, sizeof(v), 0, cudaMemcpyDeviceToHost, st) !=
                  cudaSuccess ||
              cudaStreamSynchronize(st) != cudaSuccess))
    return GQM_ERR_CUDA;
  if (reset) {
    const unsigned long long zero = 0;
    if (cudaMemcpyToSymbolAsync(gqm::g_incircle_fallbacks, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st) !=
        cudaSuccess)
      return GQM_ERR_CUDA;
  }
#endif
  if (sum) *sum += v;
  return GQM_OK;
}

extern "C" {

void gqm_default_batch_options(gqm_batch_options *b) {
  if (!b) return;
  b->threads_per_block = 0;
  b->blocks_per_sm = 0;
  b->memory_fraction = 0.0;
}

int gqm_refine_batch_persistent(int ndomains, const gqm_cdt_in *in, gqm_cdt_out *out, const gqm_options *opt,
                                gqm_stats *stats, const gqm_batch_options *bopt, gqm_batch_report *report,
                                int *failed_domain) {
  return gqm::batch_call(ndomains, in, out, opt, stats, bopt, report, failed_domain, -1, true);
}

int gqm_batch_variants(int *threads, int *blocks_per_sm, int max) {
  for (int v = 0; v < gqm::kNumVariants && v < max; ++v) {
    if (threads) threads[v] = gqm::kVariants[v].threads;
    if (blocks_per_sm) blocks_per_sm[v] = gqm::kVariants[v].minb;
  }
  return gqm::kNumVariants;
}

int gqm_batch_autotune(int ndomains, const gqm_cdt_in *in, const gqm_options *opt, gqm_batch_options *chosen,
                       double *ms_per_variant) {
  if (ndomains <= 0 || !in || !opt) return GQM_ERR_ARGUMENT;
  int best = -1;
  double best_ms = 0.0;
  for (int v = 0; v < gqm::kNumVariants; ++v) {
    gqm_batch_report r;
    int failed = -1;
    int rc = gqm::batch_call(ndomains, in, nullptr, opt, nullptr, nullptr, &r, &failed, v, false);
    if (rc) return rc;
    if (ms_per_variant) ms_per_variant[v] = r.kernel_ms;
    if (best < 0 || r.kernel_ms < best_ms) {
      best = v;
      best_ms = r.kernel_ms;
    }
  }
  const int device = opt[0].device;
  {
    std::lock_guard<std::mutex> lock(gqm::g_dev[device].mu);
    gqm::g_dev[device].tuned = best;
  }
  if (chosen) {
    chosen->threads_per_block = gqm::kVariants[best].threads;
    chosen->blocks_per_sm = gqm::kVariants[best].minb;
    chosen->memory_fraction = 0.0;
  }
  return GQM_OK;
}

void gqm_batch_release(int device) {
  if (device < 0 || device >= 16) return;
  gqm::DevCache &C = gqm::g_dev[device];
  std::lock_guard<std::mutex> lock(C.mu);
  if (!C.init) return;
  cudaSetDevice(device);
  cudaStreamSynchronize(C.st);
  void *dev[] = {C.d_in, C.d_out, C.d_arena, C.d_jobs, C.d_order, C.d_next, C.d_used, C.d_teams};
  for (void *p : dev)
    if (p) cudaFree(p);
  if (C.h_in) cudaFreeHost(C.h_in);
  if (C.h_out) cudaFreeHost(C.h_out);
  cudaEventDestroy(C.e0);
  cudaEventDestroy(C.e1);
  cudaStreamDestroy(C.st);
  const int tuned = C.tuned;
  C.d_in = C.d_out = C.d_arena = C.h_in = C.h_out = C.d_teams = nullptr;
  C.in_cap = C.out_cap = C.arena_cap = C.h_in_cap = C.h_out_cap = C.teams_cap = 0;
  C.d_jobs = nullptr;
  C.d_order = nullptr;
  C.jobs_cap = 0;
  C.d_next = nullptr;
  C.d_used = nullptr;
  C.init = false;
  C.tuned = tuned;
}

}  // extern "C"
