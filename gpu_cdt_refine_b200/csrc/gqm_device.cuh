// Device-side mesh layout and per-element helpers of the B200 refiner.
//
// Layout (structure of arrays, resident in HBM for the whole refinement):
//   pts   double2[Pcap]   vertex coordinates (one 128-bit load each)
//   ps    uint8[Pcap]     point flags: DELETED | STEINER | SEGSPLIT | NEW
//   pred  uint8[Pcap]     "redundant" flag (set concurrently by many threads)
//   tv    int4[Tcap]      triangle vertices (x, y, z), w unused
//   tn    int4[Tcap]      oriented neighbours (tri << 2 | edge), -1 boundary
//   tsg   int4[Tcap]      subsegment on each edge, -1 if none
//   tst   uint8[Tcap]     NOTNULL | BAD | CHECK
//   tflip uint8[Tcap]     flip-flop marker (set concurrently)
//   tfo   uint8[Tcap]     flip orientation code, 15 = none
//   tmark int[Tcap]       ownership marker of insertions (atomicMin)
//   fmark uint64[Tcap]    claim of a flip step (atomicMin), fstamp int[Tcap]
//   emap  int4[Tcap]      edge map of a flip step
//   s2t   u128[Scap]      subsegment -> oriented triangle in the low word,
//                         tagged with the launch epoch and the storing
//                         thread's key (see s2t_store)
//   s2seg int[Scap], enc int[Scap], segs int2[S_in]
// Edge i of a triangle joins vertices i+1 and i+2 and faces vertex i; an
// oriented triangle (t << 2 | i) names edge i of t (GPU_Refine/refine.cu:95-113).
// Flags the reference keeps in one byte (GPU_Refine/refine.h:36-205) are split
// across separate byte arrays so that concurrent writers never share a byte.
#pragma once
#include <cstdint>

#include "predicates.h"

namespace gqm {

constexpr int kMaxInt = 2147483647;
// subseg2tri entry: bits 127..64 launch epoch, 63..32 writer key, 31..0 oriented triangle
typedef unsigned __int128 s2t_t;
constexpr int kCavityCap = 50;  // MyList capacity, GPU_Refine/refine.h:30

enum : uint8_t { PS_DELETED = 1, PS_STEINER = 2, PS_SEGSPLIT = 4, PS_NEW = 8 };
enum : uint8_t { TS_NOTNULL = 1, TS_BAD = 2, TS_CHECK = 4 };

struct Mesh {
  double2 *pts;
  uint8_t *ps, *pred;
  int4 *tv, *tn, *tsg;
  uint8_t *tst, *tflip, *tfo;
  int *tmark;
  int *fstamp;  // generation that last queued the triangle for a flip step
  unsigned long long *fmark;  // claim of a flip step (see claim_key)
  int4 *emap;  // where the triangle's edges went in the flip step of generation w
  s2t_t *s2t;
  int *s2seg, *enc;
  const int2 *segs;
  int *err;  // first error code raised on the device
  double gc2;  // cos^2(theta), computed on the device as the reference does
  double max_area;  // area bound (0: none): larger triangles are bad whatever their angles
  int mode;    // 1 Ruppert, 0 Chew
};

__device__ __forceinline__ int dtri(int o) { return o >= 0 ? (o >> 2) : -1; }
__device__ __forceinline__ int dori(int o) { return o & 3; }
__device__ __forceinline__ int etri(int t, int o) { return t >= 0 ? ((t << 2) | o) : -1; }
__device__ __forceinline__ int negate_idx(int i) { return -i - 3; }
__device__ __forceinline__ int m3(int i) { return i >= 3 ? i - 3 : i; }

__device__ __forceinline__ int comp(const int4 &v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : v.z); }
__device__ __forceinline__ void setc(int4 &v, int i, int x) {
  if (i == 0)
    v.x = x;
  else if (i == 1)
    v.y = x;
  else
    v.z = x;
}
// single-component stores into an int4 row
__device__ __forceinline__ void st1(int4 *a, int t, int i, int x) { reinterpret_cast<int *>(a + t)[i] = x; }
__device__ __forceinline__ int ld1(const int4 *a, int t, int i) { return reinterpret_cast<const int *>(a + t)[i]; }

__device__ __forceinline__ int s2t_get(const Mesh &M, int s) { return (int)(uint32_t)M.s2t[s]; }
__device__ __forceinline__ s2t_t s2t_plain(int v) { return (s2t_t)(uint32_t)v; }  // epoch 0: older than any launch
// Key of a store into subseg2tri by the thread at position `pos` of a launch,
// `slot` being the store's place in the kernel's program order.  When threads
// of one launch store into the same entry, the largest key is kept: within a
// warp the later store instruction (a warp issues its stores in order) and,
// for one instruction, the lower lane; across warps the lower warp.  That is
// the order in which the reference's racing stores (GPU_Refine/refine.cu:
// 1362-1372, 1419-1424, 1533-1544, 2844-2850, 2900-2903, 4744-4876) were seen
// to land on a B200, and the oracle applies the same key.
__device__ __forceinline__ uint32_t wkey(int pos, int slot) {
  return ((0x7FFFFFu - ((uint32_t)pos >> 5)) << 9) | ((uint32_t)slot << 5) | (31u - ((uint32_t)pos & 31u));
}
// A value stored in an earlier launch always loses to one of this launch; in
// one launch the larger (epoch, key) wins.  The loop reads the entry with the
// compare-and-swap itself, so a torn read is never acted on.
__device__ __forceinline__ void s2t_store(const Mesh &M, int s, int v, uint32_t epoch, uint32_t key) {
  const s2t_t nw = ((s2t_t)epoch << 64) | ((s2t_t)key << 32) | (uint32_t)v;
  s2t_t cur = 0;
  for (;;) {
    const s2t_t o = atomicCAS(M.s2t + s, cur, nw);
    if (o == cur || (o >> 32) >= (nw >> 32)) return;
    cur = o;
  }
}

// A store that no other thread of the launch competes with.
__device__ __forceinline__ void s2t_put(const Mesh &M, int s, int v, uint32_t epoch) {
  M.s2t[s] = ((s2t_t)epoch << 64) | ((s2t_t)0xFFFFFFFFu << 32) | (uint32_t)v;
}

// Slot in a list whose length *n many threads bump at once: the lanes of a
// warp that arrive together take consecutive slots with one atomic, issued by
// the lowest of them, instead of one atomic each on the same word.  The order
// of the entries within a list is not used by any step.
__device__ __forceinline__ int list_slot(int *n) {
#ifdef GQM_HOST_EMU
  return atomicAdd(n, 1);
#else
  const unsigned m = __activemask();
  const int lane = (int)(threadIdx.x & 31u), leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(n, __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
#endif
}
// Two consecutive slots.
__device__ __forceinline__ int list_slot2(int *n) {
#ifdef GQM_HOST_EMU
  return atomicAdd(n, 2);
#else
  const unsigned m = __activemask();
  const int lane = (int)(threadIdx.x & 31u), leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(n, 2 * __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + 2 * __popc(m & ((1u << lane) - 1u));
#endif
}
// The same for an event counter: one atomic per warp.
__device__ __forceinline__ void count_event(unsigned long long *c) {
#ifdef GQM_HOST_EMU
  atomicAdd(c, 1ull);
#else
  const unsigned m = __activemask();
  if ((int)(threadIdx.x & 31u) == __ffs(m) - 1) atomicAdd(c, (unsigned long long)__popc(m));
#endif
}
__device__ __forceinline__ void raise_err(const Mesh &M, int code) { atomicCAS(M.err, 0, code); }

// ---------------------------------------------------------------------------
// Predicates with the reference's effective arithmetic (PRED = 0) or exact
// (PRED = 1).  Orientation: cuda_fast / cuda_ccw.  Incircle: the
// "cuda_inCircle, then cuda_inCircle_exact if 0" pattern used by every caller.
// ---------------------------------------------------------------------------
template <int PRED>
__device__ __forceinline__ double orient(double2 a, double2 b, double2 c) {
  if (PRED == 0) return gqm_orient_ref(a.x, a.y, b.x, b.y, c.x, c.y);
  return gqm_orient_exact(a.x, a.y, b.x, b.y, c.x, c.y);
}
// Incircle tests that needed the expansion path (determinant exactly zero with
// the reference's arithmetic, filter inconclusive with exact arithmetic),
// summed over every refinement on the device since the last reset (one
// counter per compiled module).
static __device__ unsigned long long g_incircle_fallbacks;
template <int PRED>
__device__ __noinline__ double incircle_slow(double2 a, double2 b, double2 c, double2 d) {
  atomicAdd(&g_incircle_fallbacks, 1ull);
  if (PRED == 0) return gqm_incircle_zero_fallback_ref(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y);
  return gqm_incircle_exact(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y);
}
// The test before any fallback; *open is set when its sign is not decided.
template <int PRED>
__device__ __forceinline__ double incircle_fast(double2 a, double2 b, double2 c, double2 d, bool *open) {
  if (PRED == 0) {
    const double r = gqm_incircle_det_ref(a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y);
    if (r == 0) *open = true;
    return r;
  }
  // exact: filter then exact expansion
  double adx = a.x - d.x, bdx = b.x - d.x, cdx = c.x - d.x;
  double ady = a.y - d.y, bdy = b.y - d.y, cdy = c.y - d.y;
  double bdxcdy = bdx * cdy, cdxbdy = cdx * bdy, alift = adx * adx + ady * ady;
  double cdxady = cdx * ady, adxcdy = adx * cdy, blift = bdx * bdx + bdy * bdy;
  double adxbdy = adx * bdy, bdxady = bdx * ady, clift = cdx * cdx + cdy * cdy;
  double det = alift * (bdxcdy - cdxbdy) + blift * (cdxady - adxcdy) + clift * (adxbdy - bdxady);
  double perm = (fabs(bdxcdy) + fabs(cdxbdy)) * alift + (fabs(cdxady) + fabs(adxcdy)) * blift +
                (fabs(adxbdy) + fabs(bdxady)) * clift;
  double eb = (10.0 + 96.0 * GQM_EPS) * GQM_EPS * perm;
  if (!(det > eb || -det > eb)) *open = true;
  return det;
}
template <int PRED>
__device__ __forceinline__ double incircle(double2 a, double2 b, double2 c, double2 d) {
  bool open = false;
  const double r = incircle_fast<PRED>(a, b, c, d, &open);
  return open ? incircle_slow<PRED>(a, b, c, d) : r;
}

// checkseg4encroach, GPU_Refine/refine.cu:115-139 (goodcoss squared once).
__device__ __forceinline__ bool encroached(double2 o, double2 d, double2 a, double gc2, int mode) {
  double dot = gqm_madd(o.x - a.x, d.x - a.x, (o.y - a.y) * (d.y - a.y));
  if (dot < 0.0) {
    if (mode || dot * dot >= (2.0 * gc2 - 1.0) * (2.0 * gc2 - 1.0) *
                                   gqm_madd(o.x - a.x, o.x - a.x, (o.y - a.y) * (o.y - a.y)) *
                                   gqm_madd(d.x - a.x, d.x - a.x, (d.y - a.y) * (d.y - a.y)))
      return true;
  }
  return false;
}

}  // namespace gqm
