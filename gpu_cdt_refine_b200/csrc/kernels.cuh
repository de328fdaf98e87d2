// Kernels of the B200 refiner.  Each kernel restates one step of the
// reference's GPU pipeline (GPU_Refine/refine.cu; the line ranges are cited at
// every kernel) over the structure-of-arrays mesh of gqm_device.cuh.  Kernels
// are grid-stride loops whose element count is read from device memory, so a
// launch never waits for the host to learn a count.
#pragma once
#include "gqm_device.cuh"
#include "learned.cuh"
#include "team.cuh"

// Register budget of the latency-bound walk kernels (flip checks, cavity
// walks, link updates): ask for at least this many resident 256-thread blocks
// per SM, so enough warps are in flight to cover their dependent loads.
#ifndef GQM_WALK_MIN_BLOCKS
#define GQM_WALK_MIN_BLOCKS 2
#endif

// Three compilations of the same kernels:
//  * grid mode (default): every step below is a __global__ kernel whose
//    grid-stride loop covers its items across the whole grid;
//  * CTA mode (GQM_CTA_MODE, batch.cu): every step is a __device__ function
//    that a team of one or more thread blocks runs over one domain's items, the
//    team's threads striding over them; the caller separates steps with the
//    team's barrier (engine.cuh);
//  * cluster mode (GQM_CLUSTER_MODE, flipcl.cu): the same with the whole grid
//    as the team; of the steps below only the flip-flop loop is used there.
#if defined(GQM_CTA_MODE)
#define GQM_KERNEL __device__
#define GQM_WALK_BOUNDS
#define GQM_BOUNDS(minb)
#define GQM_GTID ((int)(gqm_team_rank * blockDim.x + threadIdx.x))
#define GQM_GSIZE ((int)(gqm_team_blocks * blockDim.x))
#define GQM_BLOCK0 (gqm_team_rank == 0)
#define GQM_WALK_CALL __noinline__
#elif defined(GQM_CLUSTER_MODE)
#define GQM_KERNEL __device__
#define GQM_WALK_BOUNDS
#define GQM_BOUNDS(minb)
#define GQM_GTID ((int)(blockIdx.x * blockDim.x + threadIdx.x))
#define GQM_GSIZE ((int)(gridDim.x * blockDim.x))
#define GQM_BLOCK0 (blockIdx.x == 0)
#define GQM_WALK_CALL
#else
#define GQM_KERNEL __global__
#define GQM_WALK_BOUNDS __launch_bounds__(256, GQM_WALK_MIN_BLOCKS)
#define GQM_BOUNDS(minb) __launch_bounds__(256, minb)
#define GQM_GTID ((int)(blockIdx.x * blockDim.x + threadIdx.x))
#define GQM_GSIZE ((int)(gridDim.x * blockDim.x))
#define GQM_BLOCK0 (blockIdx.x == 0)
#define GQM_WALK_CALL
#endif

namespace gqm {

#if defined(GQM_CTA_MODE)
// the block's place in its team, and the team's blocks
__shared__ int gqm_team_rank, gqm_team_blocks;
#endif

#define GS_LOOP(i, n) for (int i = GQM_GTID; i < (n); i += GQM_GSIZE)

// Counts and slot lists that some kernels take either as values (the
// block-mode engine, whose driver holds them in registers) or as device words
// that an earlier kernel of the same CUDA graph wrote (the single-domain
// engine, whose driver state lives on the device).
struct DevInt {
  const int *p;
};
__device__ __forceinline__ int nval(int n) { return n; }
__device__ __forceinline__ int nval(DevInt d) { return *d.p; }
// free slots handed out from base[*off] on
struct DevSlots {
  const int *base;
  const int *off;
};
__device__ __forceinline__ const int *slots_of(const int *p) { return p; }
__device__ __forceinline__ const int *slots_of(DevSlots s) { return s.base + *s.off; }

// ============================================================================
// Initialisation (refine.cu:5557-5747, 3105-3151)
// ============================================================================

// findIncidentOri (refine.cu:35-93): edge index, in neighbour n, of the edge
// shared with t; -1 when they do not share two vertices.
__device__ __forceinline__ int incident_ori(const int *tri, int t, int n) {
  if (t < 0 || n < 0) return -1;
  int inc0 = -1, inc1 = -1, count = 0;
  for (int i = 0; i < 3; i++) {
    int a = tri[3 * t + i];
    for (int j = 0; j < 3; j++)
      if (a == tri[3 * n + j]) {
        if (count == 0) {
          inc0 = j;
          count = 1;
          continue;
        }
        inc1 = j;
        break;
      }
  }
  if (inc0 == -1 || inc1 == -1) return -1;
  int d = inc0 - inc1;
  int idx = (d == -1 || d == 2) ? inc0 : inc1;
  return idx == 0 ? 2 : (idx == 1 ? 0 : 1);
}

// Input index check, run before anything dereferences the input: vertices in
// [0, np), neighbours in [-1, nt), segment endpoints in [0, np) and distinct,
// coordinates finite.  The reference trusts its input; a bad index here would
// make the initialisation read outside the input arrays.
GQM_KERNEL void k_check_input(const double2 *pts, int np, const int *tri, const int *nbr, int nt,
                              const int *seg, int ns, int *err) {
  int bad = 0;
  GS_LOOP(i, np) {
    double2 p = pts[i];
    if (!isfinite(p.x) || !isfinite(p.y)) bad = 1;
  }
  GS_LOOP(t, nt) {
    for (int k = 0; k < 3; k++) {
      unsigned v = (unsigned)tri[3 * t + k];
      int n = nbr[3 * t + k];
      if (v >= (unsigned)np || n < -1 || n >= nt) bad = 1;
    }
  }
  GS_LOOP(s, ns) {
    unsigned a = (unsigned)seg[2 * s], b = (unsigned)seg[2 * s + 1];
    if (a >= (unsigned)np || b >= (unsigned)np || a == b) bad = 1;
  }
  if (bad) atomicCAS(err, 0, GQM_ERR_ARGUMENT);
}

// free slots
__device__ __forceinline__ void clear_point(const Mesh &M, int i) {
  M.pts[i] = make_double2(0.0, 0.0);
  M.ps[i] = PS_DELETED;
  M.pred[i] = 0;
}
__device__ __forceinline__ void clear_tri_flags(const Mesh &M, int t) {
  M.tsg[t] = make_int4(-1, -1, -1, 0);
  M.tflip[t] = 0;
  M.tfo[t] = 0;
  M.tmark[t] = 0;
}
__device__ __forceinline__ void clear_tri(const Mesh &M, int t) {
  M.tv[t] = make_int4(0, 0, 0, 0);
  M.tn[t] = make_int4(0, 0, 0, 0);
  M.tst[t] = 0;
  clear_tri_flags(M, t);
}

GQM_KERNEL void k_init_tris(Mesh M, const int *tri, const int *nbr, int nt, int tcap) {
  GS_LOOP(t, tcap) {
    if (t < nt) {
      M.tv[t] = make_int4(tri[3 * t], tri[3 * t + 1], tri[3 * t + 2], 0);
      int4 nb;
      nb.x = etri(nbr[3 * t], incident_ori(tri, t, nbr[3 * t]));
      nb.y = etri(nbr[3 * t + 1], incident_ori(tri, t, nbr[3 * t + 1]));
      nb.z = etri(nbr[3 * t + 2], incident_ori(tri, t, nbr[3 * t + 2]));
      nb.w = 0;
      M.tn[t] = nb;
      M.tst[t] = TS_NOTNULL | TS_CHECK;
      clear_tri_flags(M, t);
    } else {
      clear_tri(M, t);
    }
  }
}

GQM_KERNEL void k_init_points(Mesh M, const double2 *pts, int np, int pcap) {
  GS_LOOP(i, pcap) {
    if (i < np) {
      M.pts[i] = pts[i];
      M.ps[i] = 0;
      M.pred[i] = 0;
    } else {
      clear_point(M, i);
    }
  }
}

// cos^2(theta) exactly as the reference evaluates it on the device
// (refine.cu:418, 123-124).
#define GQM_PI 3.141592653589793238462643383279502884197169399375105820974944592308
GQM_KERNEL void k_goodcos(double theta, double *out) {
  if (threadIdx.x == 0 && GQM_BLOCK0) {
    double c = cos(theta * GQM_PI / 180.0);
    out[0] = c * c;
    out[1] = cos(theta * GQM_PI / 180.0) * cos(theta * GQM_PI / 180.0);
  }
}

__device__ __forceinline__ unsigned long long seg_key(int a, int b) {
  unsigned lo = (unsigned)min(a, b), hi = (unsigned)max(a, b);
  return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ unsigned seg_hash(unsigned long long k, unsigned mask) {
  return (unsigned)((k * 0x9E3779B97F4A7C15ull) >> 24) & mask;
}
GQM_KERNEL void k_seg_hash_insert(const int2 *segs, int ns, unsigned long long *keys, int *vals, unsigned mask) {
  GS_LOOP(s, ns) {
    unsigned long long k = seg_key(segs[s].x, segs[s].y);
    unsigned h = seg_hash(k, mask);
    for (unsigned probe = 0; probe <= mask; ++probe) {
      unsigned long long old = atomicCAS(keys + h, ~0ull, k);
      if (old == ~0ull) {
        vals[h] = s;
        break;
      }
      h = (h + 1) & mask;
    }
  }
}
// initSubsegs (refine.cu:5618-5747) for every triangle: edge (p0,p1) is
// orientation 2, (p1,p2) 0, (p2,p0) 1; subseg2tri keeps the largest otri
// (atomicMax), tri2subseg the largest matching subsegment.
GQM_KERNEL void k_init_subsegs(Mesh M, int nt, const unsigned long long *keys, const int *vals, unsigned mask,
                               int *s2t_int) {
  GS_LOOP(t, nt) {
    int4 v = M.tv[t];
    int4 sg = make_int4(-1, -1, -1, 0);
    const int eu[3] = {v.x, v.y, v.z}, ew[3] = {v.y, v.z, v.x}, eo[3] = {2, 0, 1};
    for (int e = 0; e < 3; ++e) {
      unsigned long long k = seg_key(eu[e], ew[e]);
      unsigned h = seg_hash(k, mask);
      for (unsigned probe = 0; probe <= mask; ++probe) {
        unsigned long long kk = keys[h];
        if (kk == ~0ull) break;
        if (kk == k) {
          int s = vals[h];
          atomicMax(s2t_int + s, (t << 2) | eo[e]);
          if (s > comp(sg, eo[e])) setc(sg, eo[e], s);
        }
        h = (h + 1) & mask;
      }
    }
    M.tsg[t] = sg;
  }
}
GQM_KERNEL void k_pack_s2t(Mesh M, const int *s2t_int, int ns) {
  GS_LOOP(s, ns) {
    M.s2t[s] = s2t_plain(s2t_int[s]);
    M.s2seg[s] = s;
  }
}

// kernelMarkAllEncsegs, refine.cu:3105-3151
template <class N>
GQM_KERNEL void k_mark_all_encsegs(Mesh M, N ns_) {
  const int ns = nval(ns_);
  GS_LOOP(s, ns) {
    int e = -1;
    int otri = s2t_get(M, s);
    if (otri >= 0) {
      int t = dtri(otri), o = dori(otri);
      int4 v = M.tv[t];
      double2 vo = M.pts[comp(v, m3(o + 1))], vd = M.pts[comp(v, m3(o + 2))], va = M.pts[comp(v, o)];
      if (encroached(vo, vd, va, M.gc2, M.mode)) e = 0;
      int on = ld1(M.tn, t, o);
      if (on != -1) {
        double2 vb = M.pts[ld1(M.tv, dtri(on), dori(on))];
        if (encroached(vd, vo, vb, M.gc2, M.mode)) e = 0;
      }
    }
    M.enc[s] = e;
  }
}

// ============================================================================
// Bad triangles (refine.cu:317-497)
// ============================================================================
// kernelComputeSmallestAngle, refine.cu:317-374: cos^2 of the smallest angle
__device__ __forceinline__ double smallest_cos2(double2 pA, double2 pO, double2 pD, int *shortest) {
  double dxod = pO.x - pD.x, dyod = pO.y - pD.y;
  double dxda = pD.x - pA.x, dyda = pD.y - pA.y;
  double dxao = pA.x - pO.x, dyao = pA.y - pO.y;
  // gqm_madd: the products the reference's contracted build fuses (see
  // predicates.h); the sums are the same in either order
  double lenOrg = gqm_madd(dyod, dyod, dxod * dxod);
  double lenDest = gqm_madd(dyda, dyda, dxda * dxda);
  double lenApex = gqm_madd(dxao, dxao, dyao * dyao);
  double ang, sh;
  if (lenOrg < lenDest && lenOrg < lenApex) {
    sh = lenOrg;
    *shortest = 0;
    ang = gqm_madd(dyda, dyao, dxda * dxao);
  } else if (lenDest < lenOrg && lenDest < lenApex) {
    sh = lenDest;
    *shortest = 1;
    ang = gqm_madd(dyod, dyao, dxod * dxao);
  } else {
    sh = lenApex;
    *shortest = 2;
    ang = gqm_madd(dyod, dyda, dxod * dxda);
  }
  return ang * ang * sh / (lenOrg * lenDest * lenApex);
}

// kernelMarkBadTriangles, refine.cu:376-497, over every triangle slot below
// ntri that is not null and has CHECK set.
template <class N>
GQM_KERNEL void k_mark_bad(Mesh M, N ntri_) {
  const int ntri = nval(ntri_);
  GS_LOOP(t, ntri) {
    uint8_t st = M.tst[t];
    if (!(st & TS_NOTNULL) || !(st & TS_CHECK)) continue;
    st = (uint8_t)((st & ~TS_CHECK) | TS_NOTNULL);
    int4 v = M.tv[t];
    double2 a = M.pts[v.x], b = M.pts[v.y], c = M.pts[v.z];
    int sh;
    double c2 = smallest_cos2(a, b, c, &sh);
    bool bad = true;
    if (c2 <= M.gc2) {
      bad = false;
    } else if (ld1(M.tsg, t, sh) == -1) {
      int eOrg = comp(v, m3(sh + 1)), eDest = comp(v, m3(sh + 2));
      if ((M.ps[eOrg] & PS_SEGSPLIT) && (M.ps[eDest] & PS_SEGSPLIT)) {
        int s1 = -1, s2 = -1;
        int cur = t, ori = sh, guard = 0;
        do {
          int o = ld1(M.tn, cur, ori);
          cur = dtri(o);
          ori = m3(dori(o) + 1);
          if (cur < 0 || ++guard > (1 << 20)) break;
          s1 = ld1(M.tsg, cur, ori);
        } while (s1 == -1);
        cur = t;
        ori = sh;
        guard = 0;
        do {
          int o = ld1(M.tn, cur, ori);
          cur = dtri(o);
          ori = m3(dori(o) + 2);
          if (cur < 0 || ++guard > (1 << 20)) break;
          s2 = ld1(M.tsg, cur, ori);
        } while (s2 == -1);
        if (s1 < 0 || s2 < 0) {
          raise_err(M, -5);
        } else {
          int2 g1 = M.segs[M.s2seg[s1]], g2 = M.segs[M.s2seg[s2]];
          int common = -1;
          if (g1.x == g2.x || g1.x == g2.y)
            common = g1.x;
          else if (g1.y == g2.x || g1.y == g2.y)
            common = g1.y;
          if (common != -1) {
            double2 vo = (sh == 0) ? b : (sh == 1 ? c : a);
            double2 vd = (sh == 0) ? c : (sh == 1 ? a : b);
            double2 vc = M.pts[common];
            double d1 = gqm_madd(vc.x - vo.x, vc.x - vo.x, (vc.y - vo.y) * (vc.y - vo.y));
            double d2 = gqm_madd(vc.x - vd.x, vc.x - vd.x, (vc.y - vd.y) * (vc.y - vd.y));
            if ((d1 < 1.001 * d2) && (d1 > 0.999 * d2)) bad = false;
          }
        }
      }
    }
    // area bound (no counterpart in the reference; Triangle's `a` switch)
    if (!bad && M.max_area > 0.0 &&
        0.5 * fabs((b.x - a.x) * (c.y - a.y) - (b.y - a.y) * (c.x - a.x)) > M.max_area)
      bad = true;
    M.tst[t] = bad ? (uint8_t)(st | TS_BAD) : (uint8_t)(st & ~TS_BAD);
  }
}

// ============================================================================
// Flip-flop (refine.cu:580-2490)
// ============================================================================
__device__ __forceinline__ bool is_red(const Mesh &M, int p) { return M.pred[p] != 0; }

// Generations that a loop (or a run's reset) advances by: the pushes for the
// next loop carry its generation, and the claims that splitTriangles makes
// before it carry the two before that.
constexpr int kGenStride = 4, kGenLocate = 3, kGenCavity = 2;
// Control block of the flip-flop loops, resident on the device.
constexpr int kFlipProfileBins = 32;
// List lengths of a flip step, indexed by the parity of the step's generation.
struct FlipCnt {
  int qn[2];     // triangles pushed for the next step
  int live[2];   // flagged live triangles the step checked
  int nred[2];   // triangles whose claim may name a redundant point
  int nlate[2];  // subseg2tri stores that another winner competes with
};
// What a run of small steps leaves for the team's other blocks.
struct FlipOut {
  FlipCnt cnt;
  int gen, steps, status;  // status: how the run ended (FLIP_*)
  unsigned epoch;
};
struct FlipCtl {
  int gen;         // generation of the pushes between loops (stamps, claims)
  unsigned epoch;  // launch epoch of the subseg2tri stores (all kernels share it)
  FlipCnt cnt;
  FlipOut out[2];  // by turns, see flip_loop
  int steps;        // flip steps executed (all loops)
  int small_steps;  // of which steps run by the small-step team
  int cap_hit;      // the step bound stopped a loop
  int ran;          // loops run since the reset
  long long cap;    // bound on the steps of one loop
  int *errp;        // device error word (GQM_ERR_ROUND_LIMIT on cap_hit)
  // device time of the loops (%globaltimer from loop entry to loop end)
  unsigned long long loop_ns, loops;
  // step profile of the run: steps and active triangles by floor(log2 |A|)
  unsigned long long prof_steps[kFlipProfileBins], prof_items[kFlipProfileBins];
};
// The loop's lists.  q0 / q1: the triangles flagged for a step, by the parity
// of the generation that pushed them; rec: the step's decision for each entry
// of its queue (see flip_check); red, late: see FlipCnt; wbits, wcnt, wsup: the
// winners of a large step, as a bitmap over the tcap triangle slots and counts
// per 2^10 and 2^15 slots (see winner_rank).
struct FlipLists {
  int *q0, *q1;
  int4 *rec;
  int *red;
  int4 *late;
  unsigned *wbits;
  int *wcnt, *wsup;
  int tcap;
  FlipCtl *c;
};
// words of wbits, wcnt and wsup, which lie one after another
__host__ __device__ inline size_t winner_words(long tcap) {
  return (size_t)(tcap / 1024 + 1) * 32 + (size_t)(tcap / 1024 + 1) + (size_t)(tcap / 32768 + 1);
}
__host__ __device__ inline void winner_carve(FlipLists &L, unsigned *words, long tcap) {
  L.wbits = words;
  L.wcnt = reinterpret_cast<int *>(words) + (tcap / 1024 + 1) * 32;
  L.wsup = L.wcnt + (tcap / 1024 + 1);
  L.tcap = (int)tcap;
}
// Queues of at most this many entries are scanned for a winner's position; the
// winners of a longer one are marked in the bitmap.  A scan reads 16 bytes an
// entry for every store to be ordered, the bitmap costs every winner three
// reductions and the step a clearing pass.  With the scan alone the late phase
// of the largest steps (hundreds of such stores, 300,000 entries) took
// milliseconds, 880 ms of a refinement of 2,000,000 points; with the bitmap 4 ms.
constexpr int kScanRank = 2048;
// A queue being filled: its entries, its length, the generation of its stamps.
struct FlipQ {
  int *q;
  int *qn;
  int gen;
};
// the queue that the kernels between two flip loops push to
__device__ __forceinline__ FlipQ entry_queue(const FlipLists &L) {
  const int g = L.c->gen;
  return FlipQ{(g & 1) ? L.q1 : L.q0, &L.c->cnt.qn[g & 1], g};
}
// Flags a triangle for the next step; the generation stamp keeps it from
// being queued twice.
__device__ __forceinline__ void push_flag(const Mesh &M, const FlipQ &Q, int t) {
  M.tflip[t] = 1;
  if (atomicExch(M.fstamp + t, Q.gen) != Q.gen) Q.q[list_slot(Q.qn)] = t;
}
// The same where no other thread can push t at the same time.
__device__ __forceinline__ void push_owned(const Mesh &M, const FlipQ &Q, int t) {
  if (M.fstamp[t] == Q.gen) return;  // queued, its flag set
  M.tflip[t] = 1;
  M.fstamp[t] = Q.gen;
  Q.q[list_slot(Q.qn)] = t;
}

// markFan, refine.cu:580-602.  The walk (one dependent load a triangle) runs
// ahead of the pushes, eight triangles at a time, so that the stamps of a
// group are exchanged together.
__device__ void mark_fan(const Mesh &M, const FlipQ &Q, int triIndex, int triOri) {
  int cur = triIndex, ori = triOri, guard = 0;
  bool more = true;
  while (more) {
    int fan[8], n = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      fan[j] = -1;
      if (!more) continue;
      fan[j] = cur;
      int nx = ld1(M.tn, cur, m3(ori + 2));
      cur = dtri(nx);
      ori = dori(nx);
      ++n;
      more = cur > -1 && cur != triIndex;
    }
    int old[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (fan[j] >= 0) {
        M.tflip[fan[j]] = 1;
        old[j] = atomicExch(M.fstamp + fan[j], Q.gen);
      }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (fan[j] >= 0 && old[j] != Q.gen) Q.q[list_slot(Q.qn)] = fan[j];
    if ((guard += n) > (1 << 20)) {
      raise_err(M, -4);
      return;
    }
  }
}

// resetEncseg, refine.cu:1879-1922
__device__ void reset_encseg(const Mesh &M, int s, int otri0, int otri1) {
  int e = -1;
  if (otri0 != -1) {
    int t = dtri(otri0), o = dori(otri0);
    int4 v = M.tv[t];
    if (encroached(M.pts[comp(v, m3(o + 1))], M.pts[comp(v, m3(o + 2))], M.pts[comp(v, o)], M.gc2, M.mode)) e = 0;
  }
  if (otri1 != -1) {
    int t = dtri(otri1), o = dori(otri1);
    int4 v = M.tv[t];
    if (encroached(M.pts[comp(v, m3(o + 1))], M.pts[comp(v, m3(o + 2))], M.pts[comp(v, o)], M.gc2, M.mode)) e = 0;
  }
  M.enc[s] = e;
}

// kernelMarkReduantPoints, refine.cu:604-677
GQM_KERNEL void k_mark_redundant(Mesh M, int *delmarker, const int *dellist, const int *dn, FlipLists L) {
  int n = *dn;
  const FlipQ Q = entry_queue(L);
  GS_LOOP(pos, n) {
    int out = -1;
    int sindex = dellist[pos];
    int otri = s2t_get(M, sindex);
    int t = dtri(otri), o = dori(otri);
    int4 v = M.tv[t];
    int pApex = comp(v, o);
    double2 vO = M.pts[comp(v, m3(o + 1))], vD = M.pts[comp(v, m3(o + 2))], vA = M.pts[pApex];
    uint8_t s = M.ps[pApex];
    if ((s & PS_STEINER) && !(s & PS_SEGSPLIT) &&
        ((vO.x - vA.x) * (vD.x - vA.x) + (vO.y - vA.y) * (vD.y - vA.y) < 0.0)) {
      M.pred[pApex] = 1;
      mark_fan(M, Q, t, m3(o + 2));
      out = sindex;
    }
    int on = ld1(M.tn, t, o);
    if (on != -1) {
      t = dtri(on);
      o = dori(on);
      pApex = ld1(M.tv, t, o);
      vA = M.pts[pApex];
      s = M.ps[pApex];
      if ((s & PS_STEINER) && !(s & PS_SEGSPLIT) &&
          ((vO.x - vA.x) * (vD.x - vA.x) + (vO.y - vA.y) * (vD.y - vA.y) < 0.0)) {
        M.pred[pApex] = 1;
        mark_fan(M, Q, t, m3(o + 2));
        out = sindex;
      }
    }
    delmarker[pos] = out;
  }
}

// Timer of one phase of the device-side loop, where CUDA events cannot
// bracket single phases (%globaltimer stamps by the lead thread).
struct KTimer {
  unsigned long long total_ns, launches, items;
  unsigned long long winners;  // flips and flops applied (small steps)
  unsigned long long first_items[4];  // items of the first four phases since the reset
  int on;
};
__device__ __forceinline__ unsigned long long global_ns() {
#ifdef GQM_HOST_EMU
  return (unsigned long long)std::chrono::duration_cast<std::chrono::nanoseconds>(
             std::chrono::steady_clock::now().time_since_epoch())
      .count();
#else
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
#endif
}
__device__ __forceinline__ void ktimer_add(KTimer *tm, unsigned long long start, long long items,
                                           long long winners = 0) {
  tm->total_ns += global_ns() - start;
  if (tm->launches < 4) tm->first_items[tm->launches] = (unsigned long long)items;
  tm->launches += 1;
  tm->items += (unsigned long long)items;
  tm->winners += (unsigned long long)winners;
}
GQM_KERNEL void k_ktimer_reset(KTimer *tm, int on) {
  if (GQM_BLOCK0 && threadIdx.x == 0) {
    tm->total_ns = tm->launches = tm->items = tm->winners = 0;
    for (int i = 0; i < 4; ++i) tm->first_items[i] = 0;
    tm->on = on;
  }
}
GQM_KERNEL void k_bump_epoch(FlipCtl *c) {
  if (GQM_BLOCK0 && threadIdx.x == 0) c->epoch++;
}
// per-run reset of the control block; gen and epoch keep growing across runs
// so that stamps, claims and subseg2tri tags left by earlier runs never collide
__device__ __forceinline__ void ctl_reset(FlipCtl *c, long long cap, int *errp, bool lead) {
  if (!lead) return;
  for (int b = 0; b < kFlipProfileBins; ++b) c->prof_steps[b] = c->prof_items[b] = 0;
  c->cnt = FlipCnt{};
  c->gen += kGenStride;
  c->steps = 0;
  c->small_steps = 0;
  c->cap_hit = 0;
  c->ran = 0;
  c->cap = cap;
  c->errp = errp;
}
GQM_KERNEL void k_ctl_reset(FlipCtl *c, long long cap, int *errp) {
  ctl_reset(c, cap, errp, GQM_BLOCK0 && threadIdx.x == 0);
}

// ---------------------------------------------------------------------------
// The flip steps (refine.cu:2328-2490), on active sets.
//
// The reference rescans every triangle slot several times per step and links
// the flipped triangles to their neighbours in three passes.  Here a step is
// three phases over its queue, separated by barriers, and each waits for two
// or three dependent loads:
//   check   every flagged triangle decides its flip and claims the triangles
//           it needs (flip_check);
//   apply   a triangle that won all its claims rewrites them at once, its
//           outer links still naming the neighbours' old edges, and leaves an
//           edge map in every triangle it rewrote or removed: where each old
//           outer edge went (flip_apply);
//   fix     it looks each outer neighbour up: one rewritten in the same step
//           is followed through its map, any other is pointed back here
//           (flip_fix).
// A fourth phase runs only in the steps that need it (flip_late): points that
// become redundant, and stores into subseg2tri from both sides of a subsegment.
//
// Claims are 64-bit words (complement of the step's generation, claimed
// value): a claim of an earlier step is larger than any of this one, so
// nothing is reset between steps and no list of claimed triangles is kept.
// Every triangle flagged between two loops was pushed where it was flagged,
// so a loop starts from a queue and not from a pass over all triangles.
// Bound by the latency of those dependent loads, in a step of any size.
// Against eight launches a step (claims reset through a list, winners
// compacted, links set up and resolved in three launches), the flip loops of a
// refinement of 2,000,000 clustered points take 48.6 ms instead of 75 ms, those
// of 10,000 uniform points 7.0 ms instead of 12.0 ms (B200).
//
// Every phase decides by the reference's rules on the data, never by the
// order of a list or by the thread layout.  The phases are functions of their
// own, so that each gets its registers and one copy serves every team.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long claim_key(int gen, int v) {
  return ((unsigned long long)(~(unsigned)gen) << 32) | ((unsigned)v ^ 0x80000000u);
}
__device__ __forceinline__ void claim(const Mesh &M, int gen, int t, int v) {
  atomicMin(M.fmark + t, claim_key(gen, v));
}
// value of this step's claim on t, kMaxInt when nobody claimed it
__device__ __forceinline__ int claimed(const Mesh &M, int gen, int t) {
  const unsigned long long w = M.fmark[t];
  return (unsigned)(w >> 32) == ~(unsigned)gen ? (int)((unsigned)w ^ 0x80000000u) : kMaxInt;
}

// Decisions in rec[k].y (rec[k].x is the triangle, .z and .w EdgeMove::link and
// third): the reference's flip orientation 0..8 (FD_OUTWARD added), or
enum : int {
  FD_CLEAR = 14,  // nothing to flip: the flag is cleared
  FD_KEEP = 15,   // no flip, the flag stays (a point is to be deleted first)
  FD_DEAD = -1,   // a queue entry whose flag or triangle is gone
  FD_WON = 16,     // added by flip_apply: all claims won
  FD_OUTWARD = 32  // added to a 4-2 flip that removes the edge's origin
};

// What one edge of a flagged triangle asks for in kernelCheckFlipping
// (refine.cu:778-1070): code -1 for nothing, else the decision, and the
// triangles to claim besides the triangle itself and its neighbour across the
// edge (-1: none).
struct EdgeMove {
  int code, n1, n2;
  int link, third;  // links of the triangle that the flip runs over: 2-2 and 4-2 the one across the
                    // edge, 4-2 the one at the point that goes; 3-1 those at ori and ori + 2
  int value;  // claimed value
  bool across;  // the neighbour across the edge is claimed too
};
// The four incircle tests of an edge O-D facing A and P: illegal when both
// triangles' circles hold the other's vertex and neither would after the flip.
// The four filters come first and one call decides what they leave open: four
// calls, each with the arguments of the others alive, cost a third of the
// check's registers.
template <int PRED>
__device__ __noinline__ bool illegal_edge_slow(double2 vA, double2 vO, double2 vD, double2 vP) {
  const double ret = incircle<PRED>(vA, vO, vD, vP), ret_opp = incircle<PRED>(vO, vP, vD, vA);
  const double ret_after = incircle<PRED>(vA, vO, vP, vD), ret_after_opp = incircle<PRED>(vP, vD, vA, vO);
  return ret > 0 && ret_opp > 0 && ret_after < 0 && ret_after_opp < 0;
}
template <int PRED>
__device__ __forceinline__ bool illegal_edge(double2 vA, double2 vO, double2 vD, double2 vP) {
  bool open = false;
  const double ret = incircle_fast<PRED>(vA, vO, vD, vP, &open), ret_opp = incircle_fast<PRED>(vO, vP, vD, vA, &open);
  const double ret_after = incircle_fast<PRED>(vA, vO, vP, vD, &open);
  const double ret_after_opp = incircle_fast<PRED>(vP, vD, vA, vO, &open);
  if (open) return illegal_edge_slow<PRED>(vA, vO, vD, vP);
  return ret > 0 && ret_opp > 0 && ret_after < 0 && ret_after_opp < 0;
}
// No flag is cleared during the check, so the neighbour flags read are the ones
// the step started with.  p, nb, sg: the triangle's rows.
template <int PRED>
__device__ __forceinline__ EdgeMove edge_move(const Mesh &M, int index, const int4 &p, const int4 &nb, const int4 &sg,
                                              int e) {
  EdgeMove mv{-1, -1, -1, comp(nb, e), -1, index, true};
  const int iA = comp(p, e), iO = comp(p, m3(e + 1)), iD = comp(p, m3(e + 2));
  const int link = comp(nb, e), pTri = dtri(link), pOri = dori(link);
  const bool use = comp(sg, e) == -1 && pTri >= 0;
  // one level of loads: the points and flags of the triangle, the neighbour's flag and vertex
  const double2 vA = M.pts[iA], vO = M.pts[iO], vD = M.pts[iD];
  const bool rA = is_red(M, iA), rO = is_red(M, iO), rD = is_red(M, iD);
  const uint8_t flag = (use && pTri < index) ? M.tflip[pTri] : 0;
  const int pOpp = use ? ld1(M.tv, pTri, pOri) : -1;
  // the next: the facing vertex
  const bool rP = use && is_red(M, pOpp);
  const double2 vP = use ? M.pts[pOpp] : vA;
  int mn = kMaxInt;
  if (rA) mn = iA;
  if (rO && iO < mn) mn = iO;
  if (rD && iD < mn) mn = iD;
  if (mn == iA || !use || !(index < pTri || !flag) || (rP && pOpp < mn)) return mv;
  if (mn != kMaxInt) {
    const bool org = mn == iO;
    const int n1 = org ? comp(nb, m3(e + 2)) : comp(nb, m3(e + 1));
    const int n2 = ld1(M.tn, pTri, org ? m3(pOri + 1) : m3(pOri + 2));
    if (dtri(n1) == dtri(n2)) {  // 3-1 flip
      mv.code = 3 + (org ? m3(e + 2) : e);
      mv.n1 = dtri(n1);
      mv.link = org ? link : n1;
      mv.third = org ? n1 : link;
      return mv;
    }
    const int n1_tri = dtri(n1), n1_ori = dori(n1), n2_tri = dtri(n2), n2_ori = dori(n2);
    const int n3 = ld1(M.tn, n1_tri, org ? m3(n1_ori + 2) : m3(n1_ori + 1));
    if (dtri(n3) == n2_tri) {
      const int n1_pOpp = ld1(M.tv, n1_tri, n1_ori), n2_pOpp = ld1(M.tv, n2_tri, n2_ori);
      const double2 v1 = M.pts[n1_pOpp], v2 = M.pts[n2_pOpp];
      bool four = false;
      if (org) {
        if (orient<PRED>(vA, vO, vP) == 0) {
          const bool f0 = orient<PRED>(vD, vA, v1) > 0 && orient<PRED>(vD, vO, v1) < 0;
          const bool f1 = orient<PRED>(vD, vO, v2) > 0 && orient<PRED>(vD, vP, v2) < 0;
          four = !f0 && !f1;
        }
      } else {
        if (orient<PRED>(vA, vD, vP) == 0) {
          const bool f0 = orient<PRED>(vO, vD, v1) > 0 && orient<PRED>(vO, vA, v1) < 0;
          const bool f1 = orient<PRED>(vO, vP, v2) > 0 && orient<PRED>(vO, vD, v2) < 0;
          four = !f0 && !f1;
        }
      }
      if (four) {
        if (is_red(M, n1_pOpp) && n1_pOpp < mn) return mv;
        mv.code = (6 + e) | (org ? FD_OUTWARD : 0);
        mv.third = n1;
        mv.n1 = n1_tri;
        mv.n2 = n2_tri;
        return mv;
      }
    }
    if (orient<PRED>(vA, vO, vP) <= 0 || orient<PRED>(vA, vD, vP) >= 0) return mv;
    mv.code = m3(e + 2);
    return mv;
  }
  if (!illegal_edge<PRED>(vA, vO, vD, vP)) return mv;
  const uint8_t sa = M.ps[iA], so = M.ps[pOpp];
  mv.code = m3(e + 2);
  if ((sa & PS_NEW) && (so & PS_NEW) && !((sa & PS_SEGSPLIT) && (so & PS_SEGSPLIT))) {
    // one of two new points is deleted instead: the claim names it
    const bool second = (sa & PS_SEGSPLIT) ? true : (so & PS_SEGSPLIT) ? false : iA < pOpp;
    mv.code = FD_KEEP;
    mv.across = second;
    mv.value = second ? negate_idx(etri(pTri, m3(pOri + 2))) : negate_idx(etri(index, m3(e + 2)));
  }
  return mv;
}
// The claims of the triangle's decision, the first move in edge order.
__device__ __forceinline__ void make_claims(const Mesh &M, int gen, int index, int pTri, const EdgeMove &mv, int *red,
                                            int *nred) {
  claim(M, gen, index, mv.value);
  if (mv.across) claim(M, gen, pTri, mv.value);
  if (mv.n1 >= 0) claim(M, gen, mv.n1, mv.value);
  if (mv.n2 >= 0) claim(M, gen, mv.n2, mv.value);
  if (mv.code == FD_KEEP) {
    const int at = list_slot2(nred);
    red[at] = index;
    red[at + 1] = mv.across ? pTri : index;
  }
}
#ifndef GQM_HOST_EMU
// Phase 1 with one thread per triangle, its edges in turn: for steps that fill
// the team's threads (see flip_check).
template <int PRED>
__device__ __noinline__ void flip_check_many(const Mesh &M, const int *q, int n, int gen, const FlipLists &L, int4 *rec,
                                             int *live, int *nred, int tid, int size) {
  const int lane = (int)(threadIdx.x & 31u);
#pragma unroll 1
  for (int base = tid - lane; base < n; base += size) {  // whole warps
    const int k = base + lane;
    bool act = false;
    if (k < n) {
      const int index = q[k];
      const uint8_t flag = M.tflip[index], st = M.tst[index];
      const int4 p = M.tv[index], nb = M.tn[index], sg = M.tsg[index];
      act = flag && (st & TS_NOTNULL);
      int4 r = make_int4(index, act ? (int)FD_CLEAR : (int)FD_DEAD, -1, -1);
      if (act) {
#pragma unroll 1
        for (int e = 0; e < 3; ++e) {
          const EdgeMove mv = edge_move<PRED>(M, index, p, nb, sg, e);
          if (mv.code < 0) continue;
          r.y = mv.code;
          r.z = mv.link;
          r.w = mv.third;
          make_claims(M, gen, index, dtri(comp(nb, e)), mv, L.red, nred);
          break;
        }
      }
      rec[k] = r;
    }
    const unsigned b = __ballot_sync(0xffffffffu, act);
    if (lane == 0 && b) atomicAdd(live, __popc(b));
  }
}
#endif
// Phase 1: the queue entries whose flag is still set on a live triangle (the
// step's active set) decide; *live counts them.  tid / size: the thread's
// place in the team that runs the step.
//
// Four lanes take one triangle, the first three an edge each.  The reference
// tries the edges in turn and stops at the first that asks for something; no
// edge's test changes anything another reads, so they are tested together and
// the first one's outcome is taken.  With one thread per triangle the three
// edges, each in any of four ways through its test, ran one after another in
// every warp: the check of a step of about 50 triangles took 5.6 us instead of
// 3.6 us; two of three steps are small.
template <int PRED>
__device__ __noinline__ void flip_check(const Mesh &M, const int *q, int n, int gen, const FlipLists &L, int4 *rec,
                                        int *live, int *nred, int tid, int size) {
  if (n > kScanRank) {  // a clean bitmap for this step's winners
    const long words = (long)winner_words(L.tcap);
    for (long i = tid; i < words; i += size) L.wbits[i] = 0u;
  }
#ifdef GQM_HOST_EMU
  for (int k = tid; k < n; k += size) {
    const int index = q[k];
    const int4 p = M.tv[index], nb = M.tn[index], sg = M.tsg[index];
    int4 r = make_int4(index, FD_DEAD, -1, 0);
    if (M.tflip[index] && (M.tst[index] & TS_NOTNULL)) {
      ++*live;
      r.y = FD_CLEAR;
      for (int e = 0; e < 3; ++e) {
        const EdgeMove mv = edge_move<PRED>(M, index, p, nb, sg, e);
        if (mv.code < 0) continue;
        r.y = mv.code;
        r.z = mv.link;
        r.w = mv.third;
        make_claims(M, gen, index, dtri(comp(nb, e)), mv, L.red, nred);
        break;
      }
    }
    rec[k] = r;
  }
#else
  // More than two triangles for every four threads: the lanes' repeated loads
  // cost more than the edges one after another (the check phases of the steps
  // by all blocks of a 2,000,000-point refinement: 17.6 ms with four lanes
  // throughout, 12.7 ms with this rule; of a 10,000-point one 0.70 ms both ways).
  if (n > size / 2) return flip_check_many<PRED>(M, q, n, gen, L, rec, live, nred, tid, size);
  const int lane = (int)(threadIdx.x & 31u), e = lane & 3, first = lane & 28;
  const int items = size >> 2;
#pragma unroll 1
  for (int base = (tid - lane) >> 2; base < n; base += items) {  // whole warps
    const int k = base + (lane >> 2);
    int index = -1, link = -1;
    bool act = false;
    EdgeMove mv{-1, -1, -1, -1, -1, 0, false};
    if (k < n) {
      index = q[k];
      const uint8_t flag = M.tflip[index], st = M.tst[index];
      const int4 p = M.tv[index], nb = M.tn[index], sg = M.tsg[index];
      act = flag && (st & TS_NOTNULL);
      if (act && e < 3) {
        link = comp(nb, e);
        mv = edge_move<PRED>(M, index, p, nb, sg, e);
      }
    }
    const unsigned moves = (__ballot_sync(0xffffffffu, mv.code >= 0) >> first) & 7u;
    if (moves ? (int)(__ffs(moves) - 1) == e : (e == 0 && k < n)) {
      rec[k] = make_int4(index, moves ? mv.code : (act ? (int)FD_CLEAR : (int)FD_DEAD), mv.link, mv.third);
      if (moves) make_claims(M, gen, index, dtri(link), mv, L.red, nred);
    }
    const unsigned b = __ballot_sync(0xffffffffu, act && e == 0);
    if (lane == 0 && b) atomicAdd(live, __popc(b));
  }
#endif
}

__device__ __forceinline__ int4 tri_row(int a, int b, int c, int ori) {  // a, b on edge ori, c facing it
  int4 v;
  setc(v, m3(ori + 1), a);
  setc(v, m3(ori + 2), b);
  setc(v, ori, c);
  v.w = 0;
  return v;
}
// a row with x at ori, y at ori + 1, z at ori + 2
__device__ __forceinline__ int4 ori_row(int x, int y, int z, int ori, int w = 0) {
  int4 v;
  setc(v, ori, x);
  setc(v, m3(ori + 1), y);
  setc(v, m3(ori + 2), z);
  v.w = w;
  return v;
}

// A point leaves the mesh: its byte shares a word with other points' that may
// leave in the same phase; nobody waits for the answer.
__device__ __forceinline__ void delete_point(const Mesh &M, int p) {
  atomicOr(reinterpret_cast<unsigned *>(M.ps + (p & ~3)), (unsigned)PS_DELETED << ((p & 3) * 8));
}
// The winner test of kernelMarkFlipWinner (refine.cu:1072-1170) and, for a
// winner, kernelInitLinklist and kernelUpdatePhase1 (1172-1552): the triangles
// it owns get their new vertices and subsegments, their links still naming the
// outer neighbours' old edges.  Returns the decision, FD_WON added for a winner.
// The check has named every triangle but one of the 4-2 flip and the edges they
// share, so the claims and the single words that the new rows are made of are
// loaded together, before any triangle is known to be owned: a row that another
// winner is rewriting is not used.
// One function for each kind of flip: together they took more registers than
// the launch has (1,140 bytes of spills, and 6.0 us instead of 3.0 us for the
// phase in a small step of the 2,000,000-point refinement).
__device__ __noinline__ int apply_31(const Mesh &M, int gen, int4 r) {
  const int index = r.x, code = r.y & 15, c0 = claimed(M, gen, index);
  if (r.z < 0 || r.w < 0) {  // a redundant point on the boundary: no such flip, and none in the steps to come
    raise_err(M, -5);
    M.tflip[index] = 0;
    return r.y;
  }
  // 3-1 with the triangles across ori (r.z) and ori + 2 (r.w)
  const int ori = m3(code - 3 + 1), o1 = m3(ori + 1), o2 = m3(ori + 2);
  const int t1 = dtri(r.z), t2 = dtri(r.w), a = dori(r.z), b = dori(r.w), a2 = m3(a + 2), b1 = m3(b + 1);
  const int c1 = claimed(M, gen, t1), c2 = claimed(M, gen, t2);
  const int gone = ld1(M.tv, index, o1), vDest = ld1(M.tv, index, o2), vApex = ld1(M.tv, index, ori);
  const int vOrg = ld1(M.tv, t1, a);
  const int n0 = ld1(M.tn, t1, a2), n1 = ld1(M.tn, index, o1), n2 = ld1(M.tn, t2, b1);
  const int s0 = ld1(M.tsg, t1, a2), s1 = ld1(M.tsg, index, o1), s2 = ld1(M.tsg, t2, b1);
  const uint8_t sti = M.tst[index], st1b = M.tst[t1], st2b = M.tst[t2];
  if (c0 != index || c1 != index || c2 != index) return r.y;
  delete_point(M, gone);
  M.tv[index] = tri_row(vOrg, vDest, vApex, ori);
  M.tn[index] = ori_row(n0, n1, n2, ori);
  M.tsg[index] = ori_row(s0, s1, s2, ori);
  M.emap[index] = ori_row(-1, etri(index, o1), -1, ori, gen);
  M.emap[t1] = ori_row(-1, -1, etri(index, ori), a, gen);
  M.emap[t2] = ori_row(-1, etri(index, o2), -1, b, gen);
  M.tst[index] = (uint8_t)(sti | TS_CHECK);
  M.tst[t1] = (uint8_t)(st1b & ~TS_NOTNULL);
  M.tst[t2] = (uint8_t)(st2b & ~TS_NOTNULL);
  return r.y | FD_WON;
}
__device__ __noinline__ int apply_42(const Mesh &M, int gen, int4 r) {
  const int index = r.x, code = r.y & 15, c0 = claimed(M, gen, index);
  // 4-2 across r.z: t (r.w) is the triangle's own other neighbour at the point
  // that goes (the edge's origin, FD_OUTWARD, or its destination), t2 its
  // partner's; index and t stay.  k: the side of the outer edges.
  const bool outw = (r.y & FD_OUTWARD) != 0;
  const int ori = code - 6, p = dtri(r.z), o = dori(r.z), t = dtri(r.w), a = dori(r.w);
  const int k = outw ? 1 : 2, k2 = 3 - k;  // index keeps its edge ori + k, p brings o + k2
  const int c1 = claimed(M, gen, p), c2 = claimed(M, gen, t), e2 = ld1(M.tn, p, m3(o + k));
  const int vOrg = ld1(M.tv, index, m3(ori + 1)), vDest = ld1(M.tv, index, m3(ori + 2));
  const int vApex = ld1(M.tv, index, ori), vO = ld1(M.tv, p, o), vOpp = ld1(M.tv, t, a);
  const int n0 = ld1(M.tn, p, m3(o + k2)), nk = ld1(M.tn, index, m3(ori + k));
  const int m0 = ld1(M.tn, t, a), mk = ld1(M.tn, t, m3(a + k));
  const int s0 = ld1(M.tsg, p, m3(o + k2)), sk = ld1(M.tsg, index, m3(ori + k));
  const int sk2 = ld1(M.tsg, index, m3(ori + k2)), u0 = ld1(M.tsg, t, a), uk = ld1(M.tsg, t, m3(a + k));
  const uint8_t sti = M.tst[index], stp = M.tst[p], stt = M.tst[t];
  if (c0 != index || c1 != index || c2 != index) return r.y;
  const int t2 = dtri(e2), b = dori(e2);
  const int c3 = claimed(M, gen, t2), m2 = ld1(M.tn, t2, m3(b + k2)), u2 = ld1(M.tsg, t2, m3(b + k2));
  const uint8_t st2b = M.tst[t2];
  if (c3 != index) return r.y;
  delete_point(M, outw ? vOrg : vDest);
  M.tv[index] = outw ? tri_row(vO, vDest, vApex, ori) : tri_row(vOrg, vO, vApex, ori);
  M.tv[t] = outw ? tri_row(vO, vApex, vOpp, a) : tri_row(vApex, vO, vOpp, a);
  // rows: entry at the corner, at +k, at +k2
  M.tn[index] = outw ? ori_row(n0, nk, r.w, ori) : ori_row(n0, r.w, nk, ori);
  M.tn[t] = outw ? ori_row(m0, mk, m2, a) : ori_row(m0, m2, mk, a);
  M.tsg[index] = outw ? ori_row(s0, sk, sk2, ori) : ori_row(s0, sk2, sk, ori);
  M.tsg[t] = outw ? ori_row(u0, uk, u2, a) : ori_row(u0, u2, uk, a);
  // edge maps of the old edges: p's o + k2, index's ori + k, t's a + k, t2's b + k2
  const int ep = etri(index, ori), ei = etri(index, m3(ori + k)), et = etri(t, m3(a + k)), e4 = etri(t, m3(a + k2));
  M.emap[p] = outw ? ori_row(-1, -1, ep, o, gen) : ori_row(-1, ep, -1, o, gen);
  M.emap[index] = outw ? ori_row(-1, ei, -1, ori, gen) : ori_row(-1, -1, ei, ori, gen);
  M.emap[t] = outw ? ori_row(-1, et, -1, a, gen) : ori_row(-1, -1, et, a, gen);
  M.emap[t2] = outw ? ori_row(-1, -1, e4, b, gen) : ori_row(-1, e4, -1, b, gen);
  M.tst[index] = (uint8_t)(sti | TS_CHECK);
  M.tst[t] = (uint8_t)(stt | TS_CHECK);
  M.tst[p] = (uint8_t)(stp & ~TS_NOTNULL);
  M.tst[t2] = (uint8_t)(st2b & ~TS_NOTNULL);
  return r.y | FD_WON;
}
__device__ __noinline__ int apply_22(const Mesh &M, int gen, int4 r) {
  const int index = r.x, code = r.y, c0 = claimed(M, gen, index);
  // 2-2 across r.z
  const int p = dtri(r.z), o = dori(r.z), ori = code;
  const int o1 = m3(ori + 1), o2 = m3(ori + 2), q1 = m3(o + 1), q2 = m3(o + 2);
  const int c1 = claimed(M, gen, p);
  const int vOrg = ld1(M.tv, index, o1), vDest = ld1(M.tv, index, o2), vApex = ld1(M.tv, index, ori);
  const int vO = ld1(M.tv, p, o);
  const int n0 = ld1(M.tn, index, ori), n2 = ld1(M.tn, index, o2), n1 = ld1(M.tn, p, q1), n3 = ld1(M.tn, p, q2);
  const int s0 = ld1(M.tsg, index, ori), s2 = ld1(M.tsg, index, o2), s1 = ld1(M.tsg, p, q1), s3 = ld1(M.tsg, p, q2);
  const uint8_t sti = M.tst[index], stp = M.tst[p];
  if (c0 != index || c1 != index) return r.y;
  M.tv[index] = tri_row(vOrg, vDest, vO, ori);
  M.tv[p] = tri_row(vApex, vOrg, vO, o);
  M.tn[index] = ori_row(n0, n1, etri(p, q1), ori);
  M.tn[p] = ori_row(n2, etri(index, o2), n3, o);
  M.tsg[index] = ori_row(s0, s1, -1, ori);
  M.tsg[p] = ori_row(s2, -1, s3, o);
  M.emap[index] = ori_row(etri(index, ori), -1, etri(p, o), ori, gen);
  M.emap[p] = ori_row(-1, etri(index, o1), etri(p, q2), o, gen);
  M.tst[index] = (uint8_t)(sti | TS_CHECK);
  M.tst[p] = (uint8_t)(stp | TS_CHECK);
  return r.y | FD_WON;
}
// Phase 2: flags kept or cleared, winners applied.
__device__ __noinline__ void flip_apply(const Mesh &M, int n, const FlipQ &Q, const FlipLists &L, int4 *rec, int tid,
                                        int size) {
#pragma unroll 1
  for (int k = tid; k < n; k += size) {
    const int4 r = rec[k];
    if (r.y == FD_DEAD) continue;
    if (r.y == FD_CLEAR) {
      M.tflip[r.x] = 0;
      continue;
    }
    M.fstamp[r.x] = Q.gen;  // keeps its flag (only its own thread pushes it in this phase)
    Q.q[list_slot(Q.qn)] = r.x;
    if (r.y == FD_KEEP) continue;
    const int y = (r.y & 15) < 3 ? apply_22(M, Q.gen, r) : (r.y & 15) < 6 ? apply_31(M, Q.gen, r) : apply_42(M, Q.gen, r);
    if (!(y & FD_WON)) continue;
    rec[k].y = y;
    if (n > kScanRank) {
      atomicOr(L.wbits + (r.x >> 5), 1u << (r.x & 31));
      atomicAdd(L.wcnt + (r.x >> 10), 1);
      atomicAdd(L.wsup + (r.x >> 15), 1);
    }
  }
}

// Outer edge j (0..3) of a winner, for kernelUpdatePhase2 / 3
// (refine.cu:1598-2296): its link names the neighbour's old edge, and the
// neighbour's edge map says where that went.  The reference's store into
// subseg2tri (its phase 1, instruction `slot`) is made here when no other
// winner can store into the same entry, i.e. unless the neighbour was rewritten
// in this step.
__device__ __forceinline__ void fix_edge(const Mesh &M, const FlipQ &Q, uint32_t epoch, const FlipLists &L,
                                         const int4 &r, int j, int *nlate) {
  const int gen = Q.gen, index = r.x, code = r.y & 15;
  int t = index, e, slot;
  int in = -1, a = 0, oin = 0;  // 4-2: the inner edge that is left, at both its triangles
  if (code < 3) {
    const int p = dtri(r.z), o = dori(r.z);
    t = j < 2 ? index : p;
    e = j == 0 ? code : j == 1 ? m3(code + 1) : j == 2 ? o : m3(o + 2);
    slot = j;
    if (j == 2) push_owned(M, Q, p);
  } else if (code < 6) {
    if (j == 3) return;
    const int ori = m3(code - 3 + 1);
    e = j == 0 ? m3(ori + 1) : j == 1 ? ori : m3(ori + 2);
    slot = 4 + j;
  } else {
    const int ori = code - 6;
    const bool outw = (r.y & FD_OUTWARD) != 0;
    in = dtri(r.w);
    a = dori(r.w);
    oin = outw ? m3(ori + 2) : m3(ori + 1);
    t = j < 2 ? index : in;
    e = j == 0 ? ori : j == 1 ? (outw ? m3(ori + 1) : m3(ori + 2)) : j == 2 ? m3(a + 1) : m3(a + 2);
    slot = j == 0 ? 7 : j == 1 ? (outw ? 8 : 9) : j == 2 ? 11 : 12;
    if (j == 2) push_owned(M, Q, in);
  }
  const int old = ld1(M.tn, t, e), s = ld1(M.tsg, t, e);
  if (code >= 6 && j == 0) {  // the inner edge's own stores, in the reference's order
    const int s0 = ld1(M.tsg, index, oin), s1 = ld1(M.tsg, in, a);
    if (s0 != -1) s2t_put(M, s0, etri(index, oin), epoch);
    if (s1 != -1) s2t_put(M, s1, etri(in, a), epoch);
  }
  int nn = old;
  bool moved = false;
  if (old >= 0) {
    const int4 m = M.emap[dtri(old)];
    moved = m.w == gen;
    if (moved) {
      nn = comp(m, dori(old));
      st1(M.tn, t, e, nn);
    } else {
      st1(M.tn, dtri(old), dori(old), etri(t, e));
    }
  }
  if (s != -1) {
    if (moved)
      L.late[list_slot(nlate)] = make_int4(s, etri(t, e), index, slot);
    else
      s2t_put(M, s, etri(t, e), epoch);
    reset_encseg(M, s, etri(t, e), nn);
  }
}
// Phase 3: four lanes take one winner, an edge each.
__device__ __noinline__ void flip_fix(const Mesh &M, int n, const FlipQ &Q, uint32_t epoch, const FlipLists &L,
                                      const int4 *rec, int *nlate, int tid, int size) {
#ifdef GQM_HOST_EMU
  for (int k = tid; k < n; k += size)
    if (rec[k].y >= 0 && (rec[k].y & FD_WON))
      for (int j = 0; j < 4; ++j) fix_edge(M, Q, epoch, L, rec[k], j, nlate);
#else
#pragma unroll 1
  for (int k = tid >> 2; k < n; k += size >> 2) {
    const int4 r = rec[k];
    if (r.y >= 0 && (r.y & FD_WON)) fix_edge(M, Q, epoch, L, r, (int)(threadIdx.x & 3u), nlate);
  }
#endif
}

// Number of this step's winners with a smaller index, by a whole warp (lane of
// lanes); the sum is valid in lane 0.
__device__ __forceinline__ int winner_rank(const FlipLists &L, const int4 *rec, int n, int index, int lane, int lanes) {
  int r = 0;
  if (n <= kScanRank) {
    for (int k = lane; k < n; k += lanes) {
      const int4 x = rec[k];
      r += (x.y >= 0 && (x.y & FD_WON) && x.x < index) ? 1 : 0;
    }
  } else {
    const int w = index >> 5, c = index >> 10, sc = index >> 15;
    for (int i = lane; i < sc; i += lanes) r += L.wsup[i];
    for (int i = (sc << 5) + lane; i < c; i += lanes) r += L.wcnt[i];
    for (int i = (c << 5) + lane; i < w; i += lanes) r += __popc(L.wbits[i]);
    if (lane == 0) r += __popc(L.wbits[w] & ((1u << (index & 31)) - 1u));
  }
#ifndef GQM_HOST_EMU
  for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
#endif
  return r;
}
// Phase 4, only in a step with something to do: kernelMarkReduntantSteiner
// (refine.cu:2298-2326) on the triangles claimed for a deletion, and the
// stores into subseg2tri that both sides of a subsegment make in this step.
// The latter are ordered as the reference's racing stores land (see wkey) by
// the winners' positions in its winner list, which is in triangle order.
__device__ __noinline__ void flip_late(const Mesh &M, int n, const FlipQ &Q, uint32_t epoch, const FlipLists &L,
                                          const int4 *rec, int nred, int nlate, int tid, int size) {
  for (int k = tid; k < nred; k += size) {
    const int index = L.red[k];
    const int v = claimed(M, Q.gen, index);
    if (v >= 0) continue;
    const int otri = negate_idx(v);
    const int triIndex = dtri(otri), triOri = dori(otri);
    if (triIndex != index) push_flag(M, Q, index);
    M.pred[ld1(M.tv, triIndex, m3(triOri + 1))] = 1;
    mark_fan(M, Q, triIndex, triOri);
  }
#ifdef GQM_HOST_EMU
  const int lane = 0, lanes = 1;
#else
  const int lane = (int)(threadIdx.x & 31u), lanes = 32;
#endif
  for (int e = tid / lanes; e < nlate; e += size / lanes) {
    const int4 x = L.late[e];
    const int rank = winner_rank(L, rec, n, x.z, lane, lanes);
    if (lane == 0) s2t_store(M, x.x, x.y, epoch, wkey(rank, x.w));
  }
}

// One flip-flop loop (refine.cu:2328-2490) by one team of threads: a thread
// block, or several blocks.  Team has tid(), size(), lead() and sync(), which
// is a barrier for the team that returns false once a wait has run out.
// cnt points at the step's list lengths (the control block's, or a copy in
// shared memory).  Registers of every thread: the generation of the last
// pushes, the epoch and the steps done.
struct FlipRegs {
  int gen;
  unsigned epoch;
  int steps;
};
enum { FLIP_GO = 0, FLIP_DONE = 1, FLIP_BROKEN = 2 };
template <int PRED, class Team>
__device__ __forceinline__ int flip_step(const Mesh &M, const FlipLists &L, FlipCnt *cnt, FlipRegs &R, int entry_steps,
                                         Team &T, const int *cur, int n, int4 *rec, KTimer *tm, int *wins) {
  FlipCtl *c = L.c;
  const int g = R.gen, s = g + 1;
  const unsigned long long t0 = (tm && T.lead()) ? global_ns() : 0;
  const FlipQ Q{(s & 1) ? L.q1 : L.q0, &cnt->qn[s & 1], s};
  if (T.lead()) cnt->qn[s & 1] = 0;  // the queue two generations ago, read to its end before the last barrier
  flip_check<PRED>(M, cur, n, s, L, rec, &cnt->live[s & 1], &cnt->nred[s & 1], T.tid(), T.size());
  if (!T.sync()) return FLIP_BROKEN;
  const int live = vload(&cnt->live[s & 1]);
  R.gen = s;
  if (tm && T.lead()) ktimer_add(tm, t0, live);
  if (live == 0) return FLIP_DONE;
  if ((long long)(R.steps - entry_steps) >= c->cap) {
    if (T.lead()) {
      c->cap_hit = 1;
      atomicCAS(c->errp, 0, -2);
    }
    return FLIP_DONE;
  }
  R.steps++;
  R.epoch++;
  if (T.lead()) {
    const int b = 31 - __clz(live);
    atomicAdd(&c->prof_steps[b], 1ull);
    atomicAdd(&c->prof_items[b], (unsigned long long)live);
    cnt->live[g & 1] = cnt->nred[g & 1] = cnt->nlate[g & 1] = 0;  // the next step's
  }
  flip_apply(M, n, Q, L, rec, T.tid(), T.size());
  if (!T.sync()) return FLIP_BROKEN;
  flip_fix(M, n, Q, R.epoch, L, rec, &cnt->nlate[s & 1], T.tid(), T.size());
  if (!T.sync()) return FLIP_BROKEN;
  const int nred = vload(&cnt->nred[s & 1]), nlate = vload(&cnt->nlate[s & 1]);
  if (nred | nlate) {
    flip_late(M, n, Q, R.epoch, L, rec, nred, nlate, T.tid(), T.size());
    if (!T.sync()) return FLIP_BROKEN;
  }
  if (wins) {  // probe only
    if (T.lead())
      for (int k = 0; k < n; ++k) *wins += (rec[k].y >= 0 && (rec[k].y & FD_WON)) ? 1 : 0;
    if (!T.sync()) return FLIP_BROKEN;
  }
  return FLIP_GO;
}
// the loop's state back in the control block, ready for the next pushes (and the
// claims of splitTriangles, which use the generations in between)
__device__ __forceinline__ void flip_close(FlipCtl *c, const FlipRegs &R) {
  c->cnt = FlipCnt{};
  c->gen = R.gen + kGenStride;
  c->epoch = R.epoch;
  c->steps = R.steps;
}

// shared-memory copies of the small steps' lists
constexpr int kSmallCap = 1024;
struct SmallLists {
  FlipCnt cnt;
  int4 rec[kSmallCap];
};
// One flip-flop loop (refine.cu:2328-2490) by the team G.  Most steps are
// small: of the ~1,030 steps of a 2,000,000-point refinement, ~700 have at most
// 1,024 queued triangles, and a barrier of all blocks would cost more than such
// a step's work.  Those are run by the team's first block alone, whose barrier
// is __syncthreads() and which keeps the list lengths and the decisions in
// shared memory, or by the team S of the first few, while the other blocks wait
// at one barrier.  ktm / stm: timers of the check phase of the steps run by all
// blocks and of the small steps (probe), or null.  False when a barrier's wait
// ran out.
template <int PRED>
__device__ __forceinline__ bool flip_loop(const Mesh &M, const FlipLists &L, SmallLists &sh, GridTeam &G, int small_limit,
                                          GridTeam *S, KTimer *ktm, KTimer *stm) {
  FlipCtl *c = L.c;
  FlipRegs R{vload(&c->gen), (unsigned)vload((const int *)&c->epoch), vload(&c->steps)};
  FlipCnt *cnt = &c->cnt;
  const int entry = R.steps;
  const int timed = ktm ? ktm->on : 0;
  const int small_blocks = S ? S->nb : 1;
  const unsigned long long t0 = G.lead() ? global_ns() : 0;
  int status = FLIP_GO, turn = 0;
  // Every block takes the same way through the loop: the words it decides on
  // were complete before the last barrier of all blocks (before the launch, at
  // the loop's entry) and stay as they are until the next.  A run of small steps
  // therefore works on a copy of the list lengths and leaves what it comes to
  // in c->out[turn], which the others read behind that barrier; the one it left
  // before is not read any more by then.
  while (status == FLIP_GO) {
    const int n = vload(&cnt->qn[R.gen & 1]);
    if (n == 0) break;
    if (n > small_limit) {
      status = flip_step<PRED>(M, L, cnt, R, entry, G, (R.gen & 1) ? L.q1 : L.q0, n, L.rec, timed ? ktm : nullptr,
                               nullptr);
      continue;
    }
    FlipOut *o = &c->out[turn];
    turn ^= 1;
    if (G.rank < small_blocks) {
      const unsigned long long s0 = timed && G.lead() ? global_ns() : 0;
      const int steps0 = R.steps;
      int items = 0, wins = 0, m = n;
      if (!S) {
        BlockTeam B;
        if (B.lead()) sh.cnt = *cnt;
        B.sync();
        while (status == FLIP_GO && m > 0 && m <= small_limit) {
          items += m;
          status = flip_step<PRED>(M, L, &sh.cnt, R, entry, B, (R.gen & 1) ? L.q1 : L.q0, m,
                                   m <= kSmallCap ? sh.rec : L.rec, nullptr, timed ? &wins : nullptr);
          m = vload(&sh.cnt.qn[R.gen & 1]);
        }
        if (B.lead()) o->cnt = sh.cnt;
      } else {
        if (S->lead()) o->cnt = *cnt;
        if (!S->sync()) status = FLIP_BROKEN;
        while (status == FLIP_GO && m > 0 && m <= small_limit) {
          items += m;
          status = flip_step<PRED>(M, L, &o->cnt, R, entry, *S, (R.gen & 1) ? L.q1 : L.q0, m, L.rec, nullptr,
                                   timed ? &wins : nullptr);
          m = vload(&o->cnt.qn[R.gen & 1]);
        }
      }
      if (G.lead()) {
        o->gen = R.gen;
        o->epoch = R.epoch;
        o->steps = R.steps;
        o->status = status;
        c->small_steps += R.steps - steps0;
        if (timed) ktimer_add(stm, s0, items, wins);
      }
    }
    if (!G.sync()) return false;
    cnt = &o->cnt;
    R.gen = vload(&o->gen);
    R.epoch = (unsigned)vload((const int *)&o->epoch);
    R.steps = vload(&o->steps);
    status = vload(&o->status);
  }
  if (status == FLIP_BROKEN || !G.sync()) return false;  // nobody reads the control block any more
  if (G.lead()) {
    flip_close(c, R);
    c->ran++;
    c->loop_ns += global_ns() - t0;
    c->loops++;
  }
  return true;
}

// ============================================================================
// Midpoint insertion (refine.cu:2492-3070)
// ============================================================================
__device__ __forceinline__ void reset_tri_and_nbrs(const Mesh &M, int t, bool mark) {
  if (mark) M.tmark[t] = kMaxInt;
  M.tfo[t] = 15;
  int4 nb = M.tn[t];
  if (nb.x != -1) M.tfo[dtri(nb.x)] = 15;
  if (nb.y != -1) M.tfo[dtri(nb.y)] = 15;
  if (nb.z != -1) M.tfo[dtri(nb.z)] = 15;
}
// kernelResetMidInsertionMarker, refine.cu:2492-2542
GQM_KERNEL void k_reset_mid(Mesh M, const int *mids, const int *dn, const int *imark) {
  int n = *dn;
  GS_LOOP(pos, n) {
    int sindex = imark[mids[pos]];
    int otri = s2t_get(M, sindex);
    int t = dtri(otri), o = dori(otri);
    reset_tri_and_nbrs(M, t, true);
    int on = ld1(M.tn, t, o);
    if (on != -1) reset_tri_and_nbrs(M, dtri(on), true);
  }
}
// kernelMarkMidInsertion, refine.cu:2544-2579
GQM_KERNEL void k_mark_mid(Mesh M, const int *mids, const int *dn, const int *imark) {
  int n = *dn;
  GS_LOOP(pos, n) {
    int sindex = imark[mids[pos]];
    int otri = s2t_get(M, sindex);
    int t = dtri(otri), o = dori(otri);
    atomicMin(M.tmark + t, sindex);
    int on = ld1(M.tn, t, o);
    if (on != -1) atomicMin(M.tmark + dtri(on), sindex);
  }
}
// Snapshot of subseg2tri for every candidate before any winner writes
// (the reference reads it at refine.cu:2636 in the same kernel that rewrites
// it at 2844-2850).
GQM_KERNEL void k_mid_snapshot(Mesh M, const int *mids, const int *dn, const int *imark, int *snap) {
  int n = *dn;
  GS_LOOP(pos, n) snap[pos] = s2t_get(M, imark[mids[pos]]);
}

// kernelInsertMidPoints, refine.cu:2594-2927 (debug printing left out)
template <class S, class N>
GQM_KERNEL void GQM_WALK_BOUNDS k_insert_mid(Mesh M, const int *mids, const int *dn, int *imark, const int *snap,
                                             S pslots_, S tslots_, N nsub_, FlipLists L,
                                             unsigned long long *counter) {
  const int *pslots = slots_of(pslots_), *tslots = slots_of(tslots_);
  const int nsub = nval(nsub_);
  int n = *dn;
  const FlipQ Q = entry_queue(L);
  uint32_t epoch = L.c->epoch;
  GS_LOOP(pos, n) {
    int tindex = mids[pos];
    int sindex = imark[tindex];
    int otri = snap[pos];
    int tri[4], triOri[2];
    tri[0] = dtri(otri);
    triOri[0] = dori(otri);
    if (M.tmark[tri[0]] != sindex) continue;
    int4 s0 = M.tsg[tri[0]];
    bool acutedest = comp(s0, m3(triOri[0] + 1)) != -1;
    bool acuteorg = comp(s0, m3(triOri[0] + 2)) != -1;
    int4 n0 = M.tn[tri[0]];
    int on = comp(n0, triOri[0]);
    tri[2] = dtri(on);
    triOri[1] = dori(on);
    if (tri[2] != -1 && M.tmark[tri[2]] != sindex) continue;
    int4 s2 = make_int4(-1, -1, -1, 0);
    if (tri[2] != -1) {
      s2 = M.tsg[tri[2]];
      if (comp(s2, m3(triOri[1] + 1)) != -1) acuteorg = true;
      if (comp(s2, m3(triOri[1] + 2)) != -1) acutedest = true;
    }
    int newp = pslots[tindex];
    tri[1] = tslots[2 * tindex];
    tri[3] = tslots[2 * tindex + 1];
    M.ps[newp] = PS_STEINER | PS_NEW | PS_SEGSPLIT;
    M.pred[newp] = 0;
    M.enc[sindex] = -1;
    M.enc[nsub + tindex] = -1;
    int4 v0 = M.tv[tri[0]];
    int p[3] = {comp(v0, m3(triOri[0] + 1)), comp(v0, m3(triOri[0] + 2)), comp(v0, triOri[0])};
    double2 a = M.pts[p[0]], b = M.pts[p[1]], c = M.pts[p[2]];
    double segmentlength = sqrt(gqm_madd(a.x - b.x, a.x - b.x, (a.y - b.y) * (a.y - b.y)));
    double split = 0.5;
    if (acuteorg || acutedest) {
      double npt = 1.0;
      while (segmentlength > 3.0 * npt) npt *= 2.0;
      while (segmentlength < 1.5 * npt) npt *= 0.5;
      split = npt / segmentlength;
      if (acutedest) split = 1.0 - split;
    }
    double2 m = make_double2(gqm_madd(b.x - a.x, split, a.x), gqm_madd(b.y - a.y, split, a.y));
    double multiplier = gqm_orient_ref(a.x, a.y, b.x, b.y, m.x, m.y);
    double divisor = gqm_madd(a.x - b.x, a.x - b.x, (a.y - b.y) * (a.y - b.y));
    if ((multiplier != 0.0) && (divisor != 0.0)) {
      multiplier = multiplier / divisor;
      if (multiplier == multiplier) {
        m.x = gqm_madd(multiplier, b.y - a.y, m.x);
        m.y = gqm_madd(multiplier, a.x - b.x, m.y);
      }
    }
    M.pts[newp] = m;
    int seg[3] = {comp(s0, triOri[0]), comp(s0, m3(triOri[0] + 1)), comp(s0, m3(triOri[0] + 2))};
    M.tsg[tri[0]] = make_int4(seg[2], seg[0], -1, 0);
    M.tsg[tri[1]] = make_int4(seg[1], -1, nsub + tindex, 0);
    s2t_store(M, seg[0], (tri[0] << 2) | 1, epoch, wkey(pos, 0));
    s2t_store(M, nsub + tindex, (tri[1] << 2) | 2, epoch, wkey(pos, 1));
    M.s2seg[nsub + tindex] = M.s2seg[seg[0]];
    if (seg[1] != -1) s2t_store(M, seg[1], (tri[1] << 2) | 0, epoch, wkey(pos, 2));
    if (seg[2] != -1) s2t_store(M, seg[2], (tri[0] << 2) | 0, epoch, wkey(pos, 3));
    int e_s = -1, e_n = -1;
    if (encroached(a, m, c, M.gc2, M.mode)) e_s = 0;
    if (encroached(m, b, c, M.gc2, M.mode)) e_n = 0;
    int nb1 = comp(n0, m3(triOri[0] + 1)), nb2 = comp(n0, m3(triOri[0] + 2));
    M.tv[tri[0]] = make_int4(newp, p[2], p[0], 0);
    M.tv[tri[1]] = make_int4(newp, p[1], p[2], 0);
    if (tri[2] == -1) {
      M.tn[tri[0]] = make_int4(nb2, -1, (tri[1] << 2) | 1, 0);
      M.tn[tri[1]] = make_int4(nb1, (tri[0] << 2) | 2, -1, 0);
    } else {
      M.tn[tri[0]] = make_int4(nb2, (tri[2] << 2) | 2, (tri[1] << 2) | 1, 0);
      M.tn[tri[1]] = make_int4(nb1, (tri[0] << 2) | 2, (tri[3] << 2) | 1, 0);
    }
    M.tst[tri[0]] |= TS_CHECK;
    push_flag(M, Q, tri[0]);
    M.tfo[tri[0]] = 0;
    M.tst[tri[1]] = TS_NOTNULL | TS_CHECK;
    push_flag(M, Q, tri[1]);
    M.tfo[tri[1]] = 0;
    if (tri[2] != -1) {
      int sg2[3] = {comp(s2, triOri[1]), comp(s2, m3(triOri[1] + 1)), comp(s2, m3(triOri[1] + 2))};
      M.tsg[tri[2]] = make_int4(sg2[1], -1, sg2[0], 0);
      M.tsg[tri[3]] = make_int4(sg2[2], nsub + tindex, -1, 0);
      if (sg2[1] != -1) s2t_store(M, sg2[1], (tri[2] << 2) | 0, epoch, wkey(pos, 4));
      if (sg2[2] != -1) s2t_store(M, sg2[2], (tri[3] << 2) | 0, epoch, wkey(pos, 5));
      int4 v2 = M.tv[tri[2]];
      int q[3] = {comp(v2, m3(triOri[1] + 1)), comp(v2, m3(triOri[1] + 2)), comp(v2, triOri[1])};
      double2 qa = M.pts[q[0]], qb = M.pts[q[1]], qc = M.pts[q[2]];
      if (encroached(qa, m, qc, M.gc2, M.mode)) e_n = 0;
      if (encroached(m, qb, qc, M.gc2, M.mode)) e_s = 0;
      int4 n2 = M.tn[tri[2]];
      int m1 = comp(n2, m3(triOri[1] + 1)), m2 = comp(n2, m3(triOri[1] + 2));
      M.tv[tri[2]] = make_int4(newp, q[1], q[2], 0);
      M.tn[tri[2]] = make_int4(m1, (tri[3] << 2) | 2, (tri[0] << 2) | 1, 0);
      M.tv[tri[3]] = make_int4(newp, q[2], q[0], 0);
      M.tn[tri[3]] = make_int4(m2, (tri[1] << 2) | 2, (tri[2] << 2) | 1, 0);
      M.tst[tri[2]] |= TS_CHECK;
      push_flag(M, Q, tri[2]);
      M.tfo[tri[2]] = 0;
      M.tst[tri[3]] = TS_NOTNULL | TS_CHECK;
      push_flag(M, Q, tri[3]);
      M.tfo[tri[3]] = 0;
    }
    M.enc[sindex] = e_s;
    M.enc[nsub + tindex] = e_n;
    imark[tindex] = -1;
    count_event(counter);
  }
}

// Outer-edge relinking of new triangles (edge 0 faces outward), shared by
// kernelUpdateMidNeighbors (2929-3070) and kernelUpdateSteinerNeighbors
// (4902-5059).
__device__ void relink_outer(const Mesh &M, const int *tri, int iteration) {
  for (int i = 0; i < iteration; i++) {
    int curTri = tri[i];
    int seg = ld1(M.tsg, curTri, 0);
    int pOppTri = ld1(M.tn, curTri, 0);
    int pOpp = dtri(pOppTri), pOri = dori(pOppTri);
    int4 cv = M.tv[curTri];
    if (pOppTri < 0) {
      if (seg != -1) {
        M.enc[seg] = encroached(M.pts[cv.y], M.pts[cv.z], M.pts[cv.x], M.gc2, M.mode) ? 0 : -1;
      }
      continue;
    }
    if (M.tfo[pOpp] == 15) {
      st1(M.tn, pOpp, pOri, etri(curTri, 0));
      if (seg != -1) {
        double2 v0 = M.pts[cv.y], v1 = M.pts[cv.z], v2 = M.pts[cv.x];
        double2 v3 = M.pts[ld1(M.tv, pOpp, pOri)];
        bool e = encroached(v0, v1, v2, M.gc2, M.mode) || encroached(v1, v0, v3, M.gc2, M.mode);
        M.enc[seg] = e ? 0 : -1;
      }
    } else {
      for (int j = 0; j < 3; j++) {
        int neighbor = (j == 0) ? pOpp : dtri(ld1(M.tn, pOpp, j));
        if (neighbor > -1) {
          int4 nv = M.tv[neighbor];
          if (cv.y == nv.z && cv.z == nv.y) {
            st1(M.tn, neighbor, 0, etri(curTri, 0));
            if (seg != -1) {
              double2 v0 = M.pts[cv.y], v1 = M.pts[cv.z], v2 = M.pts[cv.x], v3 = M.pts[nv.x];
              bool e = encroached(v0, v1, v2, M.gc2, M.mode) || encroached(v1, v0, v3, M.gc2, M.mode);
              M.enc[seg] = e ? 0 : -1;
            }
            break;
          }
        }
      }
    }
  }
}

// kernelUpdateMidNeighbors, refine.cu:2929-3070
GQM_KERNEL void k_update_mid_nbrs(Mesh M, const int *mids, const int *dn, const int *imark, const int *enclist) {
  int n = *dn;
  GS_LOOP(pos, n) {
    int tindex = mids[pos];
    if (imark[tindex] != -1) continue;
    int sindex = enclist[tindex];
    int tri[4];
    tri[0] = dtri(s2t_get(M, sindex));
    int4 n0 = M.tn[tri[0]];
    tri[1] = dtri(n0.z);
    int iteration = (n0.y == -1) ? 2 : 4;
    tri[2] = dtri(n0.y);
    tri[3] = dtri(ld1(M.tn, tri[1], 2));
    relink_outer(M, tri, iteration);
  }
}

// kernelUpdatePStatus2Old, refine.cu:3072-3083
template <class N>
GQM_KERNEL void k_points_old(Mesh M, N npts_) {
  const int npts = nval(npts_);
  GS_LOOP(i, npts) {
    uint8_t s = M.ps[i];
    if (!(s & PS_DELETED)) M.ps[i] = (uint8_t)(s & ~PS_NEW);
  }
}

// ============================================================================
// Steiner points (refine.cu:3780-5105)
// ============================================================================
// computeCircumcenter, refine.cu:3780-3868
__device__ __forceinline__ double2 circumcenter(double2 vApex, double2 vOrg, double2 vDest, double offConstant,
                                                bool offcenter) {
  // gqm_madd: the products the reference's contracted build fuses (see
  // predicates.h); the sums are the same in either order
  double xdo = vDest.x - vOrg.x, ydo = vDest.y - vOrg.y;
  double xao = vApex.x - vOrg.x, yao = vApex.y - vOrg.y;
  double dodist = gqm_madd(xdo, xdo, ydo * ydo);
  double aodist = gqm_madd(xao, xao, yao * yao);
  double dadist = gqm_madd(vDest.x - vApex.x, vDest.x - vApex.x, (vDest.y - vApex.y) * (vDest.y - vApex.y));
  double tmp = xdo * yao - xao * ydo;
  double denominator = (tmp != 0) ? 0.5 / tmp : 0.5 / gqm_orient_ref(vDest.x, vDest.y, vApex.x, vApex.y, vOrg.x, vOrg.y);
  double dx = gqm_madd(yao, dodist, -(ydo * aodist)) * denominator;
  double dy = gqm_madd(xdo, aodist, -(xao * dodist)) * denominator;
  if (offcenter && (offConstant > 0.0)) {
    double dxoff, dyoff;
    if ((dodist < aodist) && (dodist < dadist)) {
      dxoff = 0.5 * xdo - offConstant * ydo;
      dyoff = gqm_madd(offConstant, xdo, 0.5 * ydo);
      if (gqm_madd(dxoff, dxoff, dyoff * dyoff) < gqm_madd(dx, dx, dy * dy)) {
        dx = dxoff;
        dy = dyoff;
      }
    } else if (aodist < dadist) {
      dxoff = 0.5 * xao + offConstant * yao;
      dyoff = 0.5 * yao - offConstant * xao;
      if (gqm_madd(dxoff, dxoff, dyoff * dyoff) < gqm_madd(dx, dx, dy * dy)) {
        dx = dxoff;
        dy = dyoff;
      }
    } else {
      dxoff = 0.5 * (vApex.x - vDest.x) - offConstant * (vApex.y - vDest.y);
      dyoff = gqm_madd(offConstant, vApex.x - vDest.x, 0.5 * (vApex.y - vDest.y));
      if (gqm_madd(dxoff, dxoff, dyoff * dyoff) < gqm_madd(dx - xdo, dx - xdo, (dy - ydo) * (dy - ydo))) {
        dx = xdo + dxoff;
        dy = ydo + dyoff;
      }
    }
  }
  return make_double2(vOrg.x + dx, vOrg.y + dy);
}

GQM_KERNEL void k_circumcenter(Mesh M, const int *bad, const int *dn, double offc, int offcenter, double2 *center) {
  int n = *dn;
  GS_LOOP(k, n) {
    int4 v = M.tv[bad[k]];
    center[k] = circumcenter(M.pts[v.x], M.pts[v.y], M.pts[v.z], offc, offcenter != 0);
  }
}

// kernelLocateSinkPoints, refine.cu:3908-4184
template <int PRED>
GQM_KERNEL void k_locate(Mesh M, const int *bad, const int *dn, const double2 *center, int *sinks, FlipLists L) {
  int n = *dn;
  const int gen = L.c->gen - kGenLocate;
  GS_LOOP(k, n) {
    int index = bad[k];
    if (!(M.tst[index] & TS_BAD)) {
      sinks[k] = -1;
      continue;
    }
    double2 cc = center[k];
    int curTri = index, curOri = 0;
    bool checkNeighbor = false, split = false;
    int dart = 3;
    int4 v = M.tv[curTri];
    double2 w0 = M.pts[v.x], w1 = M.pts[v.y], w2 = M.pts[v.z];
    double det0 = orient<PRED>(w0, w1, cc), det1 = orient<PRED>(w1, w2, cc), det2 = orient<PRED>(w2, w0, cc);
    int4 sg = M.tsg[index];
    if (det0 <= 0) {
      if (det0 == 0 || sg.z != -1) split = true;
      dart = 2;
    } else if (det1 <= 0) {
      if (det1 == 0 || sg.x != -1) split = true;
      dart = 0;
    } else if (det2 <= 0) {
      if (det2 == 0 || sg.y != -1) split = true;
      dart = 1;
    }
    if (!split && dart != 3) {
      int nb = ld1(M.tn, curTri, dart);
      if (nb < 0) {
        split = true;
      } else {
        curTri = dtri(nb);
        curOri = dori(nb);
        checkNeighbor = true;
      }
    }
    int guard = 0;
    while (checkNeighbor) {
      if (++guard > (1 << 24)) {
        raise_err(M, -3);
        break;
      }
      int4 tv = M.tv[curTri];
      double2 u[3] = {M.pts[tv.x], M.pts[tv.y], M.pts[tv.z]};
      dart = 3;
      int pOrg = m3(curOri + 1), pDest = m3(curOri + 2), pApex = curOri;
      double detLeft = orient<PRED>(u[pDest], u[pApex], cc);
      double detRight = orient<PRED>(u[pApex], u[pOrg], cc);
      bool moveleft;
      if (detLeft < 0.0) {
        if (detRight < 0.0)
          moveleft = gqm_madd(u[pDest].x - u[pOrg].x, cc.x - u[pApex].x,
                              (u[pDest].y - u[pOrg].y) * (cc.y - u[pApex].y)) >
                     0.0;
        else
          moveleft = true;
      } else {
        if (detRight < 0.0)
          moveleft = false;
        else {
          if (detLeft == 0.0) {
            split = true;
            dart = m3(curOri + 1);
            break;
          }
          if (detRight == 0.0) {
            split = true;
            dart = m3(curOri + 2);
            break;
          }
          break;
        }
      }
      dart = moveleft ? m3(curOri + 1) : m3(curOri + 2);
      int nb = ld1(M.tn, curTri, dart);
      if (nb < 0 || ld1(M.tsg, curTri, dart) != -1) {
        split = true;
        break;
      }
      curTri = dtri(nb);
      curOri = dori(nb);
    }
    claim(M, gen, curTri, index);
    if (split) {
      int nb = ld1(M.tn, curTri, dart);
      if (nb != -1) claim(M, gen, dtri(nb), index);
    }
    sinks[k] = (curTri << 2) | dart;
  }
}

// kernelRemoveLosers, refine.cu:4186-4235
GQM_KERNEL void k_remove_losers(Mesh M, const int *bad, const int *dn, const int *sinks, int *imark, FlipLists L) {
  int n = *dn;
  const int gen = L.c->gen - kGenLocate;
  GS_LOOP(k, n) {
    if (imark[k] < 0) continue;
    int sink = sinks[k] >> 2, dir = sinks[k] & 3, index = bad[k];
    if (claimed(M, gen, sink) != index) {
      imark[k] = -1;
      continue;
    }
    if (dir != 3) {
      int nb = ld1(M.tn, sink, dir);
      if (nb != -1 && claimed(M, gen, dtri(nb)) != index) imark[k] = -1;
    }
  }
}

// Cavity walk of kernelMarkCavities (4237-4368): depth-first over neighbours
// whose circumcircle contains the centre, not crossing subsegments except the
// sink's split edge, at most 50 triangles.  Returns the number of triangles in
// the cavity (stored, in visiting order, at out[j * stride]) or -1 when the
// cavity exceeds the cap.
//
// kernelCheckCavities (4422-4547) repeats the same walk and fails at the first
// triangle whose marker is not the candidate's.  Between the two launches only
// the markers change, never the mesh or the centres, so its walk visits exactly
// the triangles stored here (up to the first failure): checking the stored
// list gives the same verdict without a second walk or any predicate.
//
// The reference rescans a triangle's three edges from the first every time the
// walk comes back to it; the edges before the one it descended through were
// then rejected (circumcircle test false, a subsegment or the boundary) or lead
// to a triangle already in the region, and neither changes while the walk runs.
// So each stack frame keeps the edge to resume at: the same triangles are
// visited and claimed in the same order, each neighbour tested once.
//
// The three neighbours of a triangle are tested together when the walk first
// reaches it, with all their loads in flight at once (rows, then points), and
// the outcomes are kept in the frame; which edge the walk takes is still decided
// edge by edge from the resume point, with the region as it is then.  Nothing a
// test reads changes during the walk (only claim markers do), so the walk takes
// the same edges as one that tests each neighbour when it gets to it.
__device__ __forceinline__ unsigned cavity_hash(int t) { return ((unsigned)t * 2654435761u) >> 26; }
template <int PRED>
__device__ GQM_WALK_CALL int cavity_walk(const Mesh &M, int gen, int sink, int direction, double2 cc, int badIndex, int *out,
                           int stride) {
  int region[kCavityCap], loop[kCavityCap];  // loop: (triangle << 2) | edge to resume at
  uint8_t inside[kCavityCap];                // per frame: neighbours whose circumcircle holds cc
  // one bit per hash of the region's triangles: a clear bit proves a triangle
  // is not in the region without scanning it (a set bit still scans)
  unsigned long long rbits = 0;
  int rsize = 0, lsize = 0;
  int cur = sink, start = 0;
  for (int guard = 0; guard < 4 * kCavityCap * 3 + 16; ++guard) {
    int4 nb = make_int4(-1, -1, -1, -1);
    if (start == 0) {  // first visit (a return always resumes past the edge it left by)
      if (rsize == kCavityCap || lsize == kCavityCap) return -1;
      region[rsize++] = cur;
      rbits |= 1ull << cavity_hash(cur);
      loop[lsize++] = cur << 2;
      claim(M, gen, cur, badIndex);
      const int4 sg = M.tsg[cur];
      nb = M.tn[cur];
      int tt[3];
      int4 q[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const int si = comp(sg, i);
        bool ok = comp(nb, i) != -1;
        if (cur == sink) {
          if (direction == 3 && si != -1) ok = false;
          if (direction < 3 && si != -1 && i != direction) ok = false;
        } else if (si != -1) {
          ok = false;
        }
        tt[i] = ok ? dtri(comp(nb, i)) : -1;
      }
#pragma unroll
      for (int i = 0; i < 3; i++)
        if (tt[i] >= 0) q[i] = M.tv[tt[i]];
      unsigned bits = 0;
#pragma unroll
      for (int i = 0; i < 3; i++)
        if (tt[i] >= 0 && incircle<PRED>(M.pts[q[i].x], M.pts[q[i].y], M.pts[q[i].z], cc) > 0) bits |= 1u << i;
      inside[lsize - 1] = (uint8_t)bits;
    } else if (inside[lsize - 1] >> start) {
      nb = M.tn[cur];
    }
    int nIdx = -1, taken = -1;
    const unsigned bits = inside[lsize - 1];
    for (int i = start; i < 3; i++) {
      if (!((bits >> i) & 1u)) continue;
      const int t = dtri(comp(nb, i));
      bool seen = false;
      if ((rbits >> cavity_hash(t)) & 1ull)
        for (int r = 0; r < rsize; ++r)
          if (region[r] == t) {
            seen = true;
            break;
          }
      if (seen) continue;
      nIdx = t;
      taken = i;
      break;
    }
    if (taken >= 0) {
      loop[lsize - 1] = (cur << 2) | (taken + 1);
      cur = nIdx;
      start = 0;
    } else {
      if (lsize > 0) lsize--;
      if (lsize == 0) {
        for (int j = 0; j < rsize; ++j) out[(long)j * stride] = region[j];
        return rsize;
      }
      cur = loop[lsize - 1] >> 2;
      start = loop[lsize - 1] & 3;
    }
  }
  raise_err(M, -6);
  return 0;
}

#if defined(GQM_CTA_MODE) && !defined(GQM_HOST_EMU)
// The same cavity by sixteen lanes: the triangles found so far are a list
// spread over the lanes' registers, and every pass tests the next sixteen of
// their edges together, each with its own loads (link and subsegment, then the
// neighbour's row, then its points).  Which triangles the cavity holds does not
// depend on the order in which they are reached, so a cavity within the cap is
// claimed when it is complete; of a larger one the reference claims the first
// fifty in its own order, and that one is left to cavity_walk (-1 is returned,
// nothing is claimed).
//
// Bound by latency: the walk waits three dependent loads for every triangle, a
// pass here for every step outward from the sink.  Outside its flip loops a
// refinement of 3,000 points takes 4.2 ms instead of 5.5 ms, one of 10,000
// points 3.6 ms instead of 4.0 ms, one of 100,000 points 6.9 ms instead of 7.1 ms.
template <int PRED>
__device__ __forceinline__ int cavity_group(const Mesh &M, int gen, int sink, int direction, double2 cc, int badIndex,
                                            int *out, int stride) {
  const int lane = (int)(threadIdx.x & 31u), gl = lane & 15;
  const unsigned gm = 0xffffu << (lane & 16);
  static_assert(kCavityCap <= 64, "four entries a lane");
  int r0 = gl == 0 ? sink : -1, r1 = -1, r2 = -1, r3 = -1;  // entries gl, gl + 16, gl + 32, gl + 48
  int size = 1;
  for (int head = 0; head < 3 * size;) {
    const int p = head + gl, end = 3 * size;
    const bool has = p < end;
    const int idx = has ? p / 3 : 0, e = p - 3 * (p / 3), own = (lane & 16) | (idx & 15);
    const int t0 = __shfl_sync(gm, r0, own), t1 = __shfl_sync(gm, r1, own), t2 = __shfl_sync(gm, r2, own),
              t3 = __shfl_sync(gm, r3, own);
    const int t = idx < 16 ? t0 : idx < 32 ? t1 : idx < 48 ? t2 : t3;
    int found = -1;
    if (has) {
      const int link = ld1(M.tn, t, e), sg = ld1(M.tsg, t, e);
      if (link != -1 && (sg == -1 || (t == sink && e == direction))) {
        const int4 q = M.tv[dtri(link)];
        if (incircle<PRED>(M.pts[q.x], M.pts[q.y], M.pts[q.z], cc) > 0) found = dtri(link);
      }
    }
    head = min(head + 16, end);
    unsigned in = __ballot_sync(gm, found >= 0) & gm;
    while (in) {
      const int c = __shfl_sync(gm, found, __ffs(in) - 1);
      in &= in - 1;
      if (__any_sync(gm, r0 == c || r1 == c || r2 == c || r3 == c)) continue;
      if (size == kCavityCap) return -1;
      if (gl == (size & 15)) {
        if (size < 16)
          r0 = c;
        else if (size < 32)
          r1 = c;
        else if (size < 48)
          r2 = c;
        else
          r3 = c;
      }
      ++size;
    }
  }
  const int r[4] = {r0, r1, r2, r3};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (16 * k + gl < size) {
      claim(M, gen, r[k], badIndex);
      out[(long)(16 * k + gl) * stride] = r[k];
    }
  return size;
}
#endif

// kernelMarkCavities: claim every cavity triangle (atomicMin of the bad index);
// an oversized cavity makes its candidate an unconditional winner (negated
// index).  cavn[k] = stored cavity size (0 for an oversized one).
template <int PRED>
GQM_KERNEL void GQM_WALK_BOUNDS k_cavity_mark(Mesh M, const int *dn, const int *sinks, const double2 *center, const int *imark,
                              int *ilist, int *cav, int *cavn, int stride, FlipLists L) {
  int n = *dn;
  const int gen = L.c->gen - kGenCavity;
#if defined(GQM_CTA_MODE) && !defined(GQM_HOST_EMU)
  // Sixteen lanes a candidate while the team needs at most eight passes for
  // them; the grid kernel's inputs have more candidates than that in most rounds
  // (with both ways in it, its walk took 25 ms of a refinement of 2,000,000
  // points outside the flip loops instead of 23 ms).
  if (2 * n <= GQM_GSIZE) {
    const int gl = (int)(threadIdx.x & 15u);
    for (int k = GQM_GTID >> 4; k < n; k += GQM_GSIZE >> 4) {
      if (imark[k] < 0) continue;
      const int badIndex = ilist[k], sk = sinks[k];
      int c = cavity_group<PRED>(M, gen, sk >> 2, sk & 3, center[k], badIndex, cav + k, stride);
      __syncwarp(0xffffu << (threadIdx.x & 16u));  // every lane has read ilist[k]
      if (gl) continue;
      if (c < 0) c = cavity_walk<PRED>(M, gen, sk >> 2, sk & 3, center[k], badIndex, cav + k, stride);
      if (c < 0) ilist[k] = negate_idx(badIndex);
      cavn[k] = c < 0 ? 0 : c;
    }
    return;
  }
#endif
  GS_LOOP(k, n) {
    if (imark[k] < 0) continue;
    const int badIndex = ilist[k];
    const int c = cavity_walk<PRED>(M, gen, sinks[k] >> 2, sinks[k] & 3, center[k], badIndex, cav + k, stride);
    if (c < 0) ilist[k] = negate_idx(badIndex);
    cavn[k] = c < 0 ? 0 : c;
  }
}
// kernelCheckCavities: a candidate loses if any triangle of its cavity was
// claimed by a smaller bad index.
GQM_KERNEL void k_cavity_check(Mesh M, const int *dn, const int *cav, const int *cavn, int stride, int *imark,
                               const int *ilist, FlipLists L) {
  int n = *dn;
  const int gen = L.c->gen - kGenCavity;
  GS_LOOP(k, n) {
    if (imark[k] < 0) continue;
    int badIndex = ilist[k];
    if (badIndex < 0) continue;
    int c = cavn[k];
    for (int j = 0; j < c; ++j)
      if (claimed(M, gen, cav[(long)j * stride + k]) != badIndex) {
        imark[k] = -1;
        break;
      }
  }
}

// kernelMarkSteinerOnsegs, refine.cu:5061-5089
GQM_KERNEL void k_mark_onsegs(Mesh M, const int *wl, const int *dn, const int *sinks, int *encl2) {
  int n = *dn;
  GS_LOOP(w, n) {
    int sk = sinks[wl[w]];
    int index = sk >> 2, dir = sk & 3;
    if (dir != 3) {
      int sg = ld1(M.tsg, index, dir);
      if (sg != -1) encl2[sg] = 0;
    }
  }
}
// kernelResetSteinerInsertionMarker, refine.cu:4601-4649
GQM_KERNEL void k_reset_steiner(Mesh M, const int *wl, const int *dn, const int *sinks) {
  int n = *dn;
  GS_LOOP(w, n) {
    int sk = sinks[wl[w]];
    int index = sk >> 2, dir = sk & 3;
    reset_tri_and_nbrs(M, index, false);
    if (dir != 3) {
      int on = ld1(M.tn, index, dir);
      if (on != -1) reset_tri_and_nbrs(M, dtri(on), false);
    }
  }
}

// kernelInsertSteinerPoints, refine.cu:4651-4900
template <class S>
GQM_KERNEL void k_insert_steiner(Mesh M, const int *wl, const int *dn, const int *sinks, const double2 *center,
                                 S pslots_, S tslots_, FlipLists L, unsigned long long *counter) {
  const int *pslots = slots_of(pslots_), *tslots = slots_of(tslots_);
  int n = *dn;
  const FlipQ Q = entry_queue(L);
  uint32_t epoch = L.c->epoch;
  GS_LOOP(pos, n) {
    int tindex = wl[pos];
    int index = sinks[tindex] >> 2, direction = sinks[tindex] & 3;
    int4 s0 = M.tsg[index];
    if (direction != 3 && comp(s0, direction) != -1) continue;
    int newp = pslots[pos];
    int nt1 = tslots[2 * pos], nt2 = tslots[2 * pos + 1];
    M.ps[newp] = PS_STEINER | PS_NEW;
    M.pred[newp] = 0;
    M.pts[newp] = center[tindex];
    int4 v0 = M.tv[index];
    int4 n0 = M.tn[index];
    if (direction == 3) {
      int t0 = index, t1 = nt1, t2 = nt2;
      M.tsg[t0] = make_int4(s0.x, -1, -1, 0);
      M.tsg[t1] = make_int4(s0.y, -1, -1, 0);
      M.tsg[t2] = make_int4(s0.z, -1, -1, 0);
      if (s0.x != -1) s2t_store(M, s0.x, (t0 << 2) | 0, epoch, wkey(pos, 0));
      if (s0.y != -1) s2t_store(M, s0.y, (t1 << 2) | 0, epoch, wkey(pos, 1));
      if (s0.z != -1) s2t_store(M, s0.z, (t2 << 2) | 0, epoch, wkey(pos, 2));
      // p[i] = vertex (i+1)%3 of the old triangle; neighbour[i] = old edge i
      M.tv[t0] = make_int4(newp, v0.y, v0.z, 0);
      M.tn[t0] = make_int4(n0.x, (t1 << 2) | 2, (t2 << 2) | 1, 0);
      M.tv[t1] = make_int4(newp, v0.z, v0.x, 0);
      M.tn[t1] = make_int4(n0.y, (t2 << 2) | 2, (t0 << 2) | 1, 0);
      M.tv[t2] = make_int4(newp, v0.x, v0.y, 0);
      M.tn[t2] = make_int4(n0.z, (t0 << 2) | 2, (t1 << 2) | 1, 0);
      M.tst[t0] |= TS_CHECK;
      push_flag(M, Q, t0);
      M.tfo[t0] = 0;
      M.tst[t1] = TS_NOTNULL | TS_CHECK;
      push_flag(M, Q, t1);
      M.tfo[t1] = 0;
      M.tst[t2] = TS_NOTNULL | TS_CHECK;
      push_flag(M, Q, t2);
      M.tfo[t2] = 0;
    } else {
      int o0 = direction;
      int otri = comp(n0, o0);
      int o1 = dori(otri);
      int tri0 = index, tri1 = nt1, tri2 = dtri(otri), tri3 = nt2;
      int p0 = comp(v0, m3(o0 + 1)), p1 = comp(v0, m3(o0 + 2)), p2 = comp(v0, o0);
      int seg[3] = {comp(s0, o0), comp(s0, m3(o0 + 1)), comp(s0, m3(o0 + 2))};
      M.tsg[tri0] = make_int4(seg[2], seg[0], -1, 0);
      M.tsg[tri1] = make_int4(seg[1], -1, seg[0], 0);
      if (seg[1] != -1) s2t_store(M, seg[1], (tri1 << 2) | 0, epoch, wkey(pos, 3));
      if (seg[2] != -1) s2t_store(M, seg[2], (tri0 << 2) | 0, epoch, wkey(pos, 4));
      int nb1 = comp(n0, m3(o0 + 1)), nb2 = comp(n0, m3(o0 + 2));
      M.tv[tri0] = make_int4(newp, p2, p0, 0);
      M.tv[tri1] = make_int4(newp, p1, p2, 0);
      if (tri2 == -1) {
        M.tn[tri0] = make_int4(nb2, -1, (tri1 << 2) | 1, 0);
        M.tn[tri1] = make_int4(nb1, (tri0 << 2) | 2, -1, 0);
      } else {
        M.tn[tri0] = make_int4(nb2, (tri2 << 2) | 2, (tri1 << 2) | 1, 0);
        M.tn[tri1] = make_int4(nb1, (tri0 << 2) | 2, (tri3 << 2) | 1, 0);
      }
      M.tst[tri0] |= TS_CHECK;
      push_flag(M, Q, tri0);
      M.tfo[tri0] = 0;
      M.tst[tri1] = TS_NOTNULL | TS_CHECK;
      push_flag(M, Q, tri1);
      M.tfo[tri1] = 0;
      if (tri2 != -1) {
        int4 v2 = M.tv[tri2], n2 = M.tn[tri2], s2 = M.tsg[tri2];
        int q0 = comp(v2, m3(o1 + 1)), q1 = comp(v2, m3(o1 + 2)), q2 = comp(v2, o1);
        int sg2[3] = {comp(s2, o1), comp(s2, m3(o1 + 1)), comp(s2, m3(o1 + 2))};
        M.tsg[tri2] = make_int4(sg2[1], -1, sg2[0], 0);
        M.tsg[tri3] = make_int4(sg2[2], sg2[0], -1, 0);
        if (sg2[1] != -1) s2t_store(M, sg2[1], (tri2 << 2) | 0, epoch, wkey(pos, 5));
        if (sg2[2] != -1) s2t_store(M, sg2[2], (tri3 << 2) | 0, epoch, wkey(pos, 6));
        int m1 = comp(n2, m3(o1 + 1)), m2 = comp(n2, m3(o1 + 2));
        M.tv[tri2] = make_int4(newp, q1, q2, 0);
        M.tn[tri2] = make_int4(m1, (tri3 << 2) | 2, (tri0 << 2) | 1, 0);
        M.tv[tri3] = make_int4(newp, q2, q0, 0);
        M.tn[tri3] = make_int4(m2, (tri1 << 2) | 2, (tri2 << 2) | 1, 0);
        M.tst[tri2] |= TS_CHECK;
        push_flag(M, Q, tri2);
        M.tfo[tri2] = 0;
        M.tst[tri3] = TS_NOTNULL | TS_CHECK;
        push_flag(M, Q, tri3);
        M.tfo[tri3] = 0;
      }
    }
    count_event(counter);
  }
}

// kernelUpdateSteinerNeighbors, refine.cu:4902-5059
GQM_KERNEL void k_update_steiner_nbrs(Mesh M, const int *wl, const int *dn, const int *sinks) {
  int n = *dn;
  GS_LOOP(pos, n) {
    int tindex = wl[pos];
    int index = sinks[tindex] >> 2, direction = sinks[tindex] & 3;
    if (direction != 3 && M.tfo[index] == 15) continue;
    int tri[4], iteration;
    int4 n0 = M.tn[index];
    tri[0] = index;
    if (direction == 3) {
      iteration = 3;
      tri[1] = dtri(n0.y);
      tri[2] = dtri(n0.z);
    } else {
      tri[1] = dtri(n0.z);
      if (n0.y == -1)
        iteration = 2;
      else {
        iteration = 4;
        tri[2] = dtri(n0.y);
        tri[3] = dtri(ld1(M.tn, tri[1], 2));
      }
    }
    relink_outer(M, tri, iteration);
  }
}

// kernelUpdateSteinerOnsegs, refine.cu:5091-5105 (over all subsegments)
template <class N>
GQM_KERNEL void k_onsegs_to_enc(Mesh M, const int *encl2, N ns_) {
  const int ns = nval(ns_);
  GS_LOOP(s, ns) if (encl2[s] >= 0) M.enc[s] = 1;
}

// ============================================================================
// Output compaction (refine.cu:5758-6484)
// ============================================================================
GQM_KERNEL void k_compact_tris_move(Mesh M, const int *tail, const int *empty, const int *dn, int *newidx) {
  int n = *dn;
  GS_LOOP(k, n) {
    int from = tail[k], to = empty[k];
    M.tv[to] = M.tv[from];
    M.tn[to] = M.tn[from];
    M.tst[to] = M.tst[from];
    M.tflip[to] = M.tflip[from];
    M.tfo[to] = M.tfo[from];
    newidx[from] = to;
  }
}
GQM_KERNEL void k_newidx_init(const Mesh M, int *newidx, int n, int newn, const uint8_t *flag, uint8_t deadbit,
                              bool dead_when_set) {
  GS_LOOP(i, n) {
    bool dead = dead_when_set ? (flag[i] & deadbit) != 0 : (flag[i] & deadbit) == 0;
    newidx[i] = dead ? -1 : (i < newn ? i : -2);
  }
}
GQM_KERNEL void k_fix_nbrs(Mesh M, const int *newidx, int newn) {
  GS_LOOP(t, newn) {
    int4 nb = M.tn[t];
    if (nb.x >= 0) nb.x = etri(newidx[dtri(nb.x)], dori(nb.x));
    if (nb.y >= 0) nb.y = etri(newidx[dtri(nb.y)], dori(nb.y));
    if (nb.z >= 0) nb.z = etri(newidx[dtri(nb.z)], dori(nb.z));
    M.tn[t] = nb;
  }
}
GQM_KERNEL void k_fix_s2t(Mesh M, const int *newidx, int ns) {
  GS_LOOP(s, ns) {
    int o = s2t_get(M, s);
    if (o >= 0) M.s2t[s] = s2t_plain(etri(newidx[dtri(o)], dori(o)));
  }
}
GQM_KERNEL void k_compact_pts_move(Mesh M, const int *tail, const int *empty, const int *dn, int *newidx) {
  int n = *dn;
  GS_LOOP(k, n) {
    int from = tail[k], to = empty[k];
    M.pts[to] = M.pts[from];
    M.ps[to] = M.ps[from];
    M.pred[to] = M.pred[from];
    newidx[from] = to;
  }
}
GQM_KERNEL void k_fix_tri_vertices(Mesh M, const int *newidx, int nt) {
  GS_LOOP(t, nt) {
    int4 v = M.tv[t];
    v.x = newidx[v.x];
    v.y = newidx[v.y];
    v.z = newidx[v.z];
    M.tv[t] = v;
  }
}
// TStatus byte of an output triangle.  The reference sets every triangle's flip
// orientation to "none" when a flip-flop loop starts (refine.cu:2356-2372), and
// every insertion is followed by one: after the first loop no triangle of the
// output holds another value, before it all hold 0.
__device__ __forceinline__ uint8_t status_byte(const Mesh &M, int t, int flips_ran) {
  return (uint8_t)((M.tst[t] & 7) | (M.tflip[t] ? 8 : 0) | (flips_ran ? 15 << 4 : 0));
}
// plain output arrays (trianglelist, neighborlist via decode, segmentlist)
GQM_KERNEL void k_emit_output(Mesh M, int nt, int ns, int *tri, int *nbr, int *seg, uint8_t *tstat, const FlipCtl *c) {
  GS_LOOP(i, max(nt, ns)) {
    if (i < nt) {
      int4 v = M.tv[i], nb = M.tn[i];
      tri[3 * i] = v.x;
      tri[3 * i + 1] = v.y;
      tri[3 * i + 2] = v.z;
      nbr[3 * i] = dtri(nb.x);
      nbr[3 * i + 1] = dtri(nb.y);
      nbr[3 * i + 2] = dtri(nb.z);
      tstat[i] = status_byte(M, i, c->ran);
    }
    if (i < ns) {
      int o = s2t_get(M, i);
      if (o < 0) {
        seg[2 * i] = seg[2 * i + 1] = -1;
      } else {
        int t = dtri(o), r = dori(o);
        int4 v = M.tv[t];
        seg[2 * i] = comp(v, m3(r + 1));
        seg[2 * i + 1] = comp(v, m3(r + 2));
      }
    }
  }
}
GQM_KERNEL void k_emit_pstatus(Mesh M, int np, uint8_t *pstat) {
  GS_LOOP(i, np) pstat[i] = (uint8_t)((M.ps[i] & 15) | (M.pred[i] ? 16 : 0));
}

// ---------------------------------------------------------------------------
// The placement step and the collection of training data
// ---------------------------------------------------------------------------
#ifdef GQM_CTA_MODE
#define GQM_BID gqm_team_rank
#define GQM_NB gqm_team_blocks
#else
#define GQM_BID ((int)blockIdx.x)
#define GQM_NB ((int)gridDim.x)
#endif

// Learned placement over the bad triangles, after k_circumcenter has written
// the plain centers: up to kInferWarpsMax warps per block, 32 candidates per
// warp and pass, the network's weights staged in the block's shared memory.
// ctr[0] counts candidates, ctr[1] the points the network placed.
GQM_KERNEL void k_learned_place(Mesh M, const int *bad, const int *dn, MlpDev P, double2 *center,
                                unsigned long long *ctr) {
#ifdef GQM_HOST_EMU
  const int n = GQM_BID == 0 ? *dn : 0;
  for (int k = 0; k < n; ++k) {
    const int t = bad[k];
    const int4 v = M.tv[t];
    const double2 coff = center[k];
    const double2 cc = circumcenter(M.pts[v.x], M.pts[v.y], M.pts[v.z], 0.0, false);
    if (coff.x == cc.x && coff.y == cc.y) continue;
    float f[kFeat];
    features_of(M, t, bisector_of(M, t), 0.0, f);
    const float y = mlp_forward_row(P, f);
    ctr[0]++;
    if (y > 0.0f && y < 1.0f) {
      const double2 p = make_double2(coff.x + (double)y * (cc.x - coff.x), coff.y + (double)y * (cc.y - coff.y));
      if (!encroaches_near(M, t, p)) {
        center[k] = p;
        ctr[1]++;
      }
    }
  }
#else
  __shared__ MlpInferTiles sm;
  mlp_stage(P, sm.w);
  __syncthreads();
  const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
  const int nw = min(kInferWarpsMax, (int)(blockDim.x >> 5));
  if (warp >= nw) return;
  uint16_t *x = sm.x[warp];
  const int n = *dn;
  for (int g0 = (GQM_BID * nw + warp) * 32; g0 < n; g0 += GQM_NB * nw * 32) {
    const int k = g0 + lane;
    bool cand = false;
    int t = -1;
    double2 coff = make_double2(0.0, 0.0), cc = coff;
    if (k < n) {
      t = bad[k];
      const int4 v = M.tv[t];
      coff = center[k];
      cc = circumcenter(M.pts[v.x], M.pts[v.y], M.pts[v.z], 0.0, false);
      cand = (coff.x != cc.x || coff.y != cc.y);
    }
    const unsigned m = __ballot_sync(0xffffffffu, cand);
    if (!m) continue;
    float f[kFeat];
    if (cand) {
      const Bisector B = bisector_of(M, t);
      features_of(M, t, B, 0.0, f);
    } else {
      for (int j = 0; j < kFeat; ++j) f[j] = 0.0f;
    }
    mlp_put_row(x, lane, f);
    __syncwarp();
    const float y = mlp_forward_regs(sm.w, x);
    __syncwarp();
    bool used = false;
    if (cand && y > 0.0f && y < 1.0f) {
      const double2 p = make_double2(coff.x + (double)y * (cc.x - coff.x), coff.y + (double)y * (cc.y - coff.y));
      if (!encroaches_near(M, t, p)) {
        center[k] = p;
        used = true;
      }
    }
    const unsigned u = __ballot_sync(0xffffffffu, used);
    if (lane == 0) {
      atomicAdd(ctr, (unsigned long long)__popc(m));
      atomicAdd(ctr + 1, (unsigned long long)__popc(u));
    }
  }
#endif
}

// Number of triangles with an angle below theta among those that point c
// would form with the boundary of its Delaunay cavity (the triangles whose
// circumcircle contains c, reached from t0 without crossing a subsegment);
// 100 when the cavity has more than 64 triangles.
__device__ inline int star_bad_count(const Mesh &M, int t0, double2 c) {
  int list[64];
  int n = 0, nbad = 0;
  list[n++] = t0;
  for (int i = 0; i < n; ++i) {
    const int tri = list[i];
    const int4 v = M.tv[tri], nb = M.tn[tri], sg = M.tsg[tri];
    const int vv[3] = {v.x, v.y, v.z};
    for (int e = 0; e < 3; ++e) {
      bool boundary = comp(sg, e) >= 0 || comp(nb, e) < 0;
      if (!boundary) {
        const int nt = dtri(comp(nb, e));
        bool seen = false;
        for (int j = 0; j < n && !seen; ++j) seen = (list[j] == nt);
        if (seen) continue;
        const int4 w = M.tv[nt];
        const double2 a = M.pts[w.x], b = M.pts[w.y], d = M.pts[w.z];
        if (gqm_incircle_det_ref(a.x, a.y, b.x, b.y, d.x, d.y, c.x, c.y) > 0.0) {
          if (n == 64) return 100;
          list[n++] = nt;
          continue;
        }
        boundary = true;
      }
      // star triangle (c, u, w) on the boundary edge
      const double2 u = M.pts[vv[(e + 1) % 3]], w = M.pts[vv[(e + 2) % 3]];
      const double l0 = (u.x - w.x) * (u.x - w.x) + (u.y - w.y) * (u.y - w.y);
      const double l1 = (c.x - w.x) * (c.x - w.x) + (c.y - w.y) * (c.y - w.y);
      const double l2 = (c.x - u.x) * (c.x - u.x) + (c.y - u.y) * (c.y - u.y);
      // smallest angle is opposite the shortest side: cos^2 by the law of cosines
      double a2 = l0, b2 = l1, c2 = l2;
      if (b2 < a2) { const double tt = a2; a2 = b2; b2 = tt; }
      if (c2 < a2) { const double tt = a2; a2 = c2; c2 = tt; }
      const double num = b2 + c2 - a2;
      const double cos2 = (num * num) / (4.0 * b2 * c2);
      if (num > 0.0 && cos2 > M.gc2) nbad++;
    }
  }
  return nbad;
}

// Training rows: features and target t of every learned-placement candidate
// among the bad triangles (centers hold the plain points).
GQM_KERNEL void k_collect(Mesh M, const int *bad, const int *dn, const double2 *center, float *feat, float *target,
                          unsigned long long *count, unsigned long long cap) {
  const int n = *dn;
  GS_LOOP(k, n) {
    const int t = bad[k];
    const int4 v = M.tv[t];
    const double2 coff = center[k];
    const double2 cc = circumcenter(M.pts[v.x], M.pts[v.y], M.pts[v.z], 0.0, false);
    if (coff.x == cc.x && coff.y == cc.y) continue;
    int best = 1 << 30, bj = 0;
    for (int j = 0; j <= 8; ++j) {
      const double tj = j / 8.0;
      const double2 p = make_double2(coff.x + tj * (cc.x - coff.x), coff.y + tj * (cc.y - coff.y));
      if (j > 0 && encroaches_near(M, t, p)) continue;
      const int c = star_bad_count(M, t, p);
      if (c < best) {  // a point beyond the off-center only when it is strictly better
        best = c;
        bj = j;
      }
    }
    const unsigned long long row = atomicAdd(count, 1ull);
    if (row >= cap) continue;
    const Bisector B = bisector_of(M, t);
    features_of(M, t, B, 0.0, feat + row * kFeat);
    target[row] = bj / 8.0f;
  }
}

// ---------------------------------------------------------------------------
// Exploration runs for descendant-count labels (gqm_learn_explore).  Every
// bad triangle's candidate gets one row; the candidate inserts its point at
// t = j / (levels - 1) of the way from the off-center to the circumcenter, j
// drawn from a seeded hash of the triangle's vertices.  Lineage: every vertex
// inserted during the run carries the row of the candidate it descends from
// (vrow); a candidate's parent is the youngest such row among its bad
// triangle's vertices (the vertex whose insertion, directly or through the
// flips that followed it, made the triangle), and a midpoint descends from the
// youngest row among the vertices of the two triangles on its subsegment (the
// encroaching vertex is the apex of one of them).
// ---------------------------------------------------------------------------
struct ExploreDev {
  float *feat;     // [cap][kFeat]
  int *level;      // level j drawn (-1: off-center and circumcenter coincide)
  float *tused;    // t of the inserted point (0 when the drawn point would encroach)
  int *parent;     // parent row or -1
  uint8_t *ins;    // 1 once the candidate's point is in the mesh
  int *mids;       // midpoints that descend from the row directly
  unsigned long long *cnt;
  unsigned long long cap;
  int *vrow;       // per vertex slot: row it descends from (-1: input vertex)
  int *crow;       // per bad-list position: the candidate's row (-1: beyond cap)
  int *mlin;       // per midpoint position: its lineage, between the two kernels around k_insert_mid
  int levels;
  unsigned seed;
  // exploration around a network: with probability 1 - eps (per triangle,
  // from the same hash) the candidate takes the network's t (level -2)
  MlpDev net;
  int use_net;
  float eps;
};

// murmur3's 32-bit finaliser over the seed and the sorted vertex ids
__device__ __forceinline__ unsigned explore_mix(unsigned h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}
__device__ __forceinline__ unsigned explore_draw(unsigned seed, int a, int b, int c) {
  int lo = min(a, min(b, c)), hi = max(a, max(b, c)), mid = a + b + c - lo - hi;
  unsigned h = explore_mix(seed ^ 0x9e3779b9u);
  h = explore_mix(h ^ (unsigned)lo);
  h = explore_mix(h ^ (unsigned)mid);
  return explore_mix(h ^ (unsigned)hi);
}
__device__ __forceinline__ int explore_youngest(const int *vrow, int4 v) {
  return max(vrow[v.x], max(vrow[v.y], vrow[v.z]));
}

// after k_circumcenter: rows of the candidates, the drawn points into center
GQM_KERNEL void k_explore_place(Mesh M, const int *bad, const int *dn, double2 *center, ExploreDev E) {
  const int n = *dn;
  GS_LOOP(k, n) {
    const int t = bad[k];
    const int4 v = M.tv[t];
    const double2 coff = center[k];
    const double2 cc = circumcenter(M.pts[v.x], M.pts[v.y], M.pts[v.z], 0.0, false);
    const bool cand = (coff.x != cc.x || coff.y != cc.y);
    float f[kFeat];
    for (int q = 0; q < kFeat; ++q) f[q] = 0.0f;
    if (cand) features_of(M, t, bisector_of(M, t), 0.0, f);
    int j = -1;
    float tu = 0.0f;
    if (cand) {
      const unsigned h = explore_draw(E.seed, v.x, v.y, v.z);
      double tj = 0.0;
      if (E.use_net && (float)(explore_mix(h) >> 8) * (1.0f / 16777216.0f) >= E.eps) {
        j = -2;
        const float y = mlp_forward_row(E.net, f);
        tj = (y > 0.0f && y < 1.0f) ? (double)y : 0.0;
      } else {
        j = (int)(h % (unsigned)E.levels);
        tj = (double)j / (double)(E.levels - 1);
      }
      if (tj > 0.0) {
        const double2 p = make_double2(coff.x + tj * (cc.x - coff.x), coff.y + tj * (cc.y - coff.y));
        if (!encroaches_near(M, t, p)) {
          center[k] = p;
          tu = (float)tj;
        }
      }
    }
    const unsigned long long row = atomicAdd(E.cnt, 1ull);
    E.crow[k] = row < E.cap ? (int)row : -1;
    if (row >= E.cap) continue;
    for (int q = 0; q < kFeat; ++q) E.feat[row * kFeat + q] = f[q];
    E.level[row] = j;
    E.tused[row] = tu;
    E.parent[row] = explore_youngest(E.vrow, v);
    E.ins[row] = 0;
    E.mids[row] = 0;
  }
}

// after k_insert_steiner: the inserted points take their candidates' rows
// (a winner on a subsegment is not inserted and leaves its slot deleted)
template <class S>
GQM_KERNEL void k_explore_steiner(Mesh M, const int *wl, const int *dn, const double2 *center, S pslots_,
                                  ExploreDev E) {
  const int *pslots = slots_of(pslots_);
  const int n = *dn;
  GS_LOOP(pos, n) {
    const int k = wl[pos];
    const int newp = pslots[pos];
    if (M.ps[newp] != (PS_STEINER | PS_NEW)) continue;
    const double2 p = M.pts[newp], c = center[k];
    if (p.x != c.x || p.y != c.y) continue;
    const int row = E.crow[k];
    E.vrow[newp] = row;
    if (row >= 0) E.ins[row] = 1;
  }
}

// after k_mid_snapshot, before k_insert_mid: each midpoint's lineage
GQM_KERNEL void k_explore_mid_pre(Mesh M, const int *dn, const int *snap, ExploreDev E) {
  const int n = *dn;
  GS_LOOP(pos, n) {
    const int otri = snap[pos];
    const int t0 = dtri(otri);
    int lin = -1;
    if (t0 >= 0) {
      lin = explore_youngest(E.vrow, M.tv[t0]);
      const int on = ld1(M.tn, t0, dori(otri));
      if (on >= 0) lin = max(lin, explore_youngest(E.vrow, M.tv[dtri(on)]));
    }
    E.mlin[pos] = lin;
  }
}

// after k_insert_mid: the inserted midpoints take their lineage
template <class S>
GQM_KERNEL void k_explore_mid_post(Mesh M, const int *mids, const int *dn, S pslots_, ExploreDev E) {
  const int *pslots = slots_of(pslots_);
  const int n = *dn;
  GS_LOOP(pos, n) {
    const int newp = pslots[mids[pos]];
    if (M.ps[newp] != (PS_STEINER | PS_NEW | PS_SEGSPLIT)) continue;
    const int lin = E.mlin[pos];
    E.vrow[newp] = lin;
    if (lin >= 0) atomicAdd(E.mids + lin, 1);
  }
}

}  // namespace gqm
