// The whole refinement of one domain on the device, by one team of thread
// blocks.
//
// GPU_Refine_Quality's control flow (GPU_Refine/refine.cu:6500-7139, with its
// free-slot bookkeeping, refine.cu:149-197, 3408-3444, 3545-3562, 5259-5296,
// 5354-5368) runs in every thread of the team on the same scalars: counts come
// from team-wide compactions or from words written before a team barrier.  The
// pipeline's steps are the kernels of kernels.cuh compiled in CTA mode, striding
// over the domain's items with all the team's threads, and a barrier stands
// between two steps: __syncthreads() for a team of one block, a barrier in
// global memory (GridTeam) for several.
//
// batch.cu runs it on thousands of domains in one launch, and on one domain in
// the single-domain engine's own buffers.
#pragma once
#include "kernels.cuh"

namespace gqm {

// Capacities of one domain: the logical capacity starts as in the
// single-domain path (refine.cu:6543-6544: pointblock = (int)(0.5 N),
// triblock = 2 pointblock), the physical sizes are the buffers'.
struct Caps {
  long pointblock, triblock, pphys, tphys, sphys, cav_cap, hsz;
};
// Scratch of one domain: carved from its team's arena, or the single-domain
// engine's own buffers.
struct Scratch {
  Mesh M;
  int *emptyt, *bad, *imark, *ilist, *sinks, *wl, *newidx, *tail;
  int *emptyp, *pnew, *enclist, *encl2, *smark, *mids, *snap, *cav, *cavn;
  FlipLists fl;
  double2 *center;
  unsigned long long *hkeys;
  int *hvals, *s2ti;
};
// What the single-domain engine asks and learns of a run on its buffers.
struct EngineRun {
  const double2 *pts;
  const int *tri, *nbr;
  const int2 *seg;
  int np, nt, ns;
  int offcenter, offconstant, mode, pred, placement;
  MlpDev mlp;
  double theta, max_area;
  long long max_rounds;
  // results
  int status, need_grow, out_np, out_nt, out_ns, rounds;
  int last_point, last_triangle;
  long long bad_total;
  unsigned long long ctr[6];  // Steiner points, midpoints, -, -, learned candidates, learned points
  double goodcos2;
};

constexpr int kMaxTeam = 160;  // most blocks of a team
// Flip steps of at most this many queued triangles are run by the first block
// of a larger team (GQM_SMALL_STEP of refine.cu, for the same reason).
constexpr int kTeamSmallLimit = 256;
// State that the blocks of a team share, in global memory (or in the block's
// shared memory where the team is one block).
struct TeamState {
  FlipCtl fc;
  GridBar bar;
  unsigned long long ctr[6];
  double gc[2];
  int err;
  int job;
  int part[2][kMaxTeam];  // per-block counts of a compaction, by parity
  int stop[2];            // the error word as a compaction found it, by parity
};
// One block's own.
struct BlockState {
  Scratch S;
  SmallLists small;
  int cnt[4];
  int wsum[33];
  int stop;  // a team of one block's ts.stop
};

#ifdef GQM_CTA_MODE  // the steps as functions of a team
// predicates and maps of the compactions (the same as refine.cu's)
struct Ident {
  __device__ int operator()(int i) const { return i; }
};
struct ValueOf {
  const int *a;
  __device__ int operator()(int i) const { return a[i]; }
};
struct PNonNeg {
  const int *a;
  __device__ bool operator()(int i) const { return a[i] >= 0; }
};
struct PBad {
  const uint8_t *tst;
  __device__ bool operator()(int i) const { return (tst[i] & (TS_NOTNULL | TS_BAD)) == (TS_NOTNULL | TS_BAD); }
};
struct PTriNull {
  const uint8_t *tst;
  __device__ bool operator()(int i) const { return !(tst[i] & TS_NOTNULL); }
};
struct PTriLive {
  const uint8_t *tst;
  __device__ bool operator()(int i) const { return (tst[i] & TS_NOTNULL) != 0; }
};
struct PPtDeleted {
  const uint8_t *ps;
  __device__ bool operator()(int i) const { return (ps[i] & PS_DELETED) != 0; }
};
struct PPtLive {
  const uint8_t *ps;
  __device__ bool operator()(int i) const { return !(ps[i] & PS_DELETED); }
};

enum { C_LIST0 = 0, C_LIST1, C_LIST2, C_MISC };

// a barrier of the team; a function that returns a status leaves when one broke
#define TSYNC()                             \
  do {                                      \
    if (!T.sync()) return GQM_ERR_TOPOLOGY; \
  } while (0)

template <int PRED>
struct Engine {
  BlockState &sh;
  TeamState &ts;
  GridTeam T;
  KTimer *ktm, *stm;
  int small_limit;
  Caps c;
  long pcap, tcap;
  int last_point, last_triangle, last_subseg;
  int nempty_p, nempty_t, lenp, lent;
  int offcenter, offconstant, placement, need_grow;
  MlpDev mlp;
  long long max_rounds;
  int parity;
  int rounds;
  long long bad_total;

  __device__ bool lead() const { return T.lead(); }
  template <class V>
  __device__ void fill(V *a, long n, V v) {
    for (long i = T.tid(); i < n; i += T.size()) a[i] = v;
  }
  __device__ void copy(int *dst, const int *src, int n) {
    for (int i = T.tid(); i < n; i += T.size()) dst[i] = src[i];
  }
  // Ordered compaction: out[k] = map(i) for the k-th i in [lo, hi) with pred(i),
  // ascending; *count gets the number (the same in every thread).  A thread
  // takes 16 consecutive elements of a tile.  A range of one tile is the lead
  // block's work (one barrier); a longer one is cut into a chunk per block,
  // counted, and emitted behind the counts of the blocks before (two).
  // Returns GQM_OK, the barrier's failure, or the error that a step before it
  // has recorded: every loop of the refinement compacts in each of its rounds,
  // and none goes on with a mesh that was found inconsistent.
  template <class F, class Mp>
  __device__ __noinline__ int compact(F f, Mp m, int lo, int hi, int *out, int *count) {
#ifdef GQM_HOST_EMU
    int *part = ts.part[parity], *stop = ts.stop + parity;
    parity ^= 1;
    if (T.rank == 0) {
      *stop = ts.err;
      part[0] = 0;
      for (int i = lo; i < hi; ++i)
        if (f(i)) out[part[0]++] = m(i);
    }
    TSYNC();
    *count = part[0];
    return *stop;
#else
    constexpr int kItems = 16;
    const int tile = (int)blockDim.x * kItems, n = hi - lo;
    const bool one = T.nb == 1 || n <= tile;
    const int rank = (int)T.rank;
    int *part = ts.part[parity], *stop = T.nb == 1 ? &sh.stop : ts.stop + parity;
    parity ^= 1;
    int b0 = lo, b1 = hi, base = 0;
    const int err = T.lead() ? vload(&ts.err) : 0;  // its latency passes under the compaction's own loads
    if (!one) {
      const int chunk = ((n + T.nb - 1) / T.nb + kItems - 1) / kItems * kItems;
      b0 = min(hi, lo + rank * chunk);
      b1 = min(hi, b0 + chunk);
      int k = 0;
      for (int s = b0 + (int)threadIdx.x * kItems; s < b1; s += tile) {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
          if (s + j < b1 && f(s + j)) ++k;
      }
      for (int o = 16; o > 0; o >>= 1) k += __shfl_down_sync(0xffffffffu, k, o);
      if ((threadIdx.x & 31) == 0) sh.wsum[threadIdx.x >> 5] = k;
      __syncthreads();
      if (threadIdx.x < 32) {
        int v = threadIdx.x < (blockDim.x >> 5) ? sh.wsum[threadIdx.x] : 0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) part[rank] = v;
      }
      TSYNC();
      if (threadIdx.x < 32) {
        int before = 0, all = 0;
        for (int r = (int)threadIdx.x; r < T.nb; r += 32) {
          const int v = vload(part + r);
          all += v;
          before += r < rank ? v : 0;
        }
        for (int o = 16; o > 0; o >>= 1) {
          all += __shfl_down_sync(0xffffffffu, all, o);
          before += __shfl_down_sync(0xffffffffu, before, o);
        }
        if (threadIdx.x == 0) {
          sh.wsum[31] = before;
          sh.wsum[32] = all;
        }
      }
      __syncthreads();
      base = sh.wsum[31];
      *count = sh.wsum[32];
      __syncthreads();
    }
    if (T.lead()) *stop = err;
    if (!one || rank == 0) {
      const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5);
      for (int t0 = b0; t0 < b1; t0 += tile) {
        const int s = t0 + (int)threadIdx.x * kItems;
        unsigned bits = 0;
#pragma unroll
        for (int j = 0; j < kItems; ++j)
          if (s + j < b1 && f(s + j)) bits |= 1u << j;
        const int k = __popc(bits);
        int x = k;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (lane == 31) sh.wsum[warp] = x;
        __syncthreads();
        int woff = 0, tot = 0;
        for (int w = 0; w < nw; ++w) {
          const int v = sh.wsum[w];
          woff += w < warp ? v : 0;
          tot += v;
        }
        int pos = base + woff + x - k;
        while (bits) {
          const int j = __ffs(bits) - 1;
          bits &= bits - 1;
          out[pos++] = m(s + j);
        }
        base += tot;
        __syncthreads();
      }
      if (one) {
        *count = base;
        if (T.nb > 1 && threadIdx.x == 0) part[0] = base;
      }
    }
    TSYNC();
    if (one && T.nb > 1) *count = vload(part);
    return vload(stop);
#endif
  }
  // the device error word, read by every thread before anyone can change it
  // again (the barrier keeps the team's decision on it uniform)
  __device__ int read_err() {
    const int e = vload(&ts.err);
    return T.sync() ? e : GQM_ERR_TOPOLOGY;
  }
  // a count that the next step reads through a pointer (every block its own copy)
  __device__ int *publish(int slot, int v) {
    if (threadIdx.x == 0) sh.cnt[slot] = v;
    __syncthreads();
    return sh.cnt + slot;
  }

  // updateEmptyPoints / updateEmptyTriangles (refine.cu:149-197)
  __device__ int refresh_points() {
    const int rc = compact(PPtDeleted{sh.S.M.ps}, Ident{}, 0, (int)pcap, sh.S.emptyp, &lenp);
    nempty_p = lenp;
    return rc;
  }
  __device__ int refresh_tris() {
    const int rc = compact(PTriNull{sh.S.M.tst}, Ident{}, 0, (int)tcap, sh.S.emptyt, &lent);
    nempty_t = lent;
    return rc;
  }
  // the winners' bitmap covers the triangle slots in use, as nothing else of a
  // run depends on how large its buffers have become
  __device__ void size_winners() {
    if (threadIdx.x == 0) winner_carve(sh.S.fl, sh.S.fl.wbits, tcap);
    __syncthreads();
  }
  // growth steps of refine.cu:3408-3444 / 5259-5296 on the logical capacity
  __device__ __noinline__ int ensure_slots(int npts, int ntris) {
    if (npts > nempty_p) {
      int rc = refresh_points();
      if (rc) return rc;
      if (npts > nempty_p && c.pointblock <= 0) return GQM_ERR_ARGUMENT;
      long num = 0;
      while (npts > nempty_p + num * c.pointblock) num++;
      if (num) {
        long ncap = pcap + num * c.pointblock;
        if (ncap > c.pphys) {
          need_grow |= 1;
          return GQM_ERR_ARENA;
        }
        for (long i = pcap + T.tid(); i < ncap; i += T.size()) clear_point(sh.S.M, (int)i);
        TSYNC();
        pcap = ncap;
        rc = refresh_points();
        if (rc) return rc;
      }
    }
    if (ntris > nempty_t) {
      int rc = refresh_tris();
      if (rc) return rc;
      if (ntris > nempty_t && c.triblock <= 0) return GQM_ERR_ARGUMENT;
      long num = 0;
      while (ntris > nempty_t + num * c.triblock) num++;
      if (num) {
        long ncap = tcap + num * c.triblock;
        if (ncap > c.tphys) {
          need_grow |= 2;
          return GQM_ERR_ARENA;
        }
        for (long i = tcap + T.tid(); i < ncap; i += T.size()) clear_tri(sh.S.M, (int)i);
        TSYNC();
        tcap = ncap;
        size_winners();
        rc = refresh_tris();
        if (rc) return rc;
      }
    }
    return GQM_OK;
  }
  // slot bookkeeping after an insertion batch (refine.cu:3545-3559, 5354-5368)
  __device__ void consume_slots(int npts, int ntris) {
    int slot_after = (int)(pcap - last_point);
    int slot_before = nempty_p - slot_after;
    if (slot_before < npts) last_point += npts - slot_before;
    nempty_p -= npts;
    slot_after = (int)(tcap - last_triangle);
    slot_before = nempty_t - slot_after;
    if (slot_before < ntris) last_triangle += ntris - slot_before;
    nempty_t -= ntris;
  }
  __device__ const int *pslots() const { return sh.S.emptyp + (lenp - nempty_p); }
  __device__ const int *tslots() const { return sh.S.emptyt + (lent - nempty_t); }

  // ---- flip-flop (refine.cu:2328-2490) ----
  __device__ __noinline__ int flip_flop() {
    return flip_loop<PRED>(sh.S.M, sh.S.fl, sh.small, T, small_limit, nullptr, ktm, stm) ? GQM_OK : GQM_ERR_TOPOLOGY;
  }

  // ---- splitEncsegs (refine.cu:3180-3778) ----
  __device__ __noinline__ int split_encsegs() {
    Scratch &S = sh.S;
    long long outer = 0;
    for (;;) {
      int nenc = 0;
      int rc = compact(PNonNeg{S.M.enc}, Ident{}, 0, last_subseg, S.enclist, &nenc);
      if (rc) return rc;
      if (nenc == 0) break;
      if (++outer > max_rounds) return GQM_ERR_ROUND_LIMIT;
      // delete free Steiner points inside diametral circles
      copy(S.smark, S.enclist, nenc);
      TSYNC();
      int nmark = nenc;
      long long inner = 0;
      for (;;) {
        int ndel = 0;
        rc = compact(PNonNeg{S.smark}, ValueOf{S.smark}, 0, nmark, S.mids, &ndel);
        if (rc) return rc;
        if (ndel == 0) break;
        if (++inner > max_rounds) return GQM_ERR_ROUND_LIMIT;
        nmark = ndel;
        k_mark_redundant(S.M, S.smark, S.mids, publish(C_LIST1, ndel), S.fl);
        TSYNC();
        rc = flip_flop();
        if (rc) return rc;
      }
      rc = ensure_slots(nenc, 2 * nenc);
      if (rc) return rc;
      if (last_subseg + nenc > c.sphys) {
        need_grow |= 4;
        return GQM_ERR_ARENA;
      }
      fill(S.M.enc + last_subseg, nenc, -1);
      fill(S.M.s2t + last_subseg, nenc, (s2t_t)0);  // epoch 0: any store wins
      copy(S.smark, S.enclist, nenc);
      TSYNC();
      long long mid_iter = 0;
      for (;;) {
        int nmid = 0;
        rc = compact(PNonNeg{S.smark}, Ident{}, 0, nenc, S.mids, &nmid);
        if (rc) return rc;
        if (nmid == 0) break;
        if (++mid_iter > 64 * max_rounds) return GQM_ERR_ROUND_LIMIT;
        int *dn = publish(C_LIST1, nmid);
        k_reset_mid(S.M, S.mids, dn, S.smark);
        TSYNC();
        k_mark_mid(S.M, S.mids, dn, S.smark);
        k_mid_snapshot(S.M, S.mids, dn, S.smark, S.snap);
        if (lead()) ts.fc.epoch++;
        TSYNC();
        k_insert_mid(S.M, S.mids, dn, S.smark, S.snap, pslots(), tslots(), last_subseg, S.fl, ts.ctr + 1);
        TSYNC();
        k_update_mid_nbrs(S.M, S.mids, dn, S.smark, S.enclist);
        TSYNC();
      }
      consume_slots(nenc, 2 * nenc);
      last_subseg += nenc;
      rc = flip_flop();
      if (rc) return rc;
    }
    return GQM_OK;
  }

  // ---- splitTriangles (refine.cu:5107-5547) ----
  __device__ __noinline__ int split_triangles(int nbad) {
    Scratch &S = sh.S;
    int *dn = publish(C_LIST2, nbad);
    if (nbad > c.cav_cap) {
      need_grow |= 8;
      return GQM_ERR_ARENA;
    }
    copy(S.imark, S.bad, nbad);
    copy(S.ilist, S.bad, nbad);
    k_circumcenter(S.M, S.bad, dn, (double)offconstant, offcenter, S.center);
    TSYNC();
    if (placement == GQM_PLACE_LEARNED) {
      k_learned_place(S.M, S.bad, dn, mlp, S.center, ts.ctr + 4);
      TSYNC();
    }
    k_locate<PRED>(S.M, S.bad, dn, S.center, S.sinks, S.fl);
    TSYNC();
    k_remove_losers(S.M, S.bad, dn, S.sinks, S.imark, S.fl);
    TSYNC();
    k_cavity_mark<PRED>(S.M, dn, S.sinks, S.center, S.imark, S.ilist, S.cav, S.cavn, nbad, S.fl);
    fill(S.encl2, last_subseg, -1);
    TSYNC();
    k_cavity_check(S.M, dn, S.cav, S.cavn, nbad, S.imark, S.ilist, S.fl);
    TSYNC();
    int nst = 0;
    int rc = compact(PNonNeg{S.imark}, Ident{}, 0, nbad, S.wl, &nst);
    if (rc) return rc;
    int *dw = publish(C_LIST1, nst);
    k_mark_onsegs(S.M, S.wl, dw, S.sinks, S.encl2);
    rc = ensure_slots(nst, 2 * nst);
    if (rc) return rc;
    k_reset_steiner(S.M, S.wl, dw, S.sinks);
    if (lead()) ts.fc.epoch++;
    TSYNC();
    k_insert_steiner(S.M, S.wl, dw, S.sinks, S.center, pslots(), tslots(), S.fl, ts.ctr + 0);
    TSYNC();
    k_update_steiner_nbrs(S.M, S.wl, dw, S.sinks);
    TSYNC();
    consume_slots(nst, 2 * nst);
    rc = flip_flop();
    if (rc) return rc;
    k_onsegs_to_enc(S.M, S.encl2, last_subseg);
    TSYNC();
    return GQM_OK;
  }

  // ---- output compaction (refine.cu:5758-6428) ----
  __device__ __noinline__ int compact_output(int *out_np, int *out_nt) {
    Scratch &S = sh.S;
    int newn = 0, nmove = 0, unused = 0;
    int rc = compact(PTriLive{S.M.tst}, Ident{}, 0, last_triangle, S.tail, &newn);
    if (rc) return rc;
    k_newidx_init(S.M, S.newidx, last_triangle, newn, S.M.tst, (uint8_t)TS_NOTNULL, false);
    TSYNC();
    if (newn < last_triangle) {
      rc = compact(PTriNull{S.M.tst}, Ident{}, 0, newn, S.emptyt, &unused);
      if (rc == GQM_OK) rc = compact(PTriLive{S.M.tst}, Ident{}, newn, last_triangle, S.tail, &nmove);
      if (rc) return rc;
      k_compact_tris_move(S.M, S.tail, S.emptyt, publish(C_LIST1, nmove), S.newidx);
      TSYNC();
      k_fix_nbrs(S.M, S.newidx, newn);
      k_fix_s2t(S.M, S.newidx, last_subseg);
      TSYNC();
    }
    int newp = 0;
    rc = compact(PPtLive{S.M.ps}, Ident{}, 0, last_point, S.pnew, &newp);
    if (rc) return rc;
    k_newidx_init(S.M, S.pnew, last_point, newp, S.M.ps, (uint8_t)PS_DELETED, true);
    TSYNC();
    if (newp < last_point) {
      rc = compact(PPtDeleted{S.M.ps}, Ident{}, 0, newp, S.emptyp, &unused);
      if (rc == GQM_OK) rc = compact(PPtLive{S.M.ps}, Ident{}, newp, last_point, S.tail, &nmove);
      if (rc) return rc;
      k_compact_pts_move(S.M, S.tail, S.emptyp, publish(C_LIST1, nmove), S.pnew);
      TSYNC();
      k_fix_tri_vertices(S.M, S.pnew, newn);
      TSYNC();
    }
    *out_np = newp;
    *out_nt = newn;
    return GQM_OK;
  }

  // ---- the whole refinement of one domain (Refiner::run): everything before
  // the output arrays.  In: a Job or an EngineRun. ----
  template <class In>
  __device__ int refine(const In &J, double theta, double *goodcos2) {
    Scratch &S = sh.S;
    const int np = J.np, nt = J.nt, ns = J.ns;
    offcenter = J.offcenter;
    offconstant = J.offconstant;
    placement = J.placement;
    mlp = J.mlp;
    max_rounds = J.max_rounds;
    pcap = np + c.pointblock;
    tcap = nt + c.triblock;
    parity = 0;
    rounds = 0;
    need_grow = 0;
    bad_total = 0;
    k_check_input(J.pts, np, J.tri, J.nbr, nt, reinterpret_cast<const int *>(J.seg), ns, &ts.err);
    if (lead()) k_goodcos(theta, ts.gc);
    TSYNC();
    if (const int e = read_err()) return e;
    if (threadIdx.x == 0) {
      S.M.gc2 = *(volatile double *)ts.gc;
      S.M.mode = J.mode;
      S.M.max_area = J.max_area;
      *goodcos2 = S.M.gc2;
    }
    __syncthreads();
    // The slots in use only; ensure_slots clears those that a growth step adds.
    // The buffers keep the size of the largest mesh that a context has refined:
    // cleared whole, they made 500 points take 18.2 ms on a context that had
    // refined 2,000,000, instead of the 4.1 ms on a fresh one.
    size_winners();
    k_init_points(S.M, J.pts, np, (int)pcap);
    k_init_tris(S.M, J.tri, J.nbr, nt, (int)tcap);
    fill(S.hkeys, c.hsz, ~0ull);
    fill(S.s2ti, (long)ns + 1, -1);
    TSYNC();
    // initSubsegs via a hash of segment endpoints
    k_seg_hash_insert(J.seg, ns, S.hkeys, S.hvals, (unsigned)(c.hsz - 1));
    TSYNC();
    k_init_subsegs(S.M, nt, S.hkeys, S.hvals, (unsigned)(c.hsz - 1), S.s2ti);
    TSYNC();
    k_pack_s2t(S.M, S.s2ti, ns);
    TSYNC();
    last_point = np;
    last_triangle = nt;
    last_subseg = ns;
    int rc = refresh_points();
    if (rc == GQM_OK) rc = refresh_tris();
    if (rc) return rc;
    k_mark_all_encsegs(S.M, ns);
    TSYNC();
    rc = split_encsegs();
    while (rc == GQM_OK) {
      k_mark_bad(S.M, last_triangle);
      TSYNC();
      int nbad = 0;
      rc = compact(PBad{S.M.tst}, Ident{}, 0, last_triangle, S.bad, &nbad);
      if (rc || nbad == 0) break;
      if (rounds >= max_rounds) {
        rc = GQM_ERR_ROUND_LIMIT;
        break;
      }
      bad_total += nbad;
      rc = split_triangles(nbad);
      if (rc == GQM_OK) rc = split_encsegs();
      if (rc) break;
      // no barrier between this step and the next: k_mark_bad reads other bits of
      // the status bytes than the one that is cleared here
      k_points_old(S.M, last_point);
      rounds++;
    }
    if (rc == GQM_ERR_TOPOLOGY) return rc;
    if (const int e = read_err()) rc = rc ? rc : e;
    return rc;
  }
};
#endif  // GQM_CTA_MODE

}  // namespace gqm
