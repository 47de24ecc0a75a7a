/*
 * Persistent graph kernels for sm_103a: Lonestar BFS/SSSP worklists and
 * Pannotia colour/MIS/SSSP frontier loops, plus pull PageRank, all running in
 * one discovery-sized persistent grid synchronised by wgm_barrier.
 *
 * Reference kernels and what changed (outputs are bit-identical; each change
 * is argued where it is made):
 *   lonestar/graph_apps/bfs/device/bfs.cl:104-302   -> wgm_app_lonestar<false>
 *   lonestar/graph_apps/sssp/device/sssp.cl:104-318 -> wgm_app_lonestar<true>
 *   pannotia/graph_apps/color/device/color.cl:3-97  -> wgm_app_color
 *   pannotia/graph_apps/mis/device/mis.cl:5-125     -> wgm_app_mis
 *   pannotia/graph_apps/sssp/device/sssp.cl:10-88   -> wgm_app_pannotia_sssp
 *   (no reference)                                  -> wgm_app_pagerank
 *
 * Edge work is warp-level.  A warp owns up to 32 vertices (one per lane),
 * scans their degrees with shuffles and walks the concatenated adjacency in
 * windows of 32 edges: lane j of a window handles edge slot w+j, its owner is
 * found with one __reduce_or_sync and a clz, so col[] is read coalesced and no
 * CTA-wide __syncthreads is needed inside the edge loop (the reference's
 * block scan is serial in work-item 0, bfs.cl:43-51).  Long rows never stall
 * a level: Lonestar rows are queued in pieces, colour spreads the edges of
 * vertices above `hub_threshold` over every warp, MIS hands rows past twice
 * that to the whole grid, and PageRank and Pannotia SSSP cut theirs into parts.
 *
 * Two habits of the memory system shape what follows (measured on GB300).
 * Words that many SMs read and write at once cost about 50 ns an access, so a
 * mark is stored once, a count or a minimum leaves a group once, and hot words
 * are read through the L1 (a barrier's acquire empties it).  And a dependent
 * access costs 305 cycles from the L2 (an atomic 707) against 28 from shared
 * memory, so short phases are counted in round trips.
 */
#ifndef WGM_GRAPH_CUH
#define WGM_GRAPH_CUH

#include "wgm_device.cuh"

#define WGM_LONESTAR_INF 1000000000u /* bfs.cl:33 */
#define WGM_PANNOTIA_BIG 99999999    /* pannotia sssp.h:3, mis.cl:1 */
#define WGM_MAX_WARPS 32

/* Per-CTA shared scratch of the edge-window walker. */
struct wgm_warp_smem {
  int tab[WGM_MAX_WARPS][32];
  int acc[WGM_MAX_WARPS][32];
};

/* Walk the edge slots [w0, total) of a warp's concatenated adjacency in
 * windows of 32, window stride `wstep`.  Each lane passes its own range as
 * (off = exclusive prefix, deg, base = row start - off).  f(valid, edge,
 * owner_lane) is called by all 32 lanes once per window. */
template <class F>
__device__ __forceinline__ void wgm_for_each_edge(int off, int deg, int base, int total,
                                                  int w0, int wstep, int *tab, F &&f) {
  const int lane = wgm_lane();
  for (int w = w0; w < total; w += wstep) {
    bool in = deg > 0 && off < w + 32 && off + deg > w;
    int pos = in ? max(off - w, 0) : 0;
    unsigned mask = __reduce_or_sync(WGM_FULL, in ? (1u << pos) : 0u);
    if (in) tab[pos] = lane;
    __syncwarp();
    unsigned upto = (lane == 31) ? 0xffffffffu : ((2u << lane) - 1u);
    unsigned mm = mask & upto;
    int owner = tab[mm ? 31 - __clz(mm) : 0] & 31;
    __syncwarp();
    int eb = __shfl_sync(WGM_FULL, base, owner);
    int slot = w + lane;
    f(slot < total, eb + slot, owner);
  }
}

/* Static hub layout (host-built): hub ids, their edge prefix and, for each
 * window of 32 hub-edge slots, a 16-byte record {first hub h0, edge of the
 * window's first slot, slots belonging to h0, first edge of hub h0+1}.  Hubs
 * have degree > 32, so a window touches at most two consecutive hubs, and
 * one load of the record gives every lane its hub and edge. */
struct wgm_hubs {
  const int *ids;    /* [H] */
  const int *prefix; /* [H+1] */
  const int *wmap;   /* [4 * ceil(prefix[H]/32)] window records */
  int H;
  int total;
};

/* Hub and edge of this lane's slot in window k. */
__device__ __forceinline__ void wgm_hub_slot(const int4 &w, int lane, int *h, int *e) {
  const bool first = lane < w.z;
  *h = first ? w.x : w.x + 1;
  *e = first ? w.y + lane : w.w + (lane - w.z);
}

/* Calls f(valid, hub_index, edge) for one window of hub edges. */
template <class F>
__device__ __forceinline__ void wgm_hub_window(const wgm_hubs &hb, const int *row, int k,
                                               F &&f) {
  const int lane = wgm_lane();
  const bool valid = k * 32 + lane < hb.total;
  const int4 w = __ldg(reinterpret_cast<const int4 *>(hb.wmap) + k);
  int h, e;
  wgm_hub_slot(w, lane, &h, &e);
  (void)row;
  f(valid, h, e);
}

/* First edge of each lane's row [e, end) that `hit` accepts (warp-collective;
 * hit(valid, target, owner lane) is called by every lane).  Each lane first
 * looks at four edges of its own row, then the warp shares the rows still
 * open, 128 edges a step, split evenly among them.  At most `scan` edges of a
 * row past its first four are looked at: `wide` tells that some are left.
 * Returns whether the lane has its edge, at e; otherwise e is the first edge
 * not looked at. */
template <class Hit>
__device__ __forceinline__ bool wgm_first_edge(const int *col, bool act, int &e, int end, int scan,
                                               bool &wide, int *tab, Hit &&hit) {
  const int lane = wgm_lane();
  bool found = false;
  {
    int j[4];
    bool h[4];
#pragma unroll
    for (int q = 0; q < 4; q++) j[q] = act && q < end - e ? __ldg(&col[e + q]) : -1;
#pragma unroll
    for (int q = 0; q < 4; q++) h[q] = hit(act && q < end - e, j[q], lane);
    if (act) {
      const int e0 = e;
#pragma unroll
      for (int q = 3; q >= 0; q--)
        if (h[q]) {
          found = true;
          e = e0 + q;
        }
      if (!found) e += min(4, end - e);
    }
  }
  wide = false;
  const int elim = end - e > scan ? e + scan : end;
  unsigned open = __ballot_sync(WGM_FULL, act && !found && e < end);
  while (open) {
    const int nopen = __popc(open);
    const int ql = 31 - __clz(128 / nopen), quota = 1 << ql; /* 4 ... 128 */
    const bool mine = (open >> lane) & 1u;
    const int rank = __popc(open & wgm_lanemask_lt());
    if (mine) tab[rank] = lane;
    __syncwarp();
    int j[4], own[4];
    unsigned in = 0, h[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int sl = 32 * q + lane, oi = sl >> ql;
      own[q] = oi < nopen ? tab[oi] : 0;
      const int oe = __shfl_sync(WGM_FULL, e, own[q]), x = sl & (quota - 1);
      const int lim = __shfl_sync(WGM_FULL, elim, own[q]);
      const bool v = oi < nopen && x < lim - oe;
      j[q] = v ? __ldg(&col[oe + x]) : -1;
      in |= v ? 1u << q : 0u;
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
      h[q] = __ballot_sync(WGM_FULL, hit((in >> q) & 1u, j[q], own[q]));
    if (mine) {
      /* this row's slots are [rank * quota, (rank + 1) * quota) */
      const int s0 = rank << ql, w0 = s0 >> 5;
      unsigned x = w0 == 0 ? h[0] : w0 == 1 ? h[1] : w0 == 2 ? h[2] : h[3];
      int f = -1;
      if (ql < 5) x = (x >> (s0 & 31)) & ((1u << quota) - 1u);
      if (x) f = __ffs(x) - 1;
      if (ql >= 6 && f < 0) { /* 64 or 128 slots */
        const unsigned x1 = w0 == 0 ? h[1] : h[3];
        if (x1) f = 31 + __ffs(x1);
        if (ql == 7 && f < 0 && h[2]) f = 63 + __ffs(h[2]);
        if (ql == 7 && f < 0 && h[3]) f = 95 + __ffs(h[3]);
      }
      found = f >= 0;
      e = found ? e + f : e + min(quota, elim - e);
      wide = !found && e == elim && elim < end;
    }
    __syncwarp();
    open = __ballot_sync(WGM_FULL, mine && !found && e < elim);
  }
  return found;
}

/* ------------------------------------------------------------------------ */
/* Lonestar BFS / SSSP                                                       */
/* ------------------------------------------------------------------------ */

struct wgm_lonestar_args {
  int V;
  const int *row; /* [V+1]; row[V] may be row[V-1]-1 (Lonestar loader quirk) */
  const int *col;
  const unsigned *wt; /* SSSP weights, nullptr for BFS */
  unsigned *dist;     /* [V] output */
  /* Two worklists of `cap` pieces each, structure of arrays: a piece is up
   * to `piece` consecutive edges of one vertex. */
  int *wl_start; /* [2][cap] first edge of the piece */
  int *wl_cnt;   /* [2][cap] number of edges */
  int *wl_u;     /* [2][cap] the vertex (SSSP reads its distance); may be null for BFS */
  int cap;       /* >= V + E/piece, so no level can overflow */
  int piece;     /* edges per piece (>= 32) */
  int *cnt;      /* [3 lines]: pieces queued for each level, by level mod 3 */
  int *stamp;    /* SSSP: level a vertex was last queued at, or (packed) [2V] the
                    64-bit {level tag, distance} words, dist[] written at the end */
  int source;
  int *levels_out; /* number of levels run (written by group 0) */
  int packed = 0;  /* SSSP relaxes packed words (wgm_ls_chunk PACK) */
  int low_degree = 0; /* SSSP: average degree at most 8, no hubs (wgm_ls_narrow) */
  int *grab = nullptr; /* [3 lines] chunks of a wide level handed out, by level mod 3 */
};

/* Degree as the Lonestar kernel sees it: psrc[nn+1]-psrc[nn] (bfs.cl:165);
 * the loader quirk can make the last vertex -1, which walks no edges. */
__device__ __forceinline__ int wgm_ls_degree(const int *row, int v) {
  return max(__ldg(&row[v + 1]) - __ldg(&row[v]), 0);
}

/* Relaxation rules of one edge from a vertex at distance dsrc, at level L
 * (applied by wgm_ls_chunk):
 * BFS (bfs.cl:115-125): dist[dst]==MYINFINITY -> dist[dst]=level; the
 *   reference's unsynchronised store becomes a CAS so each vertex is queued
 *   exactly once (the stored value is identical: the level).
 * SSSP (sssp.cl:115-131): altdist = dist[src]+wt; if smaller, atomic_min and
 *   queue dst; a per-level stamp queues a vertex at most once per level (its
 *   next visit reads the final dist of the level, so the fixpoint - the
 *   shortest-path vector - is unchanged).
 * Destinations outside [0, V) and weights >= MYINFINITY are skipped
 * (bfs.cl:116, sssp.cl:120). */

/* Queue the flagged lanes' vertices as pieces (warp-aggregated: one atomic
 * per warp, __ballot_sync/__popc/__shfl_sync inside the scan and window
 * walk).  A vertex with no out-edges is not queued: its level or distance is
 * already written and it has nothing to relax.  Pieces are written by the
 * whole warp, one piece per lane per window, so the stores are coalesced. */
__device__ __forceinline__ bool wgm_ls_push(const wgm_lonestar_args &a, bool flag, int u,
                                            int *counter, int *o_start, int *o_cnt, int *o_u,
                                            int *tab) {
  int start = 0, deg = 0, np = 0;
  if (flag) {
    start = __ldg(&a.row[u]);
    deg = wgm_ls_degree(a.row, u);
    np = (deg + a.piece - 1) / a.piece;
  }
  int incl = wgm_warp_incl_scan(np);
  int total = __shfl_sync(WGM_FULL, incl, 31);
  if (total == 0) return true;
  int base = 0;
  if (wgm_lane() == 0) base = atomicAdd(counter, total);
  base = __shfl_sync(WGM_FULL, base, 0);
  if (base + total > a.cap) return false;
  int off = incl - np;
  const int P = a.piece;
  wgm_for_each_edge(off, np, -off, total, 0, 32, tab, [&](bool valid, int k, int owner) {
    /* k: piece index of `owner`'s vertex; slot = its position in the list */
    int s = __shfl_sync(WGM_FULL, start, owner);
    int d = __shfl_sync(WGM_FULL, deg, owner);
    int v = __shfl_sync(WGM_FULL, u, owner);
    int o = __shfl_sync(WGM_FULL, off, owner);
    if (valid) {
      int slot = base + o + k;
      o_start[slot] = s + k * P;
      o_cnt[slot] = min(P, d - k * P);
      if (o_u) o_u[slot] = v;
    }
  });
  return true;
}

/* Owner lane of edge slot s in a warp's concatenated ranges: the last lane
 * whose exclusive offset is <= s, by binary search over shuffles.  A lane with
 * no edges shares its successor's offset, so the search always lands on the
 * lane whose range [off, off+deg) holds s (for 0 <= s < total). */
__device__ __forceinline__ int wgm_owner_of(int off, int s) {
  int j = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    int o = __shfl_sync(WGM_FULL, off, j + step);
    if (o <= s) j += step;
  }
  return j;
}

/* Worklist a chunk pushes to.  The piece count lives in `counter`, or,
 * when `counter64` is set, in the low half of a 64-bit level word whose
 * high half counts a team's barrier arrivals.  With `far_cnt` set (packed
 * SSSP, near-far schedule) an improved vertex whose new distance is at or
 * above `T` goes to the far list as a vertex id instead of the next level
 * as pieces; `far_min` keeps the least distance stored there. */
struct wgm_ls_out {
  int *counter; /* pieces queued so far (global or shared memory) */
  unsigned long long *counter64 = nullptr;
  int *o_start, *o_cnt, *o_u;
  int cap;
  int *far_cnt = nullptr;
  unsigned *far_min = nullptr;
  int *far_list = nullptr;
  int far_cap = 0;
  unsigned T = 0xffffffffu;
  /* SSSP: relax only edges of weight in [wlo, whi) (batched near-far with
   * heavy edges deferred; the defaults relax every edge) */
  unsigned wlo = 0, whi = 0xffffffffu;
};

/* Store one piece at list slot `slot`. */
__device__ __forceinline__ void wgm_out_put(const wgm_ls_out &o, int slot, int start, int cnt,
                                            int u) {
  o.o_start[slot] = start;
  o.o_cnt[slot] = cnt;
  if (o.o_u) o.o_u[slot] = u;
}

/* Reserve n slots of the output list; returns the first. */
__device__ __forceinline__ int wgm_out_reserve(const wgm_ls_out &o, int n) {
  if (o.counter64) return (int)(unsigned)atomicAdd(o.counter64, (unsigned long long)n);
  return atomicAdd(o.counter, n);
}

/* Queue the flagged lanes' vertices (with out-edges) as pieces of size P
 * (warp-collective; each lane writes its own pieces).  False when the list
 * is full. */
__device__ __forceinline__ bool wgm_out_push_vertices(const int *row, int P, bool flag, int u,
                                                      const wgm_ls_out &o) {
  int rs = 0, dg = 0, np = 0;
  if (flag) {
    rs = __ldg(&row[u]);
    dg = max(__ldg(&row[u + 1]) - rs, 0);
    np = (dg + P - 1) / P;
  }
  const int incl = wgm_warp_incl_scan(np);
  const int total = __shfl_sync(WGM_FULL, incl, 31);
  if (total == 0) return true;
  int base = 0;
  if (wgm_lane() == 31) base = wgm_out_reserve(o, total);
  base = __shfl_sync(WGM_FULL, base, 31);
  if (base + total > o.cap) return false;
  const int s = base + incl - np;
  for (int q = 0; q < np; q++) wgm_out_put(o, s + q, rs + q * P, min(P, dg - q * P), u);
  return true;
}

/* Edges per lane per batch of the chunk walker (its default; callers may
 * pick another): a warp relaxes 32*K edges with every memory step of the K
 * windows issued together, so K chains of loads and atomics are in flight
 * per lane instead of one. */
/* Pieces of a chunk where a wide level's chunks are handed out: a chunk that
 * holds hubs no longer keeps the level's barrier waiting (RMAT-20 SSSP 1.66 ms
 * with fixed chunks of 32 pieces, 1.51 handed out, 1.45 with 16, 1.46 with 8). */
#define WGM_LS_GRAB 16
#ifndef WGM_LS_K
#define WGM_LS_K 4
#endif
/* A pushed vertex with more pieces than this is written by the whole warp. */
#define WGM_LS_LANE_PIECES 4

/* Relax the edges of one chunk (one piece per lane: first edge `start`,
 * `deg` edges, source distance `dv` for SSSP) and queue the improved
 * vertices as pieces of the next level.  Per batch of 32*K edges:
 *   col/wt loads -> dist pre-check -> atomic (CAS for BFS, min for SSSP)
 *   with row[u], row[u+1] fetched beside it -> SSSP stamp exchange ->
 *   one warp scan and one counter atomic for every piece of the batch.
 * The relaxation rules are stated above wgm_ls_push; the order of
 * relaxations inside a level does not change the fixpoint. */
/* PACK (SSSP only): `dist` points at 64-bit words {low: level tag, high:
 * distance} instead of a dist[] / stamp[] pair.  One 64-bit atomicMin of
 * (alt << 32 | L) then both relaxes and deduplicates: it lowered the
 * distance iff the old high half exceeds alt, and a lowering whose old tag
 * is already L found the vertex queued for L+1 by another lane this level
 * (its tag was set by that earlier lowering).  That is the stamp exchange's
 * rule without its dependent round trip; distances read the high halves. */
/* Pieces of a vertex with d edges: ceil(d / P), by a shift when P is a
 * power of two (lg = log2 P; -1 otherwise).  P is uniform across the warp,
 * so the branch is too. */
__device__ __forceinline__ int wgm_pieces(int d, int P, int lg) {
  return lg >= 0 ? (d + P - 1) >> lg : (d + P - 1) / P;
}
__device__ __forceinline__ int wgm_piece_log2(int P) { return (P & (P - 1)) ? -1 : __ffs(P) - 1; }

/* The tail of a relaxation batch, shared by the walkers: lane k-slot holds
 * a destination u[k] whose relaxation succeeded (f[k]), its row start rs[k]
 * and row end d[k] (read beside the atomic), and (SSSP) its new distance
 * alt[k].  Unpacked SSSP exchanges the level stamp (one queueing per level);
 * a vertex without edges is not queued; near-far parks a vertex at or above
 * the threshold in the far list; the rest are queued as pieces with one
 * warp scan and one counter reservation for the whole batch. */
template <int K, bool SSSP, bool PACK>
__device__ __forceinline__ bool wgm_ls_push_batch(const int *row, int *stamp, int P, int lg,
                                                  int L, int (&u)[K], int (&rs)[K], int (&d)[K],
                                                  const unsigned (&alt)[K], bool (&f)[K],
                                                  const wgm_ls_out &o) {
  const int lane = wgm_lane();
  bool ok = true;
  int np[K];
  int mine = 0, fmine = 0;
  bool fr[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    if (SSSP && !PACK && f[k]) f[k] = atomicExch(&stamp[u[k]], L) != L;
    d[k] = f[k] ? max(d[k] - rs[k], 0) : 0; /* a vertex without edges is not queued */
    /* near-far: a distance at or above the threshold waits in the far list */
    fr[k] = PACK && d[k] > 0 && alt[k] >= o.T;
    if (fr[k]) d[k] = 0;
    fmine += fr[k] ? 1 : 0;
    np[k] = wgm_pieces(d[k], P, lg);
    mine += np[k];
  }
  const int pincl = wgm_warp_incl_scan(mine);
  const int ptotal = __shfl_sync(WGM_FULL, pincl, 31);
  int fincl = 0, ftotal = 0;
  if (PACK && __any_sync(WGM_FULL, fmine != 0)) {
    fincl = wgm_warp_incl_scan(fmine);
    ftotal = __shfl_sync(WGM_FULL, fincl, 31);
  }
  if (ptotal == 0 && ftotal == 0) return true;
  /* the piece and far reservations go out together */
  int pbase = 0, fbase = 0;
  if (lane == 31) {
    if (ptotal) pbase = wgm_out_reserve(o, ptotal);
    if (PACK && ftotal) fbase = atomicAdd(o.far_cnt, ftotal);
  }
  pbase = __shfl_sync(WGM_FULL, pbase, 31);
  if (PACK && ftotal) {
    fbase = __shfl_sync(WGM_FULL, fbase, 31);
    int fs = fbase + fincl - fmine;
    unsigned m = 0xffffffffu;
    bool spill[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      spill[k] = false;
      if (fr[k]) {
        if (fs < o.far_cap) {
          o.far_list[fs] = u[k];
          m = min(m, alt[k]);
        } else {
          spill[k] = true; /* far list full: relax it now instead */
        }
        fs++;
      }
    }
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) m = min(m, __shfl_xor_sync(WGM_FULL, m, x));
    if (lane == 0 && m != 0xffffffffu) atomicMin(o.far_min, m);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (__any_sync(WGM_FULL, spill[k]))
        ok &= wgm_out_push_vertices(row, P, spill[k], u[k], o);
  }
  if (ptotal == 0) return ok;
  if (pbase + ptotal > o.cap) return false;
  int slot = pbase + pincl - mine;
  int sl[K];
  bool big = false;
#pragma unroll
  for (int k = 0; k < K; k++) {
    sl[k] = slot;
    if (np[k] <= WGM_LS_LANE_PIECES)
      for (int q = 0; q < np[k]; q++)
        wgm_out_put(o, slot + q, rs[k] + q * P, min(P, d[k] - q * P), u[k]);
    else
      big = true;
    slot += np[k];
  }
  /* high-degree vertices: the whole warp writes their pieces */
  if (__any_sync(WGM_FULL, big)) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      unsigned bb = __ballot_sync(WGM_FULL, np[k] > WGM_LS_LANE_PIECES);
      while (bb) {
        const int j = __ffs(bb) - 1;
        bb &= bb - 1;
        const int bs = __shfl_sync(WGM_FULL, rs[k], j), bd = __shfl_sync(WGM_FULL, d[k], j);
        const int bu = __shfl_sync(WGM_FULL, u[k], j), bsl = __shfl_sync(WGM_FULL, sl[k], j);
        const int bn = wgm_pieces(bd, P, lg);
        for (int q = lane; q < bn; q += 32)
          wgm_out_put(o, bsl + q, bs + q * P, min(P, bd - q * P), bu);
      }
    }
  }
  return ok;
}

/* Relax the edges of one chunk (one piece per lane: first edge `start`,
 * `deg` edges, source distance `dv` for SSSP) and queue the improved
 * vertices as pieces of the next level.  Per batch of 32*K edges:
 *   col/wt loads -> dist pre-check -> atomic (CAS for BFS, min for SSSP)
 *   with row[u], row[u+1] fetched beside it -> SSSP stamp exchange ->
 *   one warp scan and one counter atomic for every piece of the batch.
 * The relaxation rules are stated above wgm_ls_push; the order of
 * relaxations inside a level does not change the fixpoint. */
/* PACK (SSSP only): `dist` points at 64-bit words {low: level tag, high:
 * distance} instead of a dist[] / stamp[] pair.  One 64-bit atomicMin of
 * (alt << 32 | L) then both relaxes and deduplicates: it lowered the
 * distance iff the old high half exceeds alt, and a lowering whose old tag
 * is already L found the vertex queued for L+1 by another lane this level
 * (its tag was set by that earlier lowering).  That is the stamp exchange's
 * rule without its dependent round trip; distances read the high halves. */
template <bool SSSP, bool PRE = true, bool PACK = false, int K = WGM_LS_K>
__device__ __forceinline__ bool wgm_ls_chunk(const int *row, const int *col, const unsigned *wt,
                                             unsigned *dist, int *stamp, int V, int P, int L,
                                             int start, int deg, int src,
                                             const wgm_ls_out &o) {
  static_assert(SSSP || !PACK, "the packed word carries SSSP distances");
  constexpr int DS = PACK ? 2 : 1, DH = PACK ? 1 : 0; /* distance word of v: DS*v+DH */
  const int lane = wgm_lane();
  const int lg = wgm_piece_log2(P);
  const int incl = wgm_warp_incl_scan(deg);
  const int total = __shfl_sync(WGM_FULL, incl, 31);
  const int off = incl - deg;
  const int base = start - off;
  bool ok = true;
  for (int w = 0; w < total; w += 32 * K) {
    int e[K], u[K], rs[K], d[K], sv[K];
    unsigned alt[K];
    bool f[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int s = w + 32 * k + lane;
      f[k] = s < total;
      const int own = wgm_owner_of(off, min(s, total - 1));
      e[k] = __shfl_sync(WGM_FULL, base, own) + s;
      sv[k] = SSSP ? __shfl_sync(WGM_FULL, src, own) : 0;
    }
    /* the piece vertex's distance is read beside the edge's col and weight
     * (the lanes of one piece read the same word), not before them */
#pragma unroll
    for (int k = 0; k < K; k++) {
      u[k] = f[k] ? __ldg(&col[e[k]]) : -1;
      alt[k] = 0;
      if (SSSP) {
        unsigned wk = f[k] ? __ldg(&wt[e[k]]) : WGM_LONESTAR_INF;
        unsigned dvk = f[k] ? __ldcg(&dist[DS * sv[k] + DH]) : 0u;
        f[k] = f[k] && wk < WGM_LONESTAR_INF /* sssp.cl:120 */ && wk >= o.wlo && wk < o.whi;
        alt[k] = dvk + wk;
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      f[k] = f[k] && (unsigned)u[k] < (unsigned)V; /* bfs.cl:116 */
      if (PRE && f[k]) {
        unsigned cur = __ldcg(&dist[DS * u[k] + DH]);
        f[k] = SSSP ? (alt[k] < cur) : (cur == WGM_LONESTAR_INF);
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      rs[k] = 0;
      d[k] = 0;
      if (f[k]) {
        if (PACK) {
          const unsigned long long old =
              atomicMin(reinterpret_cast<unsigned long long *>(dist) + u[k],
                        ((unsigned long long)alt[k] << 32) | (unsigned)L);
          f[k] = (unsigned)(old >> 32) > alt[k] && (unsigned)old != (unsigned)L;
        } else if (SSSP)
          f[k] = alt[k] < atomicMin(&dist[u[k]], alt[k]);
        else
          f[k] = atomicCAS(&dist[u[k]], WGM_LONESTAR_INF, (unsigned)L) == WGM_LONESTAR_INF;
        rs[k] = __ldg(&row[u[k]]);
        d[k] = __ldg(&row[u[k] + 1]);
      }
    }
    ok &= wgm_ls_push_batch<K, SSSP, PACK>(row, stamp, P, lg, L, u, rs, d, alt, f, o);
  }
  return ok;
}

/* Relax the lanes' rows (rs, d, at most 32 edges in all; source distance
 * `from`), an edge per lane; the lanes come back with the vertices that they
 * improved and claimed (u; row rs, d; d = 0: none). */
__device__ __forceinline__ unsigned wgm_ls_relax32(const wgm_lonestar_args &a, int L, int &u,
                                                   int &rs, int &d, unsigned from) {
  const int lane = wgm_lane();
  unsigned long long *word = reinterpret_cast<unsigned long long *>(a.stamp);
  const int incl = wgm_warp_incl_scan(d), total = __shfl_sync(WGM_FULL, incl, 31);
  const int off = incl - d, own = wgm_owner_of(off, min(lane, total - 1));
  const int e = __shfl_sync(WGM_FULL, rs - off, own) + lane;
  from = __shfl_sync(WGM_FULL, from, own);
  bool f = lane < total;
  u = f ? __ldg(&a.col[e]) : -1;
  const unsigned wk = f ? __ldg(&a.wt[e]) : WGM_LONESTAR_INF;
  f = f && wk < WGM_LONESTAR_INF /* sssp.cl:120 */ && (unsigned)u < (unsigned)a.V /* bfs.cl:116 */;
  rs = d = 0;
  if (f) {
    rs = __ldg(&a.row[u]);
    d = __ldg(&a.row[u + 1]);
    const unsigned alt = from + wk;
    const unsigned long long old =
        atomicMin(&word[u], ((unsigned long long)alt << 32) | (unsigned)L);
    f = (unsigned)(old >> 32) > alt && (unsigned)old != (unsigned)L;
    d = f ? max(d - rs, 0) : 0; /* a vertex without edges is not queued */
  }
  return __ballot_sync(WGM_FULL, d > 0);
}

/* SSSP, a narrow level of low-degree vertices: the lanes' pieces (start, deg,
 * src; at most 32 edges in all), then the vertices they improve at once
 * instead of in the next level, as long as their edges fit the warp, up to
 * WGM_LS_HOPS times.  A hop is two atomics' round trips, a level also the
 * list's and the barrier's.  A vertex is given up before it is relaxed: one
 * 64-bit AND clears its level tag and returns its distance, so an improvement
 * that comes later finds another tag and queues the vertex, and one that came
 * before is in the distance that is relaxed - every improvement is still
 * followed by a relaxation that reads it.  509x517 grid: 759 levels, 3.95 ms
 * without hops; 581 and 3.45 with one, 514 and 3.39 with two, 481 and 3.16
 * with three, 455 and 3.33 with five (more hops relax distances that are not
 * final yet).
 * For graphs without hubs: there is no look at a word before its atomic, and
 * a lane writes its vertex's pieces alone.  A hub's word takes an atomic of
 * every leaf, and its pieces keep one lane long; star of 300,000 from a leaf
 * 0.172 ms this way and 0.057 by wgm_ls_piece, of 30,000 0.049 and 0.022, and
 * RMAT graphs of low degree are faster without it too (2^12 vertices of
 * factor 2: 0.067 and 0.052).  Doing both here for all graphs (a look where
 * every vertex has one edge, a warp's writes) cost grids 8 and 13 %. */
#define WGM_LS_HOPS 3
#define WGM_LS_NARROW_MOST 128 /* edges of any vertex */
__device__ __forceinline__ bool wgm_ls_narrow(const wgm_lonestar_args &a, int L, int start, int deg,
                                              int src, const wgm_ls_out &o) {
  const int lane = wgm_lane(), P = a.piece;
  unsigned long long *word = reinterpret_cast<unsigned long long *>(a.stamp);
  int u = src, rs = start, d = deg;
  unsigned from = 0;
  if (d > 0) from = __ldcg(reinterpret_cast<const unsigned *>(a.stamp) + 2 * (size_t)src + 1);
  unsigned m = wgm_ls_relax32(a, L, u, rs, d, from);
  for (int hop = 0; hop < WGM_LS_HOPS && m; hop++) {
    if (__reduce_add_sync(WGM_FULL, d) > 32) break;
    if (d > 0) from = (unsigned)(atomicAnd(&word[u], 0xffffffff00000000ull) >> 32);
    m = wgm_ls_relax32(a, L, u, rs, d, from);
  }
  if (m == 0) return true;
  const int np = d > 0 ? (d + P - 1) / P : 0, incl = wgm_warp_incl_scan(np);
  const int n = __shfl_sync(WGM_FULL, incl, 31);
  int base = 0;
  if (lane == 0) base = wgm_out_reserve(o, n);
  base = __shfl_sync(WGM_FULL, base, 0);
  if (base + n > o.cap) return false;
  for (int q = 0; q < np; q++)
    wgm_out_put(o, base + incl - np + q, rs + q * P, min(P, d - q * P), u);
  return true;
}

/* One piece on one warp, an edge per lane: the walker of a level with no more
 * pieces than warps (a high-diameter graph's).  Such a level is a chain of
 * dependent round trips, so everything that is not one is left out: no owner
 * search, no scans, and the pushes are counted by ballots unless a vertex
 * has several pieces.  A piece of more than 8 edges keeps the pre-check: on
 * a dense graph most of its atomics would fail, thousands of them on a hub's
 * word.  (SSSP of low average degree goes by wgm_ls_narrow.)  Pieces of more
 * than two windows (they are as long as the average row) go by wgm_ls_chunk,
 * which has four in flight: clique of 1000, BFS 0.069 ms here and 0.049
 * there, SSSP 0.222 and 0.180; average degree 40, SSSP 0.226 and 0.238. */
#define WGM_LS_PIECE_MOST 64
template <bool SSSP>
__device__ __forceinline__ bool wgm_ls_piece(const wgm_lonestar_args &a, int L, int start, int deg,
                                             int src, const wgm_ls_out &o) {
  const int lane = wgm_lane(), V = a.V, P = a.piece;
  unsigned long long *word = reinterpret_cast<unsigned long long *>(a.stamp);
  bool ok = true;
  for (int w = 0; w < deg; w += 32) {
    const bool in = lane < deg - w;
    const int e = start + w + lane;
    int u = in ? __ldg(&a.col[e]) : -1, rs = 0, d = 0;
    unsigned alt = 0;
    bool f = in;
    if (SSSP) {
      const unsigned wk = in ? __ldg(&a.wt[e]) : WGM_LONESTAR_INF;
      alt = __ldcg(reinterpret_cast<const unsigned *>(a.stamp) + 2 * (size_t)src + 1) + wk;
      f = wk < WGM_LONESTAR_INF; /* sssp.cl:120 */
    }
    f = f && (unsigned)u < (unsigned)V; /* bfs.cl:116 */
    if (deg > 8 && f)
      f = SSSP ? alt < __ldcg(reinterpret_cast<const unsigned *>(a.stamp) + 2 * (size_t)u + 1)
               : __ldcg(&a.dist[u]) == WGM_LONESTAR_INF;
    if (f) {
      rs = __ldg(&a.row[u]);
      d = __ldg(&a.row[u + 1]);
      if (SSSP) {
        const unsigned long long old =
            atomicMin(&word[u], ((unsigned long long)alt << 32) | (unsigned)L);
        f = (unsigned)(old >> 32) > alt && (unsigned)old != (unsigned)L;
      } else {
        f = atomicCAS(&a.dist[u], WGM_LONESTAR_INF, (unsigned)L) == WGM_LONESTAR_INF;
      }
    }
    d = f ? max(d - rs, 0) : 0; /* a vertex without edges is not queued */
    const unsigned m = __ballot_sync(WGM_FULL, d > 0);
    if (m == 0) continue;
    int at = __popc(m & wgm_lanemask_lt()), np = d > 0 ? 1 : 0, n = __popc(m);
    if (__any_sync(WGM_FULL, d > P)) {
      np = (d + P - 1) / P;
      at = wgm_warp_incl_scan(np);
      n = __shfl_sync(WGM_FULL, at, 31);
      at -= np;
    }
    int base = 0;
    if (lane == 0) base = wgm_out_reserve(o, n);
    base = __shfl_sync(WGM_FULL, base, 0);
    if (base + n > o.cap) {
      ok = false;
      continue;
    }
    if (np <= WGM_LS_LANE_PIECES)
      for (int q = 0; q < np; q++)
        wgm_out_put(o, base + at + q, rs + q * P, min(P, d - q * P), u);
    /* high-degree vertices: the whole warp writes their pieces */
    for (unsigned big = __ballot_sync(WGM_FULL, np > WGM_LS_LANE_PIECES); big; big &= big - 1) {
      const int j = __ffs(big) - 1;
      const int bs = __shfl_sync(WGM_FULL, rs, j), bd = __shfl_sync(WGM_FULL, d, j);
      const int bu = __shfl_sync(WGM_FULL, u, j), bsl = base + __shfl_sync(WGM_FULL, at, j);
      const int bn = __shfl_sync(WGM_FULL, np, j);
      for (int q = lane; q < bn; q += 32)
        wgm_out_put(o, bsl + q, bs + q * P, min(P, bd - q * P), bu);
    }
  }
  return ok;
}

/* One level: every warp takes 32 consecutive pieces of the input list (one
 * per lane) and walks their edges with wgm_ls_chunk; a piece holds at most
 * `piece` edges, so no warp ever holds more than 32*piece edges of a level. */
template <bool SSSP>
__device__ __forceinline__ bool wgm_ls_level(const wgm_launch &Lc, wgm_cta *c,
                                             const wgm_lonestar_args &a, int L, int n,
                                             const int3 &first) {
  const int lane = wgm_lane(), warp = threadIdx.x >> 5;
  const int nwarps_cta = blockDim.x >> 5;
  const int gw = c->id * nwarps_cta + warp, NW = c->ngroups * nwarps_cta;
  const size_t in_off = (size_t)(L & 1) * a.cap, out_off = (size_t)((L + 1) & 1) * a.cap;
  const int *i_start = a.wl_start + in_off, *i_cnt = a.wl_cnt + in_off;
  const int *i_u = a.wl_u ? a.wl_u + in_off : nullptr;
  wgm_ls_out o;
  o.counter = &a.cnt[((L + 1) % 3) * WGM_LINE];
  o.o_start = a.wl_start + out_off;
  o.o_cnt = a.wl_cnt + out_off;
  o.o_u = a.wl_u ? a.wl_u + out_off : nullptr;
  o.cap = a.cap;
  bool ok = true;
  const bool narrow = SSSP && a.packed && a.low_degree && n <= 8 * NW;
  if (n <= NW && (!SSSP || a.packed) && !narrow && a.piece <= WGM_LS_PIECE_MOST)
    return gw >= n || wgm_ls_piece<SSSP>(a, L, first.x, first.y, first.z, o);
  /* pieces per warp: 32, or fewer when the list is short, so a small
   * frontier spreads over every warp instead of queueing on a few */
  const int most = a.grab ? WGM_LS_GRAB : 32;
  const int per = max(1, min(most, (n + NW - 1) / NW));
  const bool hand_out = a.grab && n > 2 * NW * per;
  int *grab = a.grab + (L % 3) * WGM_LINE;
  int next = 0;
  for (int b = gw * per; b < n; b = next) {
    if (hand_out) { /* the next chunk's number comes while this one is walked */
      if (lane == 0) next = atomicAdd(grab, per);
    } else {
      next = b + NW * per;
    }
    int i = b + lane, deg = 0, start = 0, src = 0;
    if (lane < per && i < n) {
      start = __ldcg(&i_start[i]);
      deg = __ldcg(&i_cnt[i]);
      if (SSSP) src = __ldcg(&i_u[i]);
    }
    if (narrow && __reduce_add_sync(WGM_FULL, deg) <= 32)
      ok &= wgm_ls_narrow(a, L, start, deg, src, o);
    else if (SSSP && a.packed)
      ok &= wgm_ls_chunk<SSSP, true, SSSP>(a.row, a.col, a.wt,
                                           reinterpret_cast<unsigned *>(a.stamp), a.stamp, a.V,
                                           a.piece, L, start, deg, src, o);
    else
      ok &= wgm_ls_chunk<SSSP>(a.row, a.col, a.wt, a.dist, a.stamp, a.V, a.piece, L, start, deg,
                               src, o);
    if (hand_out) next = __shfl_sync(WGM_FULL, next, 0) + NW * per;
  }
  return ok;
}

/* Lonestar BFS on one CTA (standalone runs of small graphs, bfs_mode 1).
 * A level of a high-diameter graph carries a few hundred vertices, and the
 * grid form pays a chain of dependent L2 round trips per level (counter,
 * worklist pieces, columns, the claiming CAS, the pushed rows, the barrier):
 * ~4 us on the 256x256 grid whether 1 or 152 CTAs run it.  Here the whole
 * traversal lives in one CTA: visited bits in shared memory, claimed with a
 * shared-memory atomicOr; the frontier in shared memory (vertices past its
 * capacity spill to global memory); level counters triple-buffered in shared
 * memory, so a level is one __syncthreads and the round trips of its
 * adjacency.  Same levels as the Lonestar kernel: the source
 * is level 0, a vertex first reached while level L runs gets L, out-of-range
 * columns are skipped (bfs.cl:116), the loader quirk's negative last degree
 * walks nothing, and the level count is the first level whose frontier
 * walks no edge (the grid form never queues a vertex without edges).
 *
 * The adjacency: graphs of out-degree at most W = 4 or 8 keep a second copy
 * of their columns as W per vertex (wgm_k_bfs_ell; WGM_BFS_PAD fills up), so
 * one round trip brings a vertex's whole row.  W = 0 walks the CSR, four
 * columns a round trip.
 * The frontier is kept short of shared memory's size, for the L1 is what
 * serves the neighbouring rows.  256x256 grid: 1.86 us a level with one
 * column per round trip (four in a row) -> 0.94 us; 1024 threads 0.344,
 * 512 0.341, 256 0.37 ms.  Measured and left out: prefetching a found
 * vertex's row (3 % slower), a warp's reservation by ballots instead of one
 * per lane (11 % slower), skewed bit words (no change). */
#define WGM_BFS_PAD INT_MIN
extern __shared__ int wgm_bfs_dyn[]; /* [ceil(V/32)] visited bits, then 2 x F frontier */

template <int W>
__device__ __forceinline__ void wgm_bfs_cta(const wgm_lonestar_args &a, const int4 *ell, int *spill,
                                            int spill_cap, int F, int *s_cnt) {
  const int V = a.V, nw = (V + 31) >> 5, T = blockDim.x;
  unsigned *bits = reinterpret_cast<unsigned *>(wgm_bfs_dyn);
  for (int i = threadIdx.x; i < nw; i += T) bits[i] = 0u;
  for (int i = threadIdx.x; i < V; i += T) a.dist[i] = (i == a.source) ? 0u : WGM_LONESTAR_INF;
  if (threadIdx.x < 8) s_cnt[threadIdx.x] = threadIdx.x == 1; /* 0-2: level sizes by L mod 3,
                                                                 3: overflow, 4-6: the level
                                                                 walked an edge, by L mod 3 */
  __syncthreads();
  /* level 1 reads buffer 1 */
  int in = nw + F, out = nw, in_sp = spill_cap, out_sp = 0;
  if (threadIdx.x == 0) {
    bits[a.source >> 5] = 1u << (a.source & 31);
    wgm_bfs_dyn[in] = a.source;
  }
  __syncthreads();
  int L = 1;
  wgm_proto_levels w3{1, 2, 0}; /* L, L + 1, L + 2 mod 3 */
  for (;;) {
    const int n = s_cnt[w3.now];
    if (n == 0 || L > V + 1) break;
    if (threadIdx.x == 0) {
      s_cnt[w3.size_to_clear()] = 0;
      s_cnt[4 + w3.flag_to_clear()] = 0; /* not the one that late warps still read below */
    }
    /* Claim N neighbours for level L and queue the new ones: N bit words
     * read together, N claims together, one reservation. */
    auto reach = [&](auto &u) {
      constexpr int N = sizeof(u) / sizeof(u[0]);
      unsigned w[N];
      int found = 0;
#pragma unroll
      for (int q = 0; q < N; q++)
        w[q] = (unsigned)u[q] < (unsigned)V ? bits[u[q] >> 5] : 0xffffffffu;
#pragma unroll
      for (int q = 0; q < N; q++) {
        const unsigned bit = 1u << (u[q] & 31);
        if (!(w[q] & bit)) w[q] = atomicOr(&bits[u[q] >> 5], bit);
      }
#pragma unroll
      for (int q = 0; q < N; q++) {
        w[q] = ~w[q] >> (u[q] & 31) & 1u; /* now: claimed here */
        found += w[q];
      }
      if (found == 0) return;
      int k = atomicAdd(&s_cnt[w3.next], found);
#pragma unroll
      for (int q = 0; q < N; q++) {
        if (!w[q]) continue;
        a.dist[u[q]] = (unsigned)L;
        if (k < F)
          wgm_bfs_dyn[out + k] = u[q];
        else if (k - F < spill_cap)
          spill[out_sp + k - F] = u[q];
        else
          s_cnt[3] = 1;
        k++;
      }
    };
    for (int i = threadIdx.x; i < n; i += T) {
      const int v = i < F ? wgm_bfs_dyn[in + i] : __ldcg(&spill[in_sp + i - F]);
      if (W) {
        int u[W ? W : 1];
#pragma unroll
        for (int q = 0; q < W / 4; q++) {
          const int4 r = __ldg(&ell[v * (W / 4) + q]);
          u[4 * q] = r.x;
          u[4 * q + 1] = r.y;
          u[4 * q + 2] = r.z;
          u[4 * q + 3] = r.w;
        }
        if (u[0] != WGM_BFS_PAD) s_cnt[4 + w3.now] = 1;
        reach(u);
      } else {
        const int s = __ldg(&a.row[v]);
        const int d = max(__ldg(&a.row[v + 1]) - s, 0);
        if (d > 0) s_cnt[4 + w3.now] = 1;
        for (int j = 0; j < d; j += 4) {
          int u[4];
#pragma unroll
          for (int q = 0; q < 4; q++) u[q] = j + q < d ? __ldg(&a.col[s + j + q]) : -1;
          reach(u);
        }
      }
    }
    __syncthreads();
    /* the grid form queues no vertex without edges (it has no pieces): a
     * level that walked no edge is where its frontier was empty */
    if (!s_cnt[4 + w3.now]) break;
    L++;
    w3.step();
    int t = in;
    in = out;
    out = t;
    t = in_sp;
    in_sp = out_sp;
    out_sp = t;
  }
  if (threadIdx.x == 0 && a.levels_out) *a.levels_out = L;
}

/* Persistent BFS/SSSP phases: (0) device-side init; (1,L) level L.  One
 * barrier per level (the reference uses two, bfs.cl:282,295): the piece
 * counters are triple-buffered by level, so the counter a level fills was
 * cleared two levels earlier and the swap/reset step needs no barrier. */
template <bool SSSP>
static __device__ int wgm_phase_lonestar(const wgm_launch &Lc, wgm_cta *c,
                                         const wgm_lonestar_args &a, wgm_warp_smem *sm,
                                         int target, int Lv, int *next_target, int *next_round) {
  const int V = a.V;
  if (target == 0) {
    const int tid = c->id * blockDim.x + threadIdx.x, nth = c->ngroups * blockDim.x;
    /* Host init of the plugin (bfs.h:250-262) done on the device. */
    for (int i = tid; i < V; i += nth) {
      if (SSSP && a.packed) {
        reinterpret_cast<unsigned long long *>(a.stamp)[i] =
            (i == a.source) ? 0ull : (unsigned long long)WGM_LONESTAR_INF << 32;
      } else {
        a.dist[i] = (i == a.source) ? 0u : WGM_LONESTAR_INF;
        if (SSSP) a.stamp[i] = 0;
      }
    }
    if (c->id == 0 && threadIdx.x < 32) {
      /* Level 1 processes the source (bfs.cl:235-241 seeds it at iteration 0). */
      if (threadIdx.x == 0)
        for (int k = 0; k < 3; k++) {
          a.cnt[k * WGM_LINE] = 0;
          if (a.grab) a.grab[k * WGM_LINE] = 0;
        }
      __syncwarp();
      wgm_ls_push(a, threadIdx.x == 0, a.source, &a.cnt[1 * WGM_LINE], a.wl_start + a.cap,
                  a.wl_cnt + a.cap, a.wl_u ? a.wl_u + a.cap : nullptr, sm->acc[0]);
    }
    *next_target = 1;
    *next_round = 1;
    return 1;
  }
  /* this warp's piece of a short level, read beside the level's size (any
   * words, when the list is shorter) */
  int3 first = make_int3(0, 0, 0);
  const int gw = c->id * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw < a.cap) {
    const size_t i = (size_t)(Lv & 1) * a.cap + gw;
    first.x = __ldcg(&a.wl_start[i]);
    first.y = __ldcg(&a.wl_cnt[i]);
    if (SSSP) first.z = __ldcg(&a.wl_u[i]);
  }
  const int n = __ldcg(&a.cnt[(Lv % 3) * WGM_LINE]);
  if (n == 0) {
    if (c->id == 0 && threadIdx.x == 0 && a.levels_out) *a.levels_out = Lv;
    if (SSSP && a.packed) { /* the distances out of the packed words */
      const int tid = c->id * blockDim.x + threadIdx.x, nth = c->ngroups * blockDim.x;
      const unsigned *w = reinterpret_cast<const unsigned *>(a.stamp);
      for (int i = tid; i < V; i += nth) a.dist[i] = __ldcg(&w[2 * i + 1]);
    }
    return 0;
  }
  if (n > a.cap) {
    wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, Lv);
    return 0;
  }
  if (Lv > V + 2) { /* Bellman-Ford bound; only a corrupt input gets here */
    wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, Lv);
    return 0;
  }
  if (c->id == 0 && threadIdx.x == 0) {
    a.cnt[((Lv + 2) % 3) * WGM_LINE] = 0;
    if (a.grab) a.grab[((Lv + 2) % 3) * WGM_LINE] = 0;
  }
  if (!wgm_ls_level<SSSP>(Lc, c, a, Lv, n, first)) wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, Lv);
  *next_target = 1;
  *next_round = Lv + 1;
  return 1;
}

/* Lonestar BFS in two directions (standalone runs of large graphs).  A level
 * whose worklist holds a good part of the edges walks every one of them for
 * the few vertices still unreached (RMAT-20: 25 M edges for 0.2 M vertices);
 * such a level is run from the other side: each unreached vertex looks
 * through its in-edges until it meets a reached one (0.2-2 M looks).  An
 * unreached vertex's reached in-neighbours are all of the level before, or
 * it would have been reached sooner, so one bit per vertex answers a look
 * (128 KB on RMAT-20: served by the L1).  Levels and their count are the
 * worklist's: the vertex takes the running level, and a level whose new
 * vertices have no out-edge is the last.
 *
 * Phases: (1,L) the worklist's level L, or, when its pieces hold more than
 * WGM_BFS_UP_EDGES edges and a twentieth of the graph, the bits of the
 * reached vertices instead and (2,L); (2,L) and (3,L) level L from the
 * unreached side, (3,L) after the last one's verdict: nothing new to walk -
 * done; fewer than V/64 new - the worklist again, from the distances, at
 * (1,L).  RMAT-20: 0.39 -> 0.13 ms, most of it the first such level (0.6 M
 * vertices with two looks each: the round trips row, in-edge, bit). */
#define WGM_BFS_UP_EDGES (1 << 20)
#define WGM_BFS_UP_SCAN 4096 /* in-edges of a vertex that one warp looks at */
struct wgm_bfs_up_args {
  const int *trow, *tcol; /* in-edges */
  unsigned *bits;         /* [3][ceil(V/32)] reached, by level parity; without in-edges
                             (never looked at, but no answer to a look either) */
  int *cnt;               /* [3 lines] by level mod 3: new vertices, any of them with
                             out-edges */
  const int *wide;        /* vertices of more than WGM_BFS_UP_SCAN in-edges */
  int nwide;
  long long E;
};

/* Level L from the unreached side. */
__device__ __forceinline__ void wgm_bfs_up_level(const wgm_cta *c, const wgm_lonestar_args &a,
                                                 const wgm_bfs_up_args &b, int L,
                                                 wgm_warp_smem *sm) {
  __shared__ int s_new, s_walk;
  const wgm_split s(c);
  const int V = a.V, lane = s.lane, nword = (V + 31) >> 5;
  const unsigned *cur = b.bits + (size_t)(L & 1) * nword;
  unsigned *nxt = b.bits + (size_t)((L + 1) & 1) * nword;
  const unsigned *none = b.bits + 2 * (size_t)nword;
  int *cnt = &b.cnt[(L % 3) * WGM_LINE];
  if (threadIdx.x == 0) s_new = s_walk = 0;
  __syncthreads();
  auto reached = [&](bool valid, int j, int) {
    return valid && (__ldca(&cur[j >> 5]) >> (j & 31) & 1u);
  };
  auto take = [&](int v) { /* v is new: its distance, and whether it can go on */
    a.dist[v] = (unsigned)L;
    if (!s_walk && wgm_ls_degree(a.row, v) > 0) s_walk = 1;
  };
  int fresh = 0;
  for (int k = s.gw; k < nword; k += s.NW) {
    const unsigned m = __ldcg(&cur[k]), done = m | __ldcg(&none[k]);
    if (done == WGM_FULL) {
      if (lane == 0 && __ldcg(&nxt[k]) != m) atomicOr(&nxt[k], m);
      continue;
    }
    const int v = k * 32 + lane;
    const bool act = !((done >> lane) & 1u);
    int e = 0, end = 0;
    if (act) {
      e = __ldg(&b.trow[v]);
      end = __ldg(&b.trow[v + 1]);
    }
    bool wide; /* the whole grid looks on, below */
    const bool f = wgm_first_edge(b.tcol, act, e, end, WGM_BFS_UP_SCAN, wide, sm->tab[s.warp],
                                  reached);
    if (f) take(v);
    const unsigned nw = __ballot_sync(WGM_FULL, f);
    fresh += __popc(nw);
    if (lane == 0) atomicOr(&nxt[k], m | nw);
  }
  /* the rest of very long rows: S warps each, until one has its edge */
  if (b.nwide > 0) {
    const int S = max(1, s.NW / b.nwide), sub = s.gw % S, per = max(1, s.NW / S);
    for (int h = s.gw / S; h < b.nwide && s.gw < per * S; h += per) {
      const int v = __ldg(&b.wide[h]);
      if (__ldcg(&cur[v >> 5]) >> (v & 31) & 1u) continue;
      const int end = __ldg(&b.trow[v + 1]);
      bool f = false;
      for (long long x = (long long)__ldg(&b.trow[v]) + WGM_BFS_UP_SCAN + 128LL * sub;
           x < end && !f; x += 128LL * S) {
        /* another warp has it: it may be setting the bit now, so one answer for
         * the warp, which looks together */
        if (__any_sync(WGM_FULL, __ldcg(&nxt[v >> 5]) >> (v & 31) & 1u)) break;
        int j[4];
        bool h4 = false;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const bool in = x + 32 * q + lane < end;
          j[q] = in ? __ldg(&b.tcol[x + 32 * q + lane]) : -1;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) h4 |= reached(j[q] >= 0, j[q], lane);
        f = __any_sync(WGM_FULL, h4);
      }
      if (f && lane == 0) {
        const unsigned bit = 1u << (v & 31);
        if (!(atomicOr(&nxt[v >> 5], bit) & bit)) {
          take(v);
          fresh++;
        }
      }
      fresh = __shfl_sync(WGM_FULL, fresh, 0);
    }
  }
  if (lane == 0 && fresh) atomicAdd(&s_new, fresh);
  __syncthreads();
  if (threadIdx.x == 0 && s_new) {
    atomicAdd(&cnt[0], s_new);
    if (s_walk) cnt[1] = 1;
  }
}

static __device__ int wgm_phase_bfs(const wgm_launch &Lc, wgm_cta *c, const wgm_lonestar_args &a,
                                    const wgm_bfs_up_args &b, wgm_warp_smem *sm, wgm_step cur,
                                    wgm_step *nxt) {
  const wgm_split s(c);
  const int V = a.V, L = cur.round;
  if (cur.target == 1) {
    const long long n = __ldcg(&a.cnt[(L % 3) * WGM_LINE]);
    const long long edges = n * a.piece;
    if (n <= a.cap && edges > WGM_BFS_UP_EDGES && edges > b.E / 20) {
      const int nword = (V + 31) >> 5;
      for (int k = s.gw; k < nword; k += s.NW) {
        const int v = k * 32 + s.lane;
        bool r = false, none = true;
        if (v < V) {
          r = __ldcg(&a.dist[v]) != WGM_LONESTAR_INF;
          none = __ldg(&b.trow[v + 1]) == __ldg(&b.trow[v]);
        }
        const unsigned m = __ballot_sync(WGM_FULL, r), z = __ballot_sync(WGM_FULL, none);
        if (s.lane < 3) b.bits[(size_t)s.lane * nword + k] = s.lane < 2 ? m : z;
      }
      if (c->id == 0 && threadIdx.x < 3) {
        b.cnt[threadIdx.x * WGM_LINE] = 0;
        b.cnt[threadIdx.x * WGM_LINE + 1] = 0;
      }
      *nxt = {2, L};
      return WGM_PHASE_NEXT;
    }
  }
  if (cur.target < 2)
    return wgm_phase_lonestar<false>(Lc, c, a, sm, cur.target, cur.round, &nxt->target,
                                     &nxt->round);
  if (cur.target == 3) {
    const int2 r = __ldcg(reinterpret_cast<const int2 *>(&b.cnt[((L + 2) % 3) * WGM_LINE]));
    if (r.y == 0) {
      if (c->id == 0 && threadIdx.x == 0 && a.levels_out) *a.levels_out = L;
      return WGM_PHASE_DONE;
    }
    if (r.x < V / 64) {
      /* few new vertices: their pieces as level L's worklist */
      bool ok = true;
      wgm_ls_out o;
      o.counter = &a.cnt[(L % 3) * WGM_LINE];
      o.o_start = a.wl_start + (size_t)(L & 1) * a.cap;
      o.o_cnt = a.wl_cnt + (size_t)(L & 1) * a.cap;
      o.o_u = a.wl_u ? a.wl_u + (size_t)(L & 1) * a.cap : nullptr;
      o.cap = a.cap;
      for (int k = s.gw * 32; k < V; k += s.NW * 32) {
        const int v = k + s.lane;
        const bool f = v < V && __ldcg(&a.dist[v]) == (unsigned)(L - 1);
        ok &= wgm_out_push_vertices(a.row, a.piece, f, v, o);
      }
      if (!ok) wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, L);
      *nxt = {1, L};
      return WGM_PHASE_NEXT;
    }
  }
  if (L > V + 2) { /* only a corrupt input gets here */
    wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, L);
    return WGM_PHASE_DONE;
  }
  /* the worklist's counters, last read before (2,L): empty for its return */
  if (c->id == 0 && threadIdx.x < 3) {
    a.cnt[threadIdx.x * WGM_LINE] = 0;
    if (a.grab) a.grab[threadIdx.x * WGM_LINE] = 0;
    if (threadIdx.x < 2) b.cnt[((L + 1) % 3) * WGM_LINE + threadIdx.x] = 0;
  }
  wgm_bfs_up_level(c, a, b, L, sm);
  *nxt = {3, L + 1};
  return WGM_PHASE_NEXT;
}

/* ------------------------------------------------------------------------ */
/* Pannotia colour                                                           */
/* ------------------------------------------------------------------------ */

struct wgm_color_args {
  int V;
  const int *row; /* [V+1] */
  const int *col;
  const int *trow; /* in-edges (the transpose; the graph itself when symmetric) */
  const int *tcol;
  const float *node_value;
  int *color;    /* [V] output: 1-based colours */
  wgm_hubs hubs; /* static layout of out-degree > hub_threshold vertices */
  int hub_threshold;
  int *rounds_out;
  int *pending;  /* [V] larger out-neighbours not yet coloured */
  int *wl_start, *wl_cnt, *wl_u; /* [2][cap] frontier pieces of in-edges; wl_u holds
                                    the value bits of the piece's vertex */
  int cap, piece;
  int *cnt;      /* [3 lines] frontier sizes by round mod 3 */
  int2 *tcv;     /* [in-edges] {in-neighbour, its value bits}, filled at init */
};

/* Pannotia colour (color.cl:3-97) computed as the frontier recurrence it
 * implies.  In the reference a vertex v takes colour r in the first round r
 * in which no out-neighbour with a larger value is uncoloured at the start
 * of r (color.cl:66-83; a vertex coloured in round r still counts as
 * uncoloured during r).  Hence colour(v) = 1 + max colour of its larger
 * out-neighbours (1 if none), degree-1 vertices take colour 1 because they
 * skip their neighbours (color.cl:46), and the reference's round count is
 * the largest colour (its exit test, color.cl:85-87, first fails in the
 * round after the last vertex is coloured).  So: count each vertex's larger
 * out-neighbours once (`pending`), colour the vertices with none in round 1,
 * and in round r let every vertex coloured r decrement its smaller
 * in-neighbours; one that reaches zero takes colour r+1.  Same colours and
 * round count as the reference, each edge looked at twice in all instead of
 * once per round.
 * Phases: (0) init; (3,0) count larger out-neighbours; (4,0) round-1
 * frontier; (1,r) the vertices coloured r release their in-neighbours. */
/* tcv[e] = {in-neighbour w, a word about w} (one 8-byte load per edge).
 * pre(w, word, src, &tag) tests w without side effects and sets the word
 * its queue entry will carry; commit(w) claims it (true: queue it).  The
 * in-edge row bounds of every w that passes `pre` are loaded beside
 * `commit`'s atomic, not after it. */
template <class Pre, class Commit>
__device__ __forceinline__ bool wgm_frontier_chunk(const int *trow, const int2 *tcv, int P,
                                                   int start, int deg, unsigned sv,
                                                   const wgm_ls_out &o, Pre &&pre,
                                                   Commit &&commit) {
  constexpr int K = WGM_LS_K;
  const int lane = wgm_lane();
  const int incl = wgm_warp_incl_scan(deg);
  const int total = __shfl_sync(WGM_FULL, incl, 31);
  const int off = incl - deg;
  const int base = start - off;
  bool ok = true;
  for (int w = 0; w < total; w += 32 * K) {
    int u[K], rs[K], d[K], np[K], tg[K], wv[K];
    unsigned src[K];
    bool f[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int s = w + 32 * k + lane;
      f[k] = s < total;
      const int own = wgm_owner_of(off, min(s, total - 1));
      const int e = __shfl_sync(WGM_FULL, base, own) + s;
      src[k] = __shfl_sync(WGM_FULL, sv, own);
      const int2 p = f[k] ? __ldg(&tcv[e]) : make_int2(-1, 0);
      u[k] = p.x;
      wv[k] = p.y;
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      tg[k] = 0;
      f[k] = f[k] && pre(u[k], wv[k], src[k], &tg[k]);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      rs[k] = 0;
      d[k] = 0;
      if (f[k]) {
        rs[k] = __ldg(&trow[u[k]]);
        d[k] = __ldg(&trow[u[k] + 1]);
        f[k] = commit(u[k]);
      }
    }
    int mine = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      d[k] = f[k] ? max(d[k] - rs[k], 0) : 0;
      np[k] = (d[k] + P - 1) / P;
      mine += np[k];
    }
    const int pincl = wgm_warp_incl_scan(mine);
    const int ptotal = __shfl_sync(WGM_FULL, pincl, 31);
    if (ptotal == 0) continue;
    int pbase = 0;
    if (lane == 31) pbase = wgm_out_reserve(o, ptotal);
    pbase = __shfl_sync(WGM_FULL, pbase, 31);
    if (pbase + ptotal > o.cap) {
      ok = false;
      continue;
    }
    int slot = pbase + pincl - mine;
    int sl[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      sl[k] = slot;
      if (np[k] <= WGM_LS_LANE_PIECES) {
        for (int q = 0; q < np[k]; q++) {
          o.o_start[slot + q] = rs[k] + q * P;
          o.o_cnt[slot + q] = min(P, d[k] - q * P);
          o.o_u[slot + q] = tg[k];
        }
      }
      slot += np[k];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      unsigned big = __ballot_sync(WGM_FULL, np[k] > WGM_LS_LANE_PIECES);
      while (big) {
        const int j = __ffs(big) - 1;
        big &= big - 1;
        const int bs = __shfl_sync(WGM_FULL, rs[k], j), bd = __shfl_sync(WGM_FULL, d[k], j);
        const int bu = __shfl_sync(WGM_FULL, tg[k], j), bsl = __shfl_sync(WGM_FULL, sl[k], j);
        const int bn = (bd + P - 1) / P;
        for (int q = lane; q < bn; q += 32) {
          o.o_start[bsl + q] = bs + q * P;
          o.o_cnt[bsl + q] = min(P, bd - q * P);
          o.o_u[bsl + q] = bu;
        }
      }
    }
  }
  return ok;
}

/* Queue the in-edge pieces of the lanes' flagged vertices (one vertex per
 * lane, the whole warp writes); the entries carry `tag`. */
__device__ __forceinline__ bool wgm_frontier_push(const int *trow, int P, bool flag, int v,
                                                  int tag, const wgm_ls_out &o, int *tab) {
  int start = 0, deg = 0, np = 0;
  if (flag) {
    start = __ldg(&trow[v]);
    deg = max(__ldg(&trow[v + 1]) - start, 0);
    np = (deg + P - 1) / P;
  }
  int incl = wgm_warp_incl_scan(np);
  int total = __shfl_sync(WGM_FULL, incl, 31);
  if (total == 0) return true;
  int base = 0;
  if (wgm_lane() == 0) base = wgm_out_reserve(o, total);
  base = __shfl_sync(WGM_FULL, base, 0);
  if (base + total > o.cap) return false;
  int off = incl - np;
  wgm_for_each_edge(off, np, -off, total, 0, 32, tab, [&](bool valid, int k, int owner) {
    int s = __shfl_sync(WGM_FULL, start, owner);
    int d = __shfl_sync(WGM_FULL, deg, owner);
    int x = __shfl_sync(WGM_FULL, tag, owner);
    int oo = __shfl_sync(WGM_FULL, off, owner);
    if (valid) {
      int slot = base + oo + k;
      o.o_start[slot] = s + k * P;
      o.o_cnt[slot] = min(P, d - k * P);
      o.o_u[slot] = x;
    }
  });
  return true;
}

static __device__ int wgm_phase_color(const wgm_launch &Lc, wgm_cta *c, const wgm_color_args &a,
                                      wgm_warp_smem *sm, wgm_step cur, wgm_step *nxt) {
  const wgm_split s(c);
  const int V = a.V;
  const int lane = s.lane, warp = s.warp;
  if (cur.target == 0) {
    for (int i = s.tid; i < V; i += s.nth) {
      a.color[i] = -1; /* color.h:50 */
      a.pending[i] = 0;
    }
    /* every in-edge beside its neighbour's value: a release reads both at once */
    const int ET = __ldg(&a.trow[V]);
    for (int e = s.tid; e < ET; e += s.nth) {
      const int w = __ldg(&a.tcol[e]);
      a.tcv[e] = make_int2(w, __float_as_int(__ldg(&a.node_value[w])));
    }
    if (c->id == 0 && threadIdx.x < 3) a.cnt[threadIdx.x * WGM_LINE] = 0;
    *nxt = {3, 0};
    return WGM_PHASE_NEXT;
  }
  if (cur.target == 3) {
    /* larger out-neighbours of every vertex; a degree-1 vertex has none
     * (color.cl:46) */
    for (int b = s.gw * 32; b < V; b += s.NW * 32) {
      const int i = b + lane;
      int deg = 0, start = 0;
      float vi = 0.f;
      if (i < V) {
        start = __ldg(&a.row[i]);
        const int d = __ldg(&a.row[i + 1]) - start;
        deg = (d == 1 || d > a.hub_threshold) ? 0 : d;
        vi = __ldg(&a.node_value[i]);
      }
      sm->acc[warp][lane] = 0;
      int incl = wgm_warp_incl_scan(deg);
      int total = __shfl_sync(WGM_FULL, incl, 31);
      int off = incl - deg;
      __syncwarp();
      wgm_for_each_edge(off, deg, start - off, total, 0, 32, sm->tab[warp],
                        [&](bool valid, int e, int owner) {
                          const float vo = __shfl_sync(WGM_FULL, vi, owner);
                          if (valid && __ldg(&a.node_value[__ldg(&a.col[e])]) > vo)
                            atomicAdd(&sm->acc[warp][owner], 1);
                        });
      __syncwarp();
      if (i < V && deg > 0) a.pending[i] = sm->acc[warp][lane];
    }
    const int nwin = (a.hubs.total + 31) >> 5;
    for (int k = s.gw; k < nwin; k += s.NW) {
      wgm_hub_window(a.hubs, a.row, k, [&](bool valid, int h, int e) {
        int h0 = __shfl_sync(WGM_FULL, h, 0);
        int cntv = 0;
        if (valid) {
          const int v = __ldg(&a.hubs.ids[h]);
          cntv = __ldg(&a.node_value[__ldg(&a.col[e])]) > __ldg(&a.node_value[v]) ? 1 : 0;
        }
        const int n0 = __reduce_add_sync(WGM_FULL, h == h0 ? cntv : 0);
        const int n1 = __reduce_add_sync(WGM_FULL, h == h0 ? 0 : cntv);
        if (lane == 0) {
          if (n0 > 0) atomicAdd(&a.pending[__ldg(&a.hubs.ids[h0])], n0);
          if (n1 > 0 && h0 + 1 < a.hubs.H) atomicAdd(&a.pending[__ldg(&a.hubs.ids[h0 + 1])], n1);
        }
      });
    }
    *nxt = {4, 0};
    return WGM_PHASE_NEXT;
  }
  wgm_ls_out o;
  o.cap = a.cap;
  if (cur.target == 4) {
    /* round 1: every vertex without a larger out-neighbour */
    o.counter = &a.cnt[1 * WGM_LINE];
    o.o_start = a.wl_start + a.cap;
    o.o_cnt = a.wl_cnt + a.cap;
    o.o_u = a.wl_u + a.cap;
    bool ok = true;
    for (int b = s.gw * 32; b < V; b += s.NW * 32) {
      const int i = b + lane;
      const bool f = i < V && __ldcg(&a.pending[i]) == 0;
      int tag = 0;
      if (f) {
        a.color[i] = 1;
        tag = __float_as_int(__ldg(&a.node_value[i]));
      }
      ok &= wgm_frontier_push(a.trow, a.piece, f, i, tag, o, sm->tab[warp]);
    }
    if (!ok) wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, 1);
    *nxt = {1, 1};
    return WGM_PHASE_NEXT;
  }
  const int r = cur.round;
  const int n = __ldcg(&a.cnt[(r % 3) * WGM_LINE]);
  if (n == 0) {
    if (c->id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = r - 1;
    return WGM_PHASE_DONE;
  }
  if (n > a.cap || r > V + 2) {
    wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, r);
    return WGM_PHASE_DONE;
  }
  if (c->id == 0 && threadIdx.x == 0) a.cnt[((r + 2) % 3) * WGM_LINE] = 0;
  const size_t io = (size_t)(r & 1) * a.cap, oo = (size_t)((r + 1) & 1) * a.cap;
  o.counter = &a.cnt[((r + 1) % 3) * WGM_LINE];
  o.o_start = a.wl_start + oo;
  o.o_cnt = a.wl_cnt + oo;
  o.o_u = a.wl_u + oo;
  const int next_colour = r + 1;
  bool ok = true;
  /* pieces per warp: 32, or fewer when the frontier is short */
  const int per = max(1, min(32, (n + s.NW - 1) / s.NW));
  for (int b = s.gw * per; b < n; b += s.NW * per) {
    int i = b + lane, deg = 0, start = 0;
    unsigned sv = 0;
    if (lane < per && i < n) {
      start = __ldcg(&a.wl_start[io + i]);
      deg = __ldcg(&a.wl_cnt[io + i]);
      sv = (unsigned)__ldcg(&a.wl_u[io + i]); /* the coloured vertex's value bits */
    }
    ok &= wgm_frontier_chunk(
        a.trow, a.tcv, a.piece, start, deg, sv, o,
        [&](int w, int wbits, unsigned src, int *tag) {
          /* w has the coloured vertex as a larger out-neighbour */
          (void)w;
          *tag = wbits;
          return __int_as_float(wbits) < __uint_as_float(src);
        },
        [&](int w) {
          if (atomicSub(&a.pending[w], 1) != 1) return false;
          a.color[w] = next_colour;
          return true;
        });
  }
  if (!ok) wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, r);
  *nxt = {1, r + 1};
  return WGM_PHASE_NEXT;
}

/* ------------------------------------------------------------------------ */
/* Pannotia colour in priority blocks (standalone runs)                      */
/* ------------------------------------------------------------------------ */

/* colour(v) = 1 + the largest colour among v's larger out-neighbours (1 if
 * none; degree-1 vertices 1), the recurrence wgm_phase_color computes a
 * round - a grid barrier and six dependent round trips - per colour.  Here
 * the vertices are taken by rank (descending value), NB blocks of B: every
 * larger out-neighbour of a vertex is in its own block or an earlier one.
 *   - The grid looks at every edge of block b once (stage A): an edge to a
 *     block before b - 1, whose colours are final, raises the vertex's
 *     colour so far; an edge inside block b or to block b - 1 goes to a
 *     short list.
 *   - One CTA finishes the block (stage B) with the colours of blocks b - 1
 *     and b in shared memory: listed edges from block b - 1 raise their
 *     target, the inner ones (a few hundred) are relaxed all at once until a
 *     sweep changes nothing - as many sweeps as the longest chain inside
 *     the block.
 * Stage B of block b - 1 runs beside stage A of block b, so a block costs
 * one grid barrier, and a link of a colour chain a sweep of shared memory
 * instead of a round.  Colours, columns and the list all go by rank, so
 * stage B touches memory in whole lines only: one CTA gathers about 0.3
 * words a cycle, and with vertex ids it spent 10 us a block on 5700 gathers.
 * RMAT-20 (about 1650 colours): 128 blocks, 8.6 ms in rounds -> 1.6 ms.  A
 * block takes 12.5 us, and stage B sets it: 2 us to fetch the block's
 * colours and lists, 1.5 us for the late edges, 4 us for the inner ones
 * (14 links a block), 1 us to write back, and 3.5 us for a barrier that
 * waits for those writes; stage A takes 2-5 us beside it. */
#define WGM_CB_LATE 6144  /* edges listed from a block to the one before it */
#define WGM_CB_INNER 3072 /* edges listed inside a block */
#define WGM_CB_LISTS (WGM_CB_LATE + WGM_CB_INNER)
#define WGM_CB_MAX_B 8192 /* vertices of a block (a list entry packs 13 + 13 bits) */
struct wgm_color_blocks_args {
  const int4 *ord;     /* [V] by rank: {vertex, first edge, out-degree, hub index or -1} */
  const int *crank;    /* [E] col[] as ranks */
  int *colour;         /* [V] by rank: colour so far, then the colour */
  const int *blk_hub;  /* [NB+1] first hub of each block (hubs in rank order) */
  const int *hub_rank; /* [H] */
  unsigned *list;      /* [2][WGM_CB_LISTS] by block parity: late edges, then inner
                          ones, each target << 16 | source, ranks in their blocks */
  int *cnt;            /* [3 lines] by block mod 3: late edges, inner edges; word 2 of
                          line 0: largest colour */
  int *hub_max;        /* [H] largest final colour seen by a hub */
  int NB, B;
};

/* Group 0: the colours of two blocks, 2 x B, then a 0; read and written in
 * words of 16 bytes (B is a multiple of 4). */
extern __shared__ __align__(16) int wgm_cb_dyn[];
static_assert(__alignof__(wgm_cb_dyn) >= 16, "wgm_cb_finish moves int4 words");

/* Append the lanes' edges of four windows to the block's lists: target k,
 * source rank j; late when lo2 <= j < lo, inner when lo <= j < lo + k. */
__device__ __forceinline__ bool wgm_cb_emit(const int (&k)[4], const int (&j)[4], int lo, int lo2,
                                            int *counter, unsigned *list) {
  const int lane = wgm_lane();
  unsigned ml[4], mi[4];
  int nl = 0, ni = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    ml[q] = __ballot_sync(WGM_FULL, j[q] >= lo2 && j[q] < lo);
    mi[q] = __ballot_sync(WGM_FULL, j[q] >= lo && j[q] < lo + k[q]);
    nl += __popc(ml[q]);
    ni += __popc(mi[q]);
  }
  if ((nl | ni) == 0) return true;
  int base = 0; /* both counters at once */
  if (lane < 2 && (lane ? ni : nl)) base = atomicAdd(counter + lane, lane ? ni : nl);
  int bl = __shfl_sync(WGM_FULL, base, 0), bi = __shfl_sync(WGM_FULL, base, 1);
  if (bl + nl > WGM_CB_LATE || bi + ni > WGM_CB_INNER) return false;
  bi += WGM_CB_LATE;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if ((ml[q] >> lane) & 1u)
      list[bl + __popc(ml[q] & wgm_lanemask_lt())] = (unsigned)k[q] << 16 | (unsigned)(j[q] - lo2);
    if ((mi[q] >> lane) & 1u)
      list[bi + __popc(mi[q] & wgm_lanemask_lt())] = (unsigned)k[q] << 16 | (unsigned)(j[q] - lo);
    bl += __popc(ml[q]);
    bi += __popc(mi[q]);
  }
  return true;
}

/* What a warp's first step of stage A reads and no barrier orders: its
 * vertices' records and the targets of their first 128 edges. */
struct wgm_cb_first {
  int4 o;
  int own[4], j[4];
};

/* Vertices per warp of stage A: few, so that a block's edges spread over
 * every warp. */
__device__ __forceinline__ int wgm_cb_per(int n, int NW) {
  return max(1, min(32, (n + NW - 1) / NW));
}

/* Owner lane and target rank of the edge slots w .. w + 127. */
__device__ __forceinline__ void wgm_cb_load(const int *crank, int off, int base, int total, int w,
                                            int (&own)[4], int (&j)[4]) {
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const int sl = w + 32 * p + wgm_lane();
    own[p] = wgm_owner_of(off, min(sl, total - 1));
    const int e = __shfl_sync(WGM_FULL, base, own[p]) + sl;
    j[p] = sl < total ? __ldg(&crank[e]) : INT_MAX;
  }
}

/* Degree as stage A walks it: hubs go by windows, a degree-1 vertex skips
 * its neighbour (color.cl:46). */
__device__ __forceinline__ int wgm_cb_degree(const int4 &o) {
  return o.w >= 0 || o.z == 1 ? 0 : o.z;
}

__device__ __forceinline__ wgm_cb_first wgm_cb_prefetch(const wgm_color_args &a,
                                                        const wgm_color_blocks_args &q, int b,
                                                        int gw, int NW) {
  const int lane = wgm_lane(), lo = b * q.B, n = min(q.B, a.V - lo);
  const int per = wgm_cb_per(n, NW), k = gw * per + lane;
  wgm_cb_first F;
  F.o = lane < per && k < n ? __ldg(&q.ord[lo + k]) : make_int4(0, 0, 0, -1);
  const int deg = wgm_cb_degree(F.o), incl = wgm_warp_incl_scan(deg);
  const int total = __shfl_sync(WGM_FULL, incl, 31), off = incl - deg;
  wgm_cb_load(q.crank, off, F.o.y - off, total, 0, F.own, F.j);
  return F;
}

/* Stage A of block b on warp gw of NW.  Returns false on a full list. */
__device__ __forceinline__ bool wgm_cb_look(const wgm_color_args &a,
                                            const wgm_color_blocks_args &q, int b, int gw, int NW,
                                            wgm_cb_first &F, wgm_warp_smem *sm) {
  const int lane = wgm_lane(), warp = threadIdx.x >> 5;
  const int lo = b * q.B, n = min(q.B, a.V - lo), lo2 = lo - q.B; /* < 0 for block 0 */
  int *cnt = &q.cnt[(b % 3) * WGM_LINE];
  unsigned *list = q.list + (size_t)(b & 1) * WGM_CB_LISTS;
  int *acc = sm->acc[warp];
  bool ok = true;
  const int per = wgm_cb_per(n, NW);
  for (int k0 = gw * per; k0 < n; k0 += NW * per) {
    const bool mine = lane < per && k0 + lane < n, first = k0 == gw * per;
    if (!first) F.o = mine ? __ldg(&q.ord[lo + k0 + lane]) : make_int4(0, 0, 0, -1);
    const int4 o = F.o;
    const int deg = wgm_cb_degree(o);
    acc[lane] = 0;
    const int incl = wgm_warp_incl_scan(deg);
    const int total = __shfl_sync(WGM_FULL, incl, 31);
    const int off = incl - deg;
    __syncwarp();
    for (int w = 0; w < total; w += 128) {
      int c[4], k[4];
      if (!first || w) wgm_cb_load(q.crank, off, o.y - off, total, w, F.own, F.j);
#pragma unroll
      for (int p = 0; p < 4; p++) c[p] = F.j[p] < lo2 ? __ldca(&q.colour[F.j[p]]) : 0;
#pragma unroll
      for (int p = 0; p < 4; p++) {
        k[p] = k0 + F.own[p];
        if (c[p] > 0) atomicMax(&acc[F.own[p]], c[p]);
      }
      ok &= wgm_cb_emit(k, F.j, lo, lo2, cnt, list);
    }
    __syncwarp();
    if (mine) q.colour[lo + k0 + lane] = acc[lane] + 1;
    __syncwarp();
  }
  /* the block's hubs, a window of 32 edges at a time, last warps first */
  const int h0 = __ldg(&q.blk_hub[b]), h1 = __ldg(&q.blk_hub[b + 1]);
  if (h0 < h1) {
    const int w0 = __ldg(&a.hubs.prefix[h0]) >> 5, w1 = (__ldg(&a.hubs.prefix[h1]) + 31) >> 5;
    const int4 *wrec = reinterpret_cast<const int4 *>(a.hubs.wmap);
    for (int k0 = w0 + (NW - 1 - gw) * 4; k0 < w1; k0 += NW * 4) {
      int4 w[4];
      int j[4], c[4], k[4];
#pragma unroll
      for (int p = 0; p < 4; p++) w[p] = __ldg(wrec + min(k0 + p, w1 - 1));
#pragma unroll
      for (int p = 0; p < 4; p++) {
        int h, e;
        wgm_hub_slot(w[p], lane, &h, &e);
        const bool in =
            k0 + p < w1 && (k0 + p) * 32 + lane < a.hubs.total && h >= h0 && h < h1;
        j[p] = in ? __ldg(&q.crank[e]) : INT_MAX;
        k[p] = in ? __ldg(&q.hub_rank[h]) - lo : 0;
      }
#pragma unroll
      for (int p = 0; p < 4; p++) c[p] = j[p] < lo2 ? __ldca(&q.colour[j[p]]) : 0;
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const bool first = lane < w[p].z;
        const int m0 = __reduce_max_sync(WGM_FULL, first ? c[p] : 0);
        const int m1 = __reduce_max_sync(WGM_FULL, first ? 0 : c[p]);
        if (lane == 0 && m0 > 0) atomicMax(&q.hub_max[w[p].x], m0);
        if (lane == 0 && m1 > 0) atomicMax(&q.hub_max[w[p].x + 1], m1);
      }
      ok &= wgm_cb_emit(k, j, lo, lo2, cnt, list);
    }
  }
  return ok;
}

/* Stage B of block b on this CTA (every thread): returns the thread's
 * largest colour, or -1 to every thread when the block did not settle (a
 * broken layout only).  A function of its own: its registers and those of the
 * prefetched step of stage A never live at once. */
static __device__ __noinline__ int wgm_cb_finish(int V, int B, int b, int *colour,
                                                 const unsigned *lists, int *cnts,
                                                 const int *blk_hub, const int *hub_rank,
                                                 const int *hub_max) {
  const int T = blockDim.x, lo = b * B, nv = min(B, V - lo);
  const unsigned *list = lists + (size_t)(b & 1) * WGM_CB_LISTS;
  int *cnt = cnts + (b % 3) * WGM_LINE;
  int *cur = wgm_cb_dyn + (b & 1) * B;
  const int *prev = wgm_cb_dyn + ((b + 1) & 1) * B;
  /* everything a thread reads is in flight before it waits: the lists' first
   * entries beside their lengths, the block's colours */
  constexpr int KL = 8, KI = 4;
  unsigned late[KL], in[KI];
  const int2 n2 = __ldcg(reinterpret_cast<const int2 *>(cnt));
#pragma unroll
  for (int p = 0; p < KI; p++) {
    const int e = threadIdx.x + p * T;
    in[p] = e < WGM_CB_INNER ? __ldcg(&list[WGM_CB_LATE + e]) : 0u;
  }
#pragma unroll
  for (int p = 0; p < KL; p++) {
    const int e = threadIdx.x + p * T;
    late[p] = e < WGM_CB_LATE ? __ldcg(&list[e]) : 0u;
  }
  const int h0 = __ldg(&blk_hub[b]), h1 = __ldg(&blk_hub[b + 1]);
  for (int k0 = 4 * threadIdx.x; k0 < nv; k0 += 16 * T) { /* lo is a multiple of 4 */
    int4 c[4];
#pragma unroll
    for (int p = 0; p < 4; p++)
      if (k0 + 4 * p * T < nv)
        c[p] = __ldcg(reinterpret_cast<const int4 *>(&colour[lo + k0 + 4 * p * T]));
#pragma unroll
    for (int p = 0; p < 4; p++)
      if (k0 + 4 * p * T < nv) *reinterpret_cast<int4 *>(&cur[k0 + 4 * p * T]) = c[p];
  }
  const int nl = min(n2.x, WGM_CB_LATE), ni = min(n2.y, WGM_CB_INNER);
  if (threadIdx.x == 0) wgm_cb_dyn[2 * B] = 0;
  __syncthreads();
  for (int h = h0 + threadIdx.x; h < h1; h += T)
    atomicMax(&cur[__ldg(&hub_rank[h]) - lo], __ldcg(&hub_max[h]) + 1);
  for (int e0 = threadIdx.x; e0 < nl; e0 += KL * T) {
    if (e0 >= KL * T) {
#pragma unroll
      for (int p = 0; p < KL; p++) late[p] = e0 + p * T < nl ? __ldcg(&list[e0 + p * T]) : 0u;
    }
    /* few exceed what earlier blocks gave their target */
    int c[KL], d[KL];
#pragma unroll
    for (int p = 0; p < KL; p++) {
      const bool have = e0 + p * T < nl;
      c[p] = have ? prev[late[p] & 0xffffu] : 0;
      d[p] = have ? cur[late[p] >> 16] : 1;
    }
#pragma unroll
    for (int p = 0; p < KL; p++)
      if (c[p] >= d[p]) atomicMax(&cur[late[p] >> 16], c[p] + 1);
  }
  __syncthreads();
  /* Inner edges, all at once until a sweep changes nothing.  A look at four
   * edges takes about 200 cycles and a CTA barrier with its vote 260, so a
   * sweep looks three times (13 links: 4600 cycles, against 6750 with one
   * look).  An absent edge reads a word that stays 0.  Plain stores do: of
   * two that meet, the smaller may stay, but its loser is still violated at
   * the next look, and no value ever passes the true colour. */
  volatile int *col = cur;
  int src[KI], dst[KI];
#pragma unroll
  for (int p = 0; p < KI; p++) {
    const bool have = (int)threadIdx.x + p * T < ni;
    src[p] = have ? (int)(in[p] & 0xffffu) : (2 - (b & 1)) * B;
    dst[p] = have ? (int)(in[p] >> 16) : 0;
  }
  for (int sweeps = wgm_proto_chain_sweeps(ni);;) {
    bool changed = false;
#pragma unroll 1
    for (int look = 0; look < 3; look++) {
      int c[KI], d[KI];
#pragma unroll
      for (int p = 0; p < KI; p++) {
        c[p] = col[src[p]];
        d[p] = col[dst[p]];
      }
#pragma unroll
      for (int p = 0; p < KI; p++)
        if (c[p] >= d[p]) {
          col[dst[p]] = c[p] + 1;
          changed = true;
        }
    }
    for (int e = threadIdx.x + KI * T; e < ni; e += T) { /* dense blocks */
      const unsigned y = __ldcg(&list[WGM_CB_LATE + e]);
      const int c = col[y & 0xffffu] + 1;
      if (c > col[y >> 16]) {
        col[y >> 16] = c;
        changed = true;
      }
    }
    if (!__syncthreads_or(changed)) break;
    if (--sweeps == 0) return -1;
  }
  int m = 0;
  for (int k = 4 * threadIdx.x; k < nv; k += 4 * T) {
    const int4 c = *reinterpret_cast<const int4 *>(&cur[k]);
    *reinterpret_cast<int4 *>(&colour[lo + k]) = c;
    m = max(m, c.x);
    if (k + 1 < nv) m = max(m, c.y);
    if (k + 2 < nv) m = max(m, c.z);
    if (k + 3 < nv) m = max(m, c.w);
  }
  /* this line counts block b + 3 next; its pushes begin two barriers on */
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  return m;
}

/* ------------------------------------------------------------------------ */
/* Pannotia colour without rounds (standalone runs)                          */
/* ------------------------------------------------------------------------ */

/* colour(v) = 1 + the largest colour among v's larger out-neighbours (1 if
 * none; degree-1 vertices 1), the recurrence wgm_phase_color computes a
 * round at a time.  Nothing forces rounds: a vertex can take its colour the
 * moment its last larger out-neighbour has one.  So after the same counts
 * (wgm_phase_color's target 3) every warp works from a queue of release
 * pieces - up to 32 in-edges of a coloured vertex with its value and colour
 * - and, for every in-neighbour w smaller than it, raises cmax[w] to
 * colour + 1 and takes one off pending[w] with an acq_rel atomic; the lane
 * that takes the last one (it reads every raise of cmax[w], ordered before
 * the other decrements) colours w with cmax[w] and queues w's in-edges.  A
 * vertex of at most 32 in-edges goes to its warp's own stack in shared
 * memory and is released by that warp next; larger ones go to the global
 * queue in pieces.  Measured against the round form it loses: on RMAT-20
 * 16 ms against 8.3 ms (1629 colours, ~10 us per link of the longest chain
 * against ~5 us per round), because that chain runs through high-degree
 * vertices whose releases pass the global queue (a reservation, the piece
 * written and seen, its fields read) where a round spreads them over every
 * warp behind one barrier.  So rounds stay the default.  Degree-1 vertices start at
 * pending 0 (coloured 1) and releases only take them below 0, so they are
 * never coloured again - the reference's quirk (color.cl:46).  Colours are
 * the round-based form's, bit for bit; the run reports the largest colour
 * as its round count. */
#define WGM_CA_STACK 64
/* vertices of at most this many in-edges stay on their warp's stack;
 * larger ones go to the global queue in pieces.  Keeping up to 1024 on the
 * stack (32 edges a step) made RMAT-20 5x slower: the longest colour chains
 * run through high-degree vertices, whose releases must spread over many
 * warps at once. */
#define WGM_CA_LOCAL_MAX 32
struct wgm_color_async_args {
  int4 *tcv4;   /* [in-edges] {in-neighbour w, bits of w's value, w's first
                   in-edge, w's in-degree} */
  int *cmax;    /* [V] 1 + the largest releaser colour so far */
  int *q_start, *q_cnt, *q_val, *q_col; /* [qcap] release pieces (q_cnt -1 until
                                           written, with release) */
  int qcap;
  int *ctl;     /* lines: 0 queue head, 1 tail, 2 pieces done, 3 pieces in all,
                   4 largest colour */
};
struct wgm_ca_stack { /* per warp, shared memory: pieces of one edge window */
  int start[WGM_CA_STACK], cnt[WGM_CA_STACK], val[WGM_CA_STACK], col[WGM_CA_STACK];
  int n;
};

/* Init (between barriers): colours, pending counts, cmax, the in-edge
 * records, the queue's ready words and the control lines. */
__device__ __forceinline__ void wgm_color_async_init(const wgm_cta *c, const wgm_color_args &a,
                                                     const wgm_color_async_args &q) {
  const wgm_split s(c);
  const int V = a.V;
  for (int i = s.tid; i < V; i += s.nth) {
    a.color[i] = -1;
    a.pending[i] = 0;
    q.cmax[i] = 0;
  }
  const int ET = __ldg(&a.trow[V]);
  for (int e = s.tid; e < ET; e += s.nth) {
    const int w = __ldg(&a.tcol[e]);
    const int t0 = __ldg(&a.trow[w]);
    q.tcv4[e] = make_int4(w, __float_as_int(__ldg(&a.node_value[w])), t0,
                          __ldg(&a.trow[w + 1]) - t0);
  }
  for (int i = s.tid; i < q.qcap; i += s.nth) q.q_cnt[i] = -1;
  if (c->id == 0 && threadIdx.x < 5) q.ctl[threadIdx.x * WGM_LINE] = 0;
}

/* Queue the release pieces of the flagged lanes' vertices (vertex record
 * rec = tcv4-style {w, value bits, first in-edge, in-degree}, colour cw):
 * one-piece vertices onto the warp's stack while it has room, the rest onto
 * the global queue.  Warp-collective.  Returns false on a full queue. */
__device__ __forceinline__ bool wgm_ca_push(bool flag, int4 rec, int cw,
                                            const wgm_color_async_args &q, wgm_ca_stack *st) {
  const int lane = wgm_lane();
  const int deg = flag ? rec.w : 0;
  bool local = deg > 0 && deg <= WGM_CA_LOCAL_MAX;
  const unsigned lm = __ballot_sync(WGM_FULL, local);
  const int nloc = __popc(lm);
  int n0 = 0;
  if (lane == 0) n0 = st->n;
  n0 = __shfl_sync(WGM_FULL, n0, 0);
  if (n0 + nloc > WGM_CA_STACK) local = false;
  if (local) {
    const int k = n0 + __popc(lm & wgm_lanemask_lt());
    st->start[k] = rec.z;
    st->cnt[k] = deg;
    st->val[k] = rec.y;
    st->col[k] = cw;
  }
  __syncwarp();
  if (lane == 0 && n0 + nloc <= WGM_CA_STACK) st->n = n0 + nloc;
  __syncwarp();
  const int np = (deg > 0 && !local) ? (deg + 31) >> 5 : 0;
  const int incl = wgm_warp_incl_scan(np);
  const int total = __shfl_sync(WGM_FULL, incl, 31);
  if (total == 0) return true;
  int base = 0;
  if (lane == 31) base = atomicAdd(&q.ctl[1 * WGM_LINE], total);
  base = __shfl_sync(WGM_FULL, base, 31);
  if (base + total > q.qcap) return false;
  const int first = base + incl - np;
  /* a few pieces per lane, else the whole warp writes one vertex's pieces */
  if (np <= 4) {
    for (int k = 0; k < np; k++) {
      const int slot = first + k;
      q.q_start[slot] = rec.z + 32 * k;
      q.q_val[slot] = rec.y;
      q.q_col[slot] = cw;
      wgm_st_release_gpu(&q.q_cnt[slot], min(32, deg - 32 * k));
    }
  }
  unsigned big = __ballot_sync(WGM_FULL, np > 4);
  while (big) {
    const int j = __ffs(big) - 1;
    big &= big - 1;
    const int bz = __shfl_sync(WGM_FULL, rec.z, j), by = __shfl_sync(WGM_FULL, rec.y, j);
    const int bd = __shfl_sync(WGM_FULL, deg, j), bf = __shfl_sync(WGM_FULL, first, j);
    const int bc = __shfl_sync(WGM_FULL, cw, j);
    for (int k = lane; k < (bd + 31) >> 5; k += 32) {
      q.q_start[bf + k] = bz + 32 * k;
      q.q_val[bf + k] = by;
      q.q_col[bf + k] = bc;
      wgm_st_release_gpu(&q.q_cnt[bf + k], min(32, bd - 32 * k));
    }
  }
  return true;
}

/* Seeding (between barriers, after the counts): every vertex without a
 * larger out-neighbour takes colour 1 and is queued; the pieces of every
 * vertex's in-edges are counted (each vertex is coloured exactly once). */
__device__ __forceinline__ bool wgm_color_async_seed(const wgm_cta *c, const wgm_color_args &a,
                                                     const wgm_color_async_args &q,
                                                     wgm_ca_stack *st) {
  const wgm_split s(c);
  const int V = a.V, lane = s.lane;
  bool ok = true;
  int pieces = 0;
  for (int b = s.gw * 32; b < V; b += s.NW * 32) {
    const int i = b + lane;
    int4 rec = make_int4(0, 0, 0, 0);
    bool f = false;
    if (i < V) {
      const int t0 = __ldg(&a.trow[i]);
      rec = make_int4(i, __float_as_int(__ldg(&a.node_value[i])), t0, __ldg(&a.trow[i + 1]) - t0);
      pieces += (rec.w + 31) >> 5;
      f = __ldcg(&a.pending[i]) == 0;
      if (f) a.color[i] = 1;
    }
    /* seeds go to the global queue: any warp may take them */
    if (lane == 0) st->n = WGM_CA_STACK;
    __syncwarp();
    ok &= wgm_ca_push(f, rec, 1, q, st);
    __syncwarp();
  }
  if (lane == 0) st->n = 0;
  for (int o = 16; o > 0; o >>= 1) pieces += __shfl_xor_sync(WGM_FULL, pieces, o);
  if (lane == 0 && pieces) atomicAdd(&q.ctl[3 * WGM_LINE], pieces);
  if (lane == 0 && V > 0) atomicMax(&q.ctl[4 * WGM_LINE], 1);
  return ok;
}

/* The release loop (no barrier): returns false when a wait gave up or the
 * queue overflowed. */
__device__ __forceinline__ bool wgm_color_async_run(const wgm_launch &L, const wgm_color_args &a,
                                                    const wgm_color_async_args &q,
                                                    wgm_ca_stack *st) {
  const int lane = wgm_lane();
  const int T = __ldcg(&q.ctl[3 * WGM_LINE]);
  bool ok = true;
  int cmax_seen = 0;
  int mydone = 0; /* 32-edge steps released by this warp, not yet counted */
  for (;;) {
    int start = 0, cnt = 0, val = 0, col = 0, have = 0;
    if (lane == 0) {
      if (st->n > 0) {
        const int k = st->n - 1;
        start = st->start[k];
        cnt = st->cnt[k];
        val = st->val[k];
        col = st->col[k];
        have = 1;
        if (cnt > 32) { /* the rest of its in-edges stays on the stack */
          st->start[k] = start + 32;
          st->cnt[k] = cnt - 32;
          cnt = 32;
        } else {
          st->n = k;
        }
      } else {
        /* the steps this warp released count before it waits */
        if (mydone) wgm_red_add_release_gpu(&q.ctl[2 * WGM_LINE], mydone);
        mydone = 0;
        const int i = atomicAdd(&q.ctl[0], 1);
        if (i < T && i < q.qcap) {
          wgm_spin sp = wgm_spin_start(L);
          for (;;) {
            cnt = wgm_ld_acquire_gpu(&q.q_cnt[i]);
            if (cnt >= 0) {
              have = 1;
              break;
            }
            /* every piece was released elsewhere: slot i stays empty */
            if ((sp.n & 7u) == 7u && wgm_ld_relaxed_gpu(&q.ctl[2 * WGM_LINE]) >= T) break;
            if (wgm_spin_giveup(L, sp, WGM_SITE_QUEUE)) {
              ok = false;
              break;
            }
            /* a waiting warp polls gently: the releasing ones need the L2 */
            if (sp.n > 4) __nanosleep(100);
          }
          if (have) {
            start = __ldcg(&q.q_start[i]);
            val = __ldcg(&q.q_val[i]);
            col = __ldcg(&q.q_col[i]);
          }
        }
      }
    }
    have = __shfl_sync(WGM_FULL, have, 0);
    if (!have) break;
    start = __shfl_sync(WGM_FULL, start, 0);
    cnt = __shfl_sync(WGM_FULL, cnt, 0);
    val = __shfl_sync(WGM_FULL, val, 0);
    col = __shfl_sync(WGM_FULL, col, 0);
    bool ready = false;
    int4 rec = make_int4(0, 0, 0, 0);
    int cw = 0;
    if (lane < cnt) {
      rec = __ldcg(&q.tcv4[start + lane]); /* written by this launch's init */
      /* w has the released vertex as a larger out-neighbour */
      if (__int_as_float(rec.y) < __int_as_float(val)) {
        atomicMax(&q.cmax[rec.x], col + 1);
        ready = wgm_atom_add_acqrel_gpu(&a.pending[rec.x], -1) == 1;
        if (ready) {
          cw = __ldcg(&q.cmax[rec.x]);
          a.color[rec.x] = cw;
          cmax_seen = max(cmax_seen, cw);
        }
      }
    }
    ok &= wgm_ca_push(ready, rec, cw, q, st);
    mydone++;
  }
  if (lane == 0 && mydone) wgm_red_add_release_gpu(&q.ctl[2 * WGM_LINE], mydone);
  for (int o = 16; o > 0; o >>= 1) cmax_seen = max(cmax_seen, __shfl_xor_sync(WGM_FULL, cmax_seen, o));
  if (lane == 0 && cmax_seen) atomicMax(&q.ctl[4 * WGM_LINE], cmax_seen);
  return ok;
}

/* ------------------------------------------------------------------------ */
/* Pannotia MIS                                                              */
/* ------------------------------------------------------------------------ */

struct wgm_mis_args {
  int V;
  const int *row;
  const int *col;
  const float *node_value;
  int *s_array;   /* [V] output: 2 = member, 0 = not */
  int2 *word;     /* [V] {status, value bits}; status: -1 active, 2r removed in
                     round r, 2r+1 joined in r */
  int *ptr;       /* [V] first edge that can still hold a blocker */
  unsigned *mask; /* [ceil(V/32)] bit: the vertex may still be active */
  int *stop;      /* [3 lines] by round mod 3: word 0 any active, word 1 wide entries */
  int4 *wide;     /* [wide_cap] this round's {vertex, first edge, first blocker, 0} */
  int wide_cap;   /* >= vertices of more than `scan` edges */
  int scan;       /* edges of one vertex that a single warp looks at */
  int *rounds_out;
};

/* The reference's c_array/cu_array pair (mis.cl:73-118) becomes one status
 * word stamped with the round: a vertex is "active at the start of round r"
 * iff status == -1 or status>>1 == r, which is exactly what mis1/mis2 of round
 * r see in the reference (cu is only committed to c in mis3, after the
 * barrier).  That lets mis1+mis2+mis3 run between two barriers instead of
 * three; s_array, the only output the reference checks (mis.h:199-202), is
 * identical. */
__device__ __forceinline__ bool wgm_active_at(int st, int r) {
  return st == -1 || (st >> 1) == r;
}

/* Is edge target j a blocker of a vertex of value v in round r? */
__device__ __forceinline__ bool wgm_mis_blocks(const wgm_mis_args &a, int j, float v, int r) {
  const int2 w = __ldca(&a.word[j]);
  return __int_as_float(w.y) < v && wgm_active_at(w.x, r);
}

/* Remove the active targets of the lanes' edges start .. start + deg
 * (warp-collective, four 32-edge windows in flight; mis.cl:86-93). */
__device__ __forceinline__ void wgm_mis_mark(const wgm_mis_args &a, int r, int start, int deg) {
  const int lane = wgm_lane();
  const int incl = wgm_warp_incl_scan(deg);
  const int total = __shfl_sync(WGM_FULL, incl, 31);
  const int off = incl - deg, base = start - off;
  for (int w = 0; w < total; w += 128) {
    int j[4], st[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int sl = w + 32 * q + lane;
      const int o = wgm_owner_of(off, min(sl, total - 1));
      const int e = __shfl_sync(WGM_FULL, base, o) + sl;
      j[q] = sl < total ? __ldg(&a.col[e]) : -1;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) st[q] = j[q] >= 0 ? __ldcg(&a.word[j[q]].x) : 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (st[q] == -1) a.word[j[q]].x = 2 * r; /* once: a hub has many joining neighbours */
  }
}

/* First blocker among the edges of the 128-edge steps e0, e0 + stride, ...
 * below `end` (warp-collective, a step's four windows in flight); INT_MAX if
 * none. */
__device__ __forceinline__ int wgm_mis_scan(const wgm_mis_args &a, long long e0, int end,
                                            int stride, float v, int r) {
  const int lane = wgm_lane();
  for (long long x = e0; x < end; x += stride) {
    const int e = (int)x;
    int j[4];
#pragma unroll
    for (int q = 0; q < 4; q++) j[q] = 32 * q + lane < end - e ? __ldg(&a.col[e + 32 * q + lane]) : -1;
    bool hit[4];
#pragma unroll
    for (int q = 0; q < 4; q++) hit[q] = j[q] >= 0 && wgm_mis_blocks(a, j[q], v, r);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const unsigned m = __ballot_sync(WGM_FULL, hit[q]);
      if (m) return e + 32 * q + __ffs(m) - 1;
    }
  }
  return INT_MAX;
}

/* Round r of the lanes' vertices i (act: the lane has one that may still be
 * active; cleared when it is not).  Returns whether the vertex stays. */
__device__ __forceinline__ bool wgm_mis_visit(const wgm_launch &Lc, const wgm_mis_args &a, int r,
                                              int i, bool &act, int *tab) {
  const int lane = wgm_lane();
  const float BIG = (float)WGM_PANNOTIA_BIG;
  int e = 0, start = 0, end = 0;
  float v = 0.f;
  if (act) {
    const int2 w = __ldcg(&a.word[i]);
    act = wgm_active_at(w.x, r);
    v = __int_as_float(w.y);
    start = __ldg(&a.row[i]);
    end = __ldg(&a.row[i + 1]);
    e = r == 1 ? start : __ldcg(&a.ptr[i]);
  }
  const int e0 = e;
  bool wide;
  const bool blocked = wgm_first_edge(a.col, act, e, end, a.scan, wide, tab,
                                      [&](bool valid, int j, int owner) {
                                        const float ov = __shfl_sync(WGM_FULL, v, owner);
                                        return valid && wgm_mis_blocks(a, j, ov, r);
                                      });
  bool join = act && !blocked && !wide && v < BIG;
  if (join) {
    a.s_array[i] = 2;
    a.word[i].x = 2 * r + 1;
    wide = end - start > a.scan; /* its marks are the grid's */
  }
  if (wide) {
    const int b = atomicAdd(&a.stop[(r % 3) * WGM_LINE + 1], 1);
    if (b < a.wide_cap)
      a.wide[b] = make_int4(i, e, INT_MAX, 0);
    else
      wgm_fail(Lc, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, r);
  }
  if (__any_sync(WGM_FULL, join && !wide))
    wgm_mis_mark(a, r, start, join && !wide ? end - start : 0);
  if (act && !join && (e != e0 || r == 1)) a.ptr[i] = e;
  return act && !join;
}

/* A vertex joins when no active out-neighbour has a smaller value
 * (mis.cl:68-75: value < the minimum over active neighbours), so a look
 * stops at the first such neighbour - its blocker - and the next round goes
 * on from there: a neighbour that did not block (larger, or gone) never will
 * again, statuses only leave "active".  Over all rounds every edge is looked
 * at about once at most instead of once per round: on RMAT-20 (31.4 M edges,
 * 8 rounds) 5.1 M looks and 2.6 M marks against ~100 M looks, 1.37 ms ->
 * 0.23 ms.  What bounds it now is one round's chain of dependent round trips
 * (mask, status and row, column, neighbour, then the marks and the barrier:
 * 8 us for a round with a handful of vertices, 54 us for the first, which
 * touches every row).  Two details that cost more than the looks did: a
 * removed mark is stored only over "active" (a hub has tens of thousands of
 * joining neighbours; storing it each time made round 1 take 328 us), and
 * the looks read through L1 - a status read stale within a round reads as
 * the same "active at its start".
 *
 * The vertices that may still be active are kept as one mask word per 32; a
 * warp owns every NW-th word and packs the vertices left in them 32 at a
 * time, so a late round's few do not take a pass per word.  Each lane first
 * looks at four edges of its own vertex (enough for nine in ten on RMAT
 * graphs), then the warp shares the longer rows, 128 edges a step.  A vertex
 * with more than `scan` edges left to look at, or to mark, would hold one
 * warp for long: it goes to a short list that the whole grid works off in
 * two extra phases, which run only in rounds that list one.
 * Phases: (0) init; (1,r) looks, joins and marks; (2,r) looks at the listed
 * vertices, or round r+1 at once when none was listed; (3,r) their joins.
 * (1,r) first applies the reference's exit test to round r-1
 * (mis.cl:106-108). */
static __device__ int wgm_phase_mis(const wgm_launch &Lc, wgm_cta *c, const wgm_mis_args &a,
                                    wgm_warp_smem *sm, wgm_step cur, wgm_step *nxt) {
  const wgm_split s(c);
  __shared__ int s_pend[WGM_MAX_WARPS][64];
  const int V = a.V, lane = s.lane, nchunk = (V + 31) >> 5;
  const float BIG = (float)WGM_PANNOTIA_BIG;
  int *tab = sm->tab[s.warp];
  if (cur.target == 0) {
    for (int i = s.tid; i < V; i += s.nth) {
      a.s_array[i] = 0; /* mis.h:58-92 */
      a.word[i] = make_int2(-1, __float_as_int(__ldg(&a.node_value[i])));
    }
    for (int k = s.tid; k < nchunk; k += s.nth)
      a.mask[k] = V - 32 * k >= 32 ? WGM_FULL : (1u << (V & 31)) - 1u;
    if (c->id == 0 && threadIdx.x < 3) {
      a.stop[threadIdx.x * WGM_LINE] = 0;
      a.stop[threadIdx.x * WGM_LINE + 1] = 0;
    }
    *nxt = {1, 1};
    return WGM_PHASE_NEXT;
  }
  int r = cur.round;
  if (cur.target >= 2) {
    const int n = __ldcg(&a.stop[(r % 3) * WGM_LINE + 1]);
    if (n == 0) {
      r++; /* nothing listed: this phase is round r+1's first */
    } else {
      /* S warps share a listed vertex, each taking every S-th step of 128 edges */
      const int S = max(1, s.NW / n), sub = s.gw % S, per = s.NW / S;
      for (int b = s.gw / S; b < n && s.gw < per * S; b += per) {
        const int4 w = __ldcg(&a.wide[b]);
        const int row0 = __ldg(&a.row[w.x]), end = __ldg(&a.row[w.x + 1]);
        const float v = __ldg(&a.node_value[w.x]);
        if (cur.target == 2) {
          const int e = wgm_mis_scan(a, w.y + 128LL * sub, end, S * 128, v, r);
          if (lane == 0 && e != INT_MAX) atomicMin(&a.wide[b].z, e);
        } else if (w.z != INT_MAX) {
          if (lane == 0 && sub == 0) a.ptr[w.x] = w.z;
        } else if (v < BIG) {
          if (lane == 0 && sub == 0) {
            a.s_array[w.x] = 2;
            a.word[w.x].x = 2 * r + 1;
          }
          for (long long e = row0 + 128LL * sub; e < end; e += 128LL * S)
            wgm_mis_mark(a, r, (int)e, lane == 0 ? (int)min(128LL, end - e) : 0);
        }
      }
      *nxt = cur.target == 2 ? wgm_step{3, r} : wgm_step{1, r + 1};
      return WGM_PHASE_NEXT;
    }
  }
  if (r > 1 && __ldcg(&a.stop[((r - 1) % 3) * WGM_LINE]) == 0) {
    if (c->id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = r - 1;
    return WGM_PHASE_DONE;
  }
  if (r > V + 2) {
    wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, r);
    return WGM_PHASE_DONE;
  }
  if (c->id == 0 && threadIdx.x < 2) a.stop[((r + 1) % 3) * WGM_LINE + threadIdx.x] = 0;
  bool any = false;
  /* this warp's chunks are gw, gw + NW, ...: 32 of their masks in one load */
  int *pend = s_pend[s.warp];
  for (long long k0 = s.gw; k0 < nchunk; k0 += 32LL * s.NW) {
    const long long kl = k0 + (long long)lane * s.NW;
    const unsigned ml = kl < nchunk ? __ldcg(&a.mask[kl]) : 0u;
    unsigned todo = __ballot_sync(WGM_FULL, ml != 0u);
    int n = 0;
    while (todo || n) {
      /* gather up to 32 vertices: later rounds leave few in a chunk */
      while (todo && n < 32) {
        const int kc = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned m = __shfl_sync(WGM_FULL, ml, kc);
        if ((m >> lane) & 1u)
          pend[n + __popc(m & wgm_lanemask_lt())] = (int)(k0 + (long long)kc * s.NW) * 32 + lane;
        n += __popc(m);
      }
      __syncwarp();
      bool act = lane < n;
      const bool had = act;
      const int i = act ? pend[lane] : 0;
      const int rest = lane + 32 < n ? pend[lane + 32] : 0;
      __syncwarp();
      if (lane + 32 < n) pend[lane] = rest;
      n = max(n - 32, 0);
      const bool left = wgm_mis_visit(Lc, a, r, i, act, tab);
      any |= act; /* mis.cl:33 */
      if (had && !left) atomicAnd(&a.mask[i >> 5], ~(1u << (i & 31)));
    }
  }
  if (__any_sync(WGM_FULL, any) && lane == 0) a.stop[(r % 3) * WGM_LINE] = 1;
  *nxt = {2, r};
  return WGM_PHASE_NEXT;
}

/* ------------------------------------------------------------------------ */
/* Rows by falling degree (PageRank, Pannotia SSSP)                          */
/* ------------------------------------------------------------------------ */

/* Layout of the apps that pull over every row (wgm_rank_layout): vertices by
 * descending degree ("rank"), rows and columns renumbered so.  Rows of a
 * degree lie together, so a row is worked by as many lanes as it fills and no
 * lane searches for its owner:
 *   ranks [0, wide)          more than part_edges edges: a warp per part_edges
 *   bin 0 [bin_row[0], ..)   a warp, 256 edges a step
 *   bins 1..5                16, 8, 4, 2, 1 lanes, at most 8 edges a lane */
#define WGM_RANK_BINS 6
#define WGM_RANK_BATCH 4
#define WGM_RANK_ROUNDS 8
struct wgm_rank_rows {
  int rows;          /* vertices with edges */
  const int *prow;   /* [rows+1] by rank */
  const int *pcol;   /* [E] ranks */
  const int *pwt;    /* [E] weights (may be null) */
  const int *order;  /* [V] vertex of each rank */
  int wide, parts;   /* wide rows; their parts of at most part_edges each */
  int part_edges;
  const int *part_row; /* [parts] rank of a part's row */
  const int *row_part; /* [wide+1] first part of a row */
  int short_rows;      /* few edges a row on average (wgm_rank_pull) */
  int bin_row[WGM_RANK_BINS + 1];  /* first rank of each bin, then `rows` */
  int bin_task[WGM_RANK_BINS + 1]; /* first warp task of each bin, then their count */
};

/* Every row once: op.none() is the sum of nothing, op.edge(u, w) an edge's
 * term (u < 0: none), op.join(x, y) adds two; then op.row(k, n, x) gets row
 * k's n edges' sum and op.part(unit, k, x) that of one part of a wide row
 * (by lane 0), with op.after_part(unit, k) called by the whole warp.  Rows
 * that op.skip(k) names are left out (no row or part of them is reported).
 * `grab` hands out work, zero before. */
template <bool WEIGHTED, class T, class Op>
__device__ __forceinline__ void wgm_rank_pull(const wgm_rank_rows &R, const wgm_split &s, int *grab,
                                              Op &&op) {
  const int lane = s.lane;
  /* up to eight edges of a lane's row, four unless `more` */
  auto columns = [&](int r0, int n, int l, int g, bool more, int (&u)[8], int (&w)[8]) {
    auto one = [&](int q) {
      const bool in = l + q * g < n;
      u[q] = in ? __ldcs(&R.pcol[r0 + l + q * g]) : -1;
      w[q] = WEIGHTED && in ? __ldcs(&R.pwt[r0 + l + q * g]) : 0;
    };
#pragma unroll
    for (int q = 0; q < 4; q++) one(q);
    if (more) {
#pragma unroll
      for (int q = 4; q < 8; q++) one(q);
    }
  };
  auto reduce = [&](T x, int g) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const T y = __shfl_xor_sync(WGM_FULL, x, o);
      if (o < g) x = op.join(x, y);
    }
    return x;
  };
  /* the edges r0 .. r0 + n on a warp, eight a lane in flight; the next eight
   * columns are read beside this step's terms */
  auto long_row = [&](int r0, int n) {
    T x = op.none();
    int u[8], w[8];
    columns(r0, n, lane, 32, true, u, w);
    for (int i = lane; __any_sync(WGM_FULL, i < n); i += 256) {
      T v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = op.edge(u[q], w[q]);
      columns(r0, n, i + 256, 32, true, u, w);
#pragma unroll
      for (int q = 0; q < 8; q++) x = op.join(x, v[q]);
    }
    return reduce(x, 32);
  };
  /* Work in order of falling degree: a part of a wide row, a row of bin 0, or
   * `batch` warp tasks of the other bins, round the warps by number; with more
   * than WGM_RANK_ROUNDS rounds the last quarter is handed out as warps get
   * free (on fewer, every warp would queue at the counter at once). */
  const int long_units = R.parts + R.bin_task[1];
  const int tasks = R.bin_task[WGM_RANK_BINS] - R.bin_task[1];
  const int batch = max(1, min(WGM_RANK_BATCH, tasks / (4 * s.NW)));
  const int units = long_units + (tasks + batch - 1) / batch;
  const int fixed = units <= WGM_RANK_ROUNDS * s.NW
                        ? units
                        : (int)(3LL * units / 4 / s.NW) * s.NW; /* whole rounds */
  int unit = s.gw;
  while (unit < units) {
    int next = unit + s.NW;
    if (next >= fixed && fixed < units) {
      if (lane == 0) next = atomicAdd(grab, 1);
      next = __shfl_sync(WGM_FULL, next, 0) + max(fixed, s.NW);
    }
    if (unit < long_units) {
      const bool part = unit < R.parts;
      const int k = part ? __ldg(&R.part_row[unit]) : R.bin_row[0] + unit - R.parts;
      const int r0 = __ldg(&R.prow[k]), n = __ldg(&R.prow[k + 1]) - r0;
      const int off = part ? (unit - __ldg(&R.row_part[k])) * R.part_edges : 0;
      /* other parts' warps may be lowering the word that skip reads: one answer
       * for the warp, which works the row together */
      if (!(op.SKIPS && __any_sync(WGM_FULL, op.skip(k)))) {
        const T x = long_row(r0 + off, part ? min(R.part_edges, n - off) : n);
        if (lane == 0) {
          if (part) op.part(unit, k, x);
          else op.row(k, n, x);
        }
        if (part) op.after_part(unit, k, n);
      }
    } else {
      const int x0 = R.bin_task[1] + (unit - long_units) * batch;
      const int x1 = min(x0 + batch, R.bin_task[WGM_RANK_BINS]);
      /* rows of at most 8 edges a lane, in a pipeline over the tasks: the row
       * bounds of task x + 2 and the columns of task x + 1 are read beside
       * the terms of task x */
      auto locate = [&](int x, int &k, int &g, int &r0, int &n) {
        int bn = 1, first = R.bin_row[1], task = R.bin_task[1], end = R.bin_row[2];
#pragma unroll
        for (int q = 2; q < WGM_RANK_BINS; q++)
          if (x >= R.bin_task[q]) {
            bn = q;
            first = R.bin_row[q];
            task = R.bin_task[q];
            end = R.bin_row[q + 1];
          }
        g = 32 >> bn;
        k = first + ((x - task) << bn) + (lane >> (5 - bn));
        r0 = n = 0;
        if (x < x1 && k < end) {
          const bool skip = op.skip(k);
          r0 = __ldg(&R.prow[k]);
          n = skip ? 0 : __ldg(&R.prow[k + 1]) - r0;
        }
      };
      /* Where passes leave rows out and rows are short, a task is mostly
       * instructions for nothing: of rows that are all left out, of slots past
       * four edges a lane where no row has them (more than one lane a row:
       * always more than four each), of the look ahead below.  One task after
       * the other then, without them: Pannotia SSSP on a 512 x 512 grid 9.5 ->
       * 6.9 ms, RMAT of 800,000 vertices and factor 4 0.525 -> 0.455; of 900,000
       * and factor 14, 0.99 in the pipeline and 1.06 with these tests in it. */
      if (op.SKIPS && R.short_rows) {
        for (int x = x0; x < x1; x++) {
          int k0, g0, r0, n0, u[8], w[8];
          locate(x, k0, g0, r0, n0);
          if (!__any_sync(WGM_FULL, n0 > 0)) continue;
          const bool more = g0 > 1 || __any_sync(WGM_FULL, n0 > 4);
          columns(r0, n0, lane & (g0 - 1), g0, more, u, w);
          T sum = op.none();
#pragma unroll
          for (int q = 0; q < 4; q++) sum = op.join(sum, op.edge(u[q], w[q]));
          if (more) {
#pragma unroll
            for (int q = 4; q < 8; q++) sum = op.join(sum, op.edge(u[q], w[q]));
          }
          sum = reduce(sum, g0);
          if (n0 > 0 && (lane & (g0 - 1)) == 0) op.row(k0, n0, sum);
        }
        unit = next;
        continue;
      }
      /* rows of at most 8 edges a lane, in a pipeline over the tasks: the row
       * bounds of task x + 2 and the columns of task x + 1 are read beside
       * the terms of task x */
      int k0, g0, r0, n0, k1, g1, r1, n1, u[8], w[8];
      locate(x0, k0, g0, r0, n0);
      locate(x0 + 1, k1, g1, r1, n1);
      columns(r0, n0, lane & (g0 - 1), g0, true, u, w);
      for (int x = x0; x < x1; x++) {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = op.edge(u[q], w[q]);
        columns(r1, n1, lane & (g1 - 1), g1, true, u, w);
        int k2, g2, r2, n2;
        locate(x + 2, k2, g2, r2, n2);
        T sum = op.none();
#pragma unroll
        for (int q = 0; q < 8; q++) sum = op.join(sum, v[q]);
        sum = reduce(sum, g0);
        if (n0 > 0 && (lane & (g0 - 1)) == 0) op.row(k0, n0, sum);
        k0 = k1;
        g0 = g1;
        n0 = n1;
        k1 = k2;
        g1 = g2;
        r1 = r2;
        n1 = n2;
      }
    }
    unit = next;
  }
}

/* ------------------------------------------------------------------------ */
/* Pannotia SSSP (pull min-plus)                                             */
/* ------------------------------------------------------------------------ */

struct wgm_psssp_args {
  int V;
  wgm_rank_rows R;
  const int *rank; /* [V] rank of each vertex */
  int *xr;         /* [V] cost by rank */
  int *x;          /* [V] output cost (sssp.h:168 reads x) */
  int *stop;       /* [6 lines] by round mod 3: work handed out; then least cost that
                      changed (INT_MAX: none) */
  const int *wmin; /* least edge weight; negative where a pass has to take every row */
  int source;
  int *rounds_out;
};

/* One pass of x[v] = min(x[v], min_j data[j] + x[col[j]]) (wgm_rank_pull). */
struct wgm_psssp_op {
  int *xr;
  int bound;           /* costs up to here cannot fall in this pass */
  int least = INT_MAX; /* least cost that this thread lowered */
  static constexpr bool SKIPS = true;
  __device__ __forceinline__ bool skip(int k) const { return __ldcg(&xr[k]) <= bound; }
  __device__ __forceinline__ int none() const { return INT_MAX; }
  __device__ __forceinline__ int edge(int u, int w) const {
    return u < 0 ? INT_MAX : w + __ldca(&xr[u]);
  }
  __device__ __forceinline__ int join(int x, int y) const { return min(x, y); }
  __device__ __forceinline__ void row(int k, int, int x) {
    if (x < __ldcg(&xr[k])) {
      xr[k] = x; /* the row's only writer */
      least = min(least, x);
    }
  }
  __device__ __forceinline__ void part(int, int k, int x) {
    if (x < __ldcg(&xr[k]) && atomicMin(&xr[k], x) > x) least = min(least, x);
  }
  __device__ __forceinline__ void after_part(int, int, int) {}
};

/* sssp.cl's vector_assign / spmv_min_dot_plus / vector_diff (three barriers
 * per round) become one in-place relaxation pass per round:
 * x[v] = min(x[v], min_j data[j] + x[col[j]]).  The reference's Jacobi
 * iteration and this chaotic (in-place) iteration both stop at the fixpoint
 * of the min-plus system started from x = BIG_NUM except x[source] = 0, which
 * is unique (the shortest-path distances, BIG_NUM where unreachable), so the
 * returned vector is identical; only the round count can be smaller.  Costs
 * are read through the L1: one that another SM has lowered since was lowered
 * in this round, so a next one follows and reads it (a barrier empties the
 * L1).
 * A pass leaves out the rows it cannot change.  With no negative weight, a
 * cost can only fall to (least cost that changed in the pass before) + (least
 * weight) or above: what changed earlier was read in the pass before, or was
 * too large by the same test.  Rows at or under that bound - nearly all of
 * them in the last passes - cost one word.  A 200,003-vertex RMAT graph of
 * 4.5 M edges: 12 passes of 44 us (an owner search and a shared-memory
 * minimum per edge, hubs by windows) -> 18 passes of 25 to 12 us, 0.51 ->
 * 0.33 ms; reading past the L1 takes 15 passes but 1.0 ms, for the hubs'
 * costs share a few lines.  One update of the least changed cost per group:
 * one per warp made a pass 260 us.
 * Phases: (0) init; (1,r) one relaxation pass (after the exit test of r-1);
 * the costs go out by vertex when it ends. */
static __device__ int wgm_phase_pannotia_sssp(const wgm_launch &Lc, wgm_cta *c,
                                              const wgm_psssp_args &a, wgm_step cur,
                                              wgm_step *nxt) {
  const wgm_split s(c);
  const int V = a.V;
  int *changed = a.stop + 3 * WGM_LINE;
  if (cur.target == 0) {
    const int src = __ldg(&a.rank[a.source]);
    for (int k = s.tid; k < V; k += s.nth) a.xr[k] = k == src ? 0 : WGM_PANNOTIA_BIG;
    if (c->id == 0 && threadIdx.x < 3) {
      a.stop[threadIdx.x * WGM_LINE] = 0;
      changed[threadIdx.x * WGM_LINE] = INT_MAX;
    }
    *nxt = {1, 1};
    return WGM_PHASE_NEXT;
  }
  const int r = cur.round;
  const int before = r > 1 ? __ldcg(&changed[((r - 1) % 3) * WGM_LINE]) : 0;
  if (before == INT_MAX) {
    for (int k = s.tid; k < V; k += s.nth) a.x[__ldg(&a.R.order[k])] = __ldcg(&a.xr[k]);
    if (c->id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = r - 1;
    return WGM_PHASE_DONE;
  }
  if (r > V + 2) {
    wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, r);
    return WGM_PHASE_DONE;
  }
  if (c->id == 0 && threadIdx.x == 0) {
    a.stop[((r + 1) % 3) * WGM_LINE] = 0;
    changed[((r + 1) % 3) * WGM_LINE] = INT_MAX;
  }
  const int wmin = __ldg(a.wmin);
  wgm_psssp_op op{a.xr, INT_MIN};
  if (r > 1 && wmin >= 0) op.bound = (int)min((long long)INT_MAX, (long long)before + wmin);
  __shared__ int s_least; /* one update per group: the word is everybody's */
  if (threadIdx.x == 0) s_least = INT_MAX;
  __syncthreads();
  wgm_rank_pull<true, int>(a.R, s, &a.stop[(r % 3) * WGM_LINE], op);
  if (op.least != INT_MAX) atomicMin(&s_least, op.least);
  __syncthreads();
  if (threadIdx.x == 0 && s_least != INT_MAX)
    atomicMin(&changed[(r % 3) * WGM_LINE], s_least);
  *nxt = {1, r + 1};
  return WGM_PHASE_NEXT;
}

/* ------------------------------------------------------------------------ */
/* Pull PageRank (FP32; no reference implementation)                          */
/* ------------------------------------------------------------------------ */

/* Rows by rank; the contributions read most often are the first ones: the
 * first `cached` sit in shared memory (on RMAT-22, 41,000 of 4.2 M vertices
 * take 56 % of all reads). */
struct wgm_pr_args {
  int V;
  wgm_rank_rows R;
  float *pr;         /* [V] output, by vertex */
  float *contrib;    /* [2][stride] pr/deg of the previous iteration, by rank */
  size_t stride;     /* >= V, whole 16-byte words */
  float *dang;       /* [3 lines] by iteration mod 3: dangling mass; word 1 (int):
                        work handed out */
  float *part;       /* [parts] sums */
  int *part_done;    /* [wide] parts summed, zero between iterations */
  int cached;        /* contributions kept in dynamic shared memory */
  int iterations;
  float damping;
  float dangling;    /* vertices without edges */
};

extern __shared__ __align__(16) float wgm_pr_cache[]; /* filled in float4 words */
static_assert(__alignof__(wgm_pr_cache) >= 16, "wgm_phase_pagerank moves float4 words");

/* One iteration over the rows (wgm_rank_pull). */
struct wgm_pr_op {
  const wgm_pr_args &a;
  const float *cin;
  float *cout;
  float base;
  bool last;
  static constexpr bool SKIPS = false;
  __device__ __forceinline__ bool skip(int) const { return false; }
  __device__ __forceinline__ float none() const { return 0.f; }
  __device__ __forceinline__ float edge(int u, int) const {
    return u < 0 ? 0.f : u < a.cached ? wgm_pr_cache[u] : __ldca(&cin[u]);
  }
  __device__ __forceinline__ float join(float x, float y) const { return x + y; }
  __device__ __forceinline__ void row(int k, int deg, float sum) const {
    const float p = base + a.damping * sum;
    cout[k] = p / (float)deg;
    if (last) a.pr[__ldg(&a.R.order[k])] = p;
  }
  __device__ __forceinline__ void part(int unit, int, float x) const { a.part[unit] = x; }
  /* the last part to finish adds up its row's, in their order */
  __device__ __forceinline__ void after_part(int, int k, int n) const {
    const int lane = wgm_lane(), p0 = __ldg(&a.R.row_part[k]);
    const int m = __ldg(&a.R.row_part[k + 1]) - p0;
    int done = 0;
    if (lane == 0) done = wgm_atom_add_acqrel_gpu(&a.part_done[k], 1) == m - 1;
    if (!__shfl_sync(WGM_FULL, done, 0)) return;
    float y = 0.f;
    for (int i = lane; i < m; i += 32) y += __ldcg(&a.part[p0 + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(WGM_FULL, y, o);
    if (lane == 0) {
      a.part_done[k] = 0;
      row(k, n, y);
    }
  }
};

/* pr' = (1-d)/V + d*(sum_{u in N(v)} pr[u]/deg(u) + dangling/V).  Phases:
 * (0) init; (1,t) iteration t, one barrier each.  Every row is summed by the
 * same lanes in the same order in every run, and the dangling mass needs no
 * sum: a vertex without edges has exactly the base value.
 *
 * What bounds an iteration: the gathers.  Contributions by rank put the
 * hot ones into a few lines, which thousands of warps then ask one L2 slice
 * for (1540 us an iteration with every gather from the L2); from shared
 * memory they cost a few cycles, and the L1 takes the next ones.  RMAT-22
 * (128 M edges): 566 us with vertex numbers, every gather from the L2 and an
 * owner search per 32 edges -> 255 us; 174 us if every gather hit shared
 * memory, which is what the columns and the instructions take.  The columns
 * pass by the L1 (ldcs).  RMAT-14: 26 us (two barriers of 760 groups) -> 7 us,
 * one barrier and the round trips bounds - columns - contributions - parts. */
static __device__ int wgm_phase_pagerank(const wgm_launch &Lc, wgm_cta *c, const wgm_pr_args &a,
                                         wgm_step cur, wgm_step *nxt) {
  const wgm_split s(c);
  const int V = a.V;
  const float d = a.damping;
  const int t = cur.round;
  if (cur.target == 0) {
    const float p = 1.0f / (float)V;
    for (int k = s.tid; k < a.R.rows; k += s.nth)
      a.contrib[k] = p / (float)(__ldg(&a.R.prow[k + 1]) - __ldg(&a.R.prow[k]));
    if (a.iterations == 0)
      for (int v = s.tid; v < V; v += s.nth) a.pr[v] = p;
    if (c->id == 0 && threadIdx.x < 3) {
      a.dang[threadIdx.x * WGM_LINE] = a.dangling * p;
      reinterpret_cast<int *>(a.dang)[threadIdx.x * WGM_LINE + 1] = 0;
    }
    for (int k = s.tid; k < a.R.wide; k += s.nth) a.part_done[k] = 0;
    /* a vertex without edges of its own gives nothing to rows that name it */
    for (size_t k = a.R.rows + s.tid; k < a.stride; k += s.nth)
      a.contrib[k] = a.contrib[a.stride + k] = 0.f;
    *nxt = {1, 0};
    return WGM_PHASE_NEXT;
  }
  if (t >= a.iterations) return WGM_PHASE_DONE;
  const float *cin = a.contrib + (size_t)(t & 1) * a.stride;
  float *cout = a.contrib + (size_t)((t + 1) & 1) * a.stride;
  const float base = (1.0f - d) / (float)V + d * __ldcg(&a.dang[(t % 3) * WGM_LINE]) / (float)V;
  const bool last = t + 1 == a.iterations;
  int *grab = reinterpret_cast<int *>(a.dang) + (t % 3) * WGM_LINE + 1;
  if (c->id == 0 && threadIdx.x == 0) {
    a.dang[((t + 1) % 3) * WGM_LINE] = a.dangling * base;
    reinterpret_cast<int *>(a.dang)[((t + 2) % 3) * WGM_LINE + 1] = 0;
  }
  const int cached = a.cached;
  if (cached > 0) { /* a multiple of 4, contrib's rows 16-byte aligned */
    /* each group starts elsewhere, or all would ask for the same lines at once */
    const int turn = (int)((long long)cached * c->id / c->ngroups) & ~3;
    for (int i = 4 * threadIdx.x; i < cached; i += 4 * blockDim.x) {
      const int j = i < cached - turn ? i + turn : i + turn - cached;
      *reinterpret_cast<float4 *>(&wgm_pr_cache[j]) =
          __ldcg(reinterpret_cast<const float4 *>(&cin[j]));
    }
    __syncthreads();
  }
  wgm_pr_op op{a, cin, cout, base, last};
  wgm_rank_pull<false, float>(a.R, s, grab, op);
  if (last)
    for (int k = a.R.rows + s.tid; k < V; k += s.nth) a.pr[__ldg(&a.R.order[k])] = base;
  *nxt = {1, t + 1};
  return WGM_PHASE_NEXT;
}

/* ------------------------------------------------------------------------ */
/* Pannotia betweenness centrality                                           */
/* ------------------------------------------------------------------------ */

struct wgm_bc_args {
  int V;
  const int *row, *col;   /* out-edges */
  const int *trow, *tcol; /* in-edges (the transpose; the graph when symmetric) */
  float *bc;              /* [V] output */
  int *dist;              /* [V] BFS level from the current source, -1 unreached */
  float *rho;             /* [V] shortest-path counts x 10000 */
  float *sigma;           /* [V] dependencies x 10000 */
  int *order;             /* [V] reached vertices, level by level */
  int *level_start;       /* [V + 2] first position of each level in order[] */
  int *cnt;               /* [3 lines] vertices found for a level, by level mod 3 */
  int num_sources;        /* sources 0 .. num_sources-1 (the reference: all V) */
  int *rounds_out;
};

#define WGM_BC_SCALE 10000.0f /* bc.cl:230 and :131: "scaling by 10000" */

/* bc.cl:1-235 (bc_combined: for every source s, clear, BFS with path
 * counts, backtrack with dependencies).  The reference scans every vertex
 * at every level for d[i] == level; here each level is a frontier list:
 * BFS level L relaxes the out-edges of order[level_start[L] ..] and appends
 * the vertices it discovers (one CAS each) as level L+1, so the backtrack
 * walks the same lists in reverse.  Arithmetic is the reference's: rho in
 * float scaled by 10000, rho[w] += rho[i] for every edge from level L to
 * L+1 (bc.cl:52-56), sigma[w] += rho[w] / rho[i] * (10000 + sigma[i]) for
 * every in-edge from level L-1 (bc.cl:122-124), bc[i] += sigma[i] / 10000
 * for every vertex but the source (bc.cl:131); only the order of the float
 * atomic adds differs (as between two runs of the reference).
 * Phases: target = kind | level << 2, round = source: kind 0 clears bc,
 * 1 clears the per-source state, 2 is a BFS level, 3 a backtrack level. */
static __device__ int wgm_phase_bc(const wgm_launch &Lc, wgm_cta *c, const wgm_bc_args &a,
                                   wgm_warp_smem *sm, wgm_step cur, wgm_step *nxt) {
  const wgm_split s(c);
  const int V = a.V, kind = cur.target & 3, L = cur.target >> 2, src = cur.round;
  const int lane = s.lane, warp = s.warp;
  if (kind == 0) {
    for (int i = s.tid; i < V; i += s.nth) a.bc[i] = 0.f;
    if (a.num_sources <= 0) {
      if (c->id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = 0;
      return WGM_PHASE_DONE;
    }
    *nxt = {1, 0};
    return WGM_PHASE_NEXT;
  }
  if (kind == 1) {
    /* clean_1d_array (bc.cl:165-181) */
    for (int i = s.tid; i < V; i += s.nth) {
      a.sigma[i] = 0.f;
      a.rho[i] = i == src ? WGM_BC_SCALE : 0.f;
      a.dist[i] = i == src ? 0 : -1;
    }
    if (c->id == 0 && threadIdx.x == 0) {
      a.order[0] = src;
      a.level_start[0] = 0;
      a.level_start[1] = 1;
      a.cnt[0] = 1;
      a.cnt[1 * WGM_LINE] = 0;
      a.cnt[2 * WGM_LINE] = 0;
    }
    *nxt = {2, src};
    return WGM_PHASE_NEXT;
  }
  if (kind == 2) {
    /* BFS level L (mega_bfs_kernel_func, bc.cl:16-92) */
    const int n = __ldcg(&a.cnt[(L % 3) * WGM_LINE]);
    const int S = __ldcg(&a.level_start[L]);
    if (n == 0) {
      /* no level L: the deepest is L-1, backtrack from it */
      *nxt = {3 | ((L - 1) << 2), src};
      return WGM_PHASE_NEXT;
    }
    if (L + 2 > V + 1) {
      wgm_fail(Lc, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, L);
      return WGM_PHASE_DONE;
    }
    const int S1 = S + n;
    if (c->id == 0 && threadIdx.x == 0) {
      a.level_start[L + 1] = S1;
      a.cnt[((L + 2) % 3) * WGM_LINE] = 0;
    }
    int *ncnt = &a.cnt[((L + 1) % 3) * WGM_LINE];
    for (int b = s.gw * 32; b < n; b += s.NW * 32) {
      const int k = b + lane;
      int v = 0, start = 0, deg = 0;
      float rv = 0.f;
      if (k < n) {
        v = __ldcg(&a.order[S + k]);
        start = __ldg(&a.row[v]);
        deg = __ldg(&a.row[v + 1]) - start;
        rv = __ldcg(&a.rho[v]);
      }
      const int incl = wgm_warp_incl_scan(deg);
      const int total = __shfl_sync(WGM_FULL, incl, 31);
      const int off = incl - deg;
      wgm_for_each_edge(off, deg, start - off, total, 0, 32, sm->tab[warp],
                        [&](bool valid, int e, int owner) {
                          const float ro = __shfl_sync(WGM_FULL, rv, owner);
                          bool found = false;
                          int w = 0;
                          if (valid) {
                            w = __ldg(&a.col[e]);
                            int d = __ldcg(&a.dist[w]);
                            if (d < 0) {
                              d = atomicCAS(&a.dist[w], -1, L + 1);
                              found = d == -1;
                              if (found) d = L + 1;
                            }
                            if (d == L + 1) atomicAdd(&a.rho[w], ro);
                          }
                          wgm_warp_push(found, w, ncnt, a.order + S1, V - S1, false);
                        });
    }
    *nxt = {2 | ((L + 1) << 2), src};
    return WGM_PHASE_NEXT;
  }
  /* backtrack level L (mega_backtrack_kernel_func, bc.cl:96-140) */
  const int S = __ldcg(&a.level_start[L]), E = __ldcg(&a.level_start[L + 1]);
  for (int b = S + s.gw * 32; b < E; b += s.NW * 32) {
    const int k = b + lane;
    int v = 0, start = 0, deg = 0;
    float rv = 1.f, sv = 0.f;
    if (k < E) {
      v = __ldcg(&a.order[k]);
      start = __ldg(&a.trow[v]);
      deg = L > 0 ? __ldg(&a.trow[v + 1]) - start : 0;
      rv = __ldcg(&a.rho[v]);
      sv = __ldcg(&a.sigma[v]);
    }
    const int incl = wgm_warp_incl_scan(deg);
    const int total = __shfl_sync(WGM_FULL, incl, 31);
    const int off = incl - deg;
    wgm_for_each_edge(off, deg, start - off, total, 0, 32, sm->tab[warp],
                      [&](bool valid, int e, int owner) {
                        const float ri = __shfl_sync(WGM_FULL, rv, owner);
                        const float si = __shfl_sync(WGM_FULL, sv, owner);
                        if (valid) {
                          const int w = __ldg(&a.tcol[e]);
                          if (__ldcg(&a.dist[w]) == L - 1)
                            atomicAdd(&a.sigma[w], __ldcg(&a.rho[w]) / ri * (WGM_BC_SCALE + si));
                        }
                      });
    if (k < E && v != src) a.bc[v] = a.bc[v] + sv / WGM_BC_SCALE;
  }
  if (L > 0) {
    *nxt = {3 | ((L - 1) << 2), src};
    return WGM_PHASE_NEXT;
  }
  if (src + 1 >= a.num_sources) {
    if (c->id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = src + 1;
    return WGM_PHASE_DONE;
  }
  *nxt = {1, src + 1};
  return WGM_PHASE_NEXT;
}

/* Betweenness centrality with the sources spread over CTAs: a CTA takes a
 * source from a queue and runs its BFS and backtrack alone, with dist, rho,
 * sigma, the level lists and their starts in shared memory (20 bytes per
 * vertex) and __syncthreads as the level barrier; bc gathers the
 * dependencies with global float atomics.  Same arithmetic as wgm_phase_bc,
 * no grid barrier at all: sources, not levels, are the parallel units.  A
 * vertex's dependencies are added in double precision (a sum over thousands of
 * sources in an order that changes from run to run) and rounded once.  For
 * graphs of at most WGM_BC_CTA_MAX_V vertices. */
#define WGM_BC_CTA_MAX_V 10240


/* Vertices a warp takes of a level of n at a time: at least `few` (two windows
 * of edges at the graph's average degree), and a quarter of an even share.  A
 * level of more than one share per warp is handed out, for a hub's edges
 * keep a warp long: RMAT-12, all sources, 4.14 ms with 32 vertices a warp in
 * turn, 2.72 handed out (512 threads), 2.38 with 1024, a quarter of a warp's
 * share at a time 2.31 (an eighth 2.38), and with two windows of edges in
 * flight 2.18 (four 2.22).  A vertex at a time, 128 of its edges together,
 * was slower (2.72): most rows fill less than a warp.  An edge's row comes
 * from a table of the window's row starts (five dependent shuffles: 2.25,
 * the table 2.12).  EVEN, for graphs of degree up to 4 on average, whose rows
 * differ little: 32 vertices a warp in turn and one window, fewer
 * instructions a level (grid 24 x 24 0.137 -> 0.128 ms, 15 x 8 53 -> 45 us).
 * What bounds small graphs is the chain of a level, about 2000 cycles. */
#define WGM_BC_SHARE 4
#define WGM_BC_K 2 /* 32-edge windows in flight */
__device__ __forceinline__ int wgm_bc_per(int n, int nw, int few) {
  return min(32, max(few, (n + WGM_BC_SHARE * nw - 1) / (WGM_BC_SHARE * nw)));
}
/* First vertex of the warp's next share; `turn` counts its shares. */
__device__ __forceinline__ int wgm_bc_next(int *counter, int n, int per, int warp, int nw,
                                           int turn) {
  if (n <= nw * per) return turn ? n : warp * per;
  int b = 0;
  if (wgm_lane() == 0) b = atomicAdd(counter, per);
  return __shfl_sync(WGM_FULL, b, 0);
}

/* f(valid, target, x of its row's lane) for the edges of the lanes' rows. */
template <int K, class F>
__device__ __forceinline__ void wgm_bc_windows(const int *col, int base, int off, int deg,
                                               int total, int w, float x, int *tab, F &f) {
  const int lane = wgm_lane();
  unsigned mm[K];
  int j[K], own[K];
  float xo[K];
  bool in[K];
#pragma unroll
  for (int q = 0; q < K; q++) {
    const int w1 = w + 32 * q;
    const bool mine = deg > 0 && off < w1 + 32 && off + deg > w1;
    const int pos = mine ? max(off - w1, 0) : 0;
    mm[q] = __reduce_or_sync(WGM_FULL, mine ? 1u << pos : 0u);
    if (mine) tab[32 * q + pos] = lane;
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < K; q++) {
    mm[q] &= 0xffffffffu >> (31 - lane);
    own[q] = tab[32 * q + (mm[q] ? 31 - __clz(mm[q]) : 0)] & 31;
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < K; q++) {
    const int sl = w + 32 * q + lane, e = __shfl_sync(WGM_FULL, base, own[q]) + sl;
    xo[q] = __shfl_sync(WGM_FULL, x, own[q]);
    in[q] = sl < total;
    j[q] = in[q] ? __ldg(&col[e]) : 0;
  }
#pragma unroll
  for (int q = 0; q < K; q++) f(in[q], j[q], xo[q]);
}
template <int K, class F>
__device__ __forceinline__ void wgm_bc_edges(const int *col, int start, int deg, float x, int *tab,
                                             F &&f) {
  const int incl = wgm_warp_incl_scan(deg);
  const int total = __shfl_sync(WGM_FULL, incl, 31), off = incl - deg;
  int w = 0;
  if (K > 1)
    for (; total - w > 32; w += 32 * K)
      wgm_bc_windows<K>(col, start - off, off, deg, total, w, x, tab, f);
  for (; w < total; w += 32) wgm_bc_windows<1>(col, start - off, off, deg, total, w, x, tab, f);
}

template <bool EVEN>
static __device__ void wgm_bc_cta_source(const wgm_bc_args &a, double *bc64, int src, int *dist,
                                         float *rho, float *sig, int *order, int *ls, int *s_cnt,
                                         int *tab, int few) {
  const int V = a.V, lane = wgm_lane(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  tab += warp * 32 * WGM_BC_K;
  /* by level mod 3: vertices found, shares handed out; by backtrack step mod
   * 3: shares handed out.  A level clears the next one's, so it ends in one
   * barrier. */
  int *found_n = s_cnt, *shares = s_cnt + 3, *back = s_cnt + 6;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    dist[i] = i == src ? 0 : -1;
    rho[i] = i == src ? WGM_BC_SCALE : 0.f;
    sig[i] = 0.f;
  }
  if (threadIdx.x == 0) {
    order[0] = src;
    ls[0] = 0;
    ls[1] = 1;
    for (int k = 0; k < 9; k++) s_cnt[k] = 0;
  }
  __syncthreads();
  int L = 0, S = 0, n = 1;
  for (;;) {
    const int S1 = S + n, per = EVEN ? 32 : wgm_bc_per(n, nw, few);
    int *count = &found_n[L % 3];
    if (threadIdx.x == 0) found_n[(L + 1) % 3] = shares[(L + 1) % 3] = 0;
    for (int turn = 0;; turn++) {
      const int b = EVEN ? 32 * (warp + nw * turn)
                         : wgm_bc_next(&shares[L % 3], n, per, warp, nw, turn);
      if (b >= n) break;
      const int k = b + lane;
      int start = 0, deg = 0;
      float rv = 0.f;
      if (lane < per && k < n) {
        const int v = order[S + k];
        start = __ldg(&a.row[v]);
        deg = __ldg(&a.row[v + 1]) - start;
        rv = rho[v];
      }
      wgm_bc_edges<EVEN ? 1 : WGM_BC_K>(a.col, start, deg, rv, tab, [&](bool valid, int w, float ro) {
        bool found = false;
        if (valid) {
          int d = dist[w];
          if (d < 0) {
            d = atomicCAS(&dist[w], -1, L + 1);
            found = d == -1;
            if (found) d = L + 1;
          }
          if (d == L + 1) atomicAdd(&rho[w], ro);
        }
        wgm_warp_push(found, w, count, order + S1, V - S1, false);
      });
    }
    __syncthreads();
    const int n2 = *count;
    if (threadIdx.x == 0) ls[L + 2] = S1 + n2;
    if (n2 == 0) break;
    S = S1;
    n = n2;
    L++;
  }
  __syncthreads(); /* the last level's start */
  for (int l = L; l >= 0; l--) {
    const int B = ls[l], E = ls[l + 1], step = (L - l) % 3, per = EVEN ? 32 : wgm_bc_per(E - B, nw, few);
    if (!EVEN && threadIdx.x == 0) back[(step + 1) % 3] = 0;
    for (int turn = 0;; turn++) {
      const int b = B + (EVEN ? 32 * (warp + nw * turn)
                              : wgm_bc_next(&back[step], E - B, per, warp, nw, turn));
      if (b >= E) break;
      const int k = b + lane;
      const bool have = lane < per && k < E;
      int v = 0, start = 0, deg = 0;
      float sv = 0.f, fv = 0.f; /* fv: what a predecessor takes per path */
      if (have) {
        v = order[k];
        start = __ldg(&a.trow[v]);
        deg = l > 0 ? __ldg(&a.trow[v + 1]) - start : 0;
        sv = sig[v];
        fv = (WGM_BC_SCALE + sv) / rho[v];
      }
      wgm_bc_edges<EVEN ? 1 : WGM_BC_K>(a.tcol, start, deg, fv, tab, [&](bool valid, int w, float fo) {
        if (valid && dist[w] == l - 1) atomicAdd(&sig[w], rho[w] * fo);
      });
      if (have && v != src && sv != 0.f) atomicAdd(&bc64[v], (double)(sv / WGM_BC_SCALE));
    }
    __syncthreads();
  }
}

#endif
