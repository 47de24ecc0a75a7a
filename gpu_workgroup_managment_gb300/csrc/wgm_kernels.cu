/*
 * Standalone persistent kernels (one per app) and the barrier
 * microbenchmark, compiled for sm_103a.
 */
#include "wgm_kernels.cuh"

#include <algorithm>

#define WGM_PERSISTENT_PROLOGUE                                  \
  __shared__ wgm_cta c;                                          \
  __shared__ wgm_warp_smem sm;                                   \
  if (!wgm_discover(L, &c)) return;                              \
  if (L.handshake && !wgm_standalone_handshake(L, &c)) {         \
    wgm_standalone_exit(L);                                      \
    return;                                                      \
  }

/* The same for task loops that need no per-warp edge tables. */
#define WGM_PERSISTENT_PROLOGUE_TASKS                            \
  __shared__ wgm_cta c;                                          \
  if (!wgm_discover(L, &c)) return;                              \
  if (L.handshake && !wgm_standalone_handshake(L, &c)) {         \
    wgm_standalone_exit(L);                                      \
    return;                                                      \
  }

#define WGM_PERSISTENT_EPILOGUE \
  if (L.handshake) wgm_standalone_exit(L);

/* Run a phase function from its init phase with plain barriers between. */
#define WGM_DRIVE(PHASE_CALL)                                                        \
  wgm_drive(L, &c, wgm_step{0, 0}, wgm_plain_sync(),                                \
            [&](wgm_step cur, wgm_step *nxt) { return PHASE_CALL; })

template <bool SSSP>
__device__ __forceinline__ int wgm_lonestar_step(const wgm_launch &L, wgm_cta *c,
                                                 const wgm_lonestar_args &a, wgm_warp_smem *sm,
                                                 wgm_step cur, wgm_step *nxt) {
  return wgm_phase_lonestar<SSSP>(L, c, a, sm, cur.target, cur.round, &nxt->target,
                                  &nxt->round);
}

__global__ void __launch_bounds__(1024) wgm_k_bfs(wgm_launch L, wgm_lonestar_args a) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_lonestar_step<false>(L, &c, a, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

/* The same where in-edges are at hand (wgm_phase_bfs). */
__global__ void __launch_bounds__(1024) wgm_k_bfs_two_way(wgm_launch L, wgm_lonestar_args a,
                                                          wgm_bfs_up_args b) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_phase_bfs(L, &c, a, b, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

cudaError_t wgm_launch_bfs_two_way(const wgm_launch &L, const wgm_lonestar_args &a,
                                   const wgm_bfs_up_args &b, int grid, int block, cudaStream_t s) {
  wgm_k_bfs_two_way<<<grid, block, 0, s>>>(L, a, b);
  return cudaGetLastError();
}

/* In-edges on the device: counts, their exclusive prefix, then the places
 * taken (at).  Out-of-range columns have no place. */
__global__ void __launch_bounds__(256) wgm_k_in_count(int V, long long E, const int *col, int *deg) {
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < E; e += gridDim.x * 256LL) {
    const int u = col[e];
    if ((unsigned)u < (unsigned)V) atomicAdd(&deg[u], 1);
  }
}
/* Exclusive prefix of deg[] in blocks of 8192: the blocks' sums, their
 * prefix, then every place.  deg is zeroed for the places taken; vertices of
 * more than WGM_BFS_UP_SCAN in-edges are listed (wide[0]: how many, then
 * they). */
#define WGM_IN_BLOCK 8192
__device__ __forceinline__ int wgm_cta_scan(int x, int *warp_sum, int *total) {
  const int lane = wgm_lane(), warp = threadIdx.x >> 5;
  const int incl = wgm_warp_incl_scan(x);
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  const int w = wgm_warp_incl_scan(lane < (int)(blockDim.x >> 5) ? warp_sum[lane] : 0);
  const int before = __shfl_sync(WGM_FULL, w, max(warp - 1, 0));
  *total = __shfl_sync(WGM_FULL, w, 31);
  __syncthreads();
  return incl - x + (warp ? before : 0);
}
__global__ void __launch_bounds__(1024) wgm_k_in_sums(int V, const int *deg, int *sums) {
  __shared__ int warp_sum[32];
  int x = 0, total;
  for (int q = 0; q < 8; q++) {
    const long long i = (long long)blockIdx.x * WGM_IN_BLOCK + q * 1024 + threadIdx.x;
    x += i < V ? deg[i] : 0;
  }
  wgm_cta_scan(x, warp_sum, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) wgm_k_in_bases(int n, int *sums, int *last) {
  __shared__ int warp_sum[32];
  int base = 0;
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + threadIdx.x, x = i < n ? sums[i] : 0;
    int total;
    const int p = wgm_cta_scan(x, warp_sum, &total);
    if (i < n) sums[i] = base + p;
    base += total;
  }
  if (threadIdx.x == 0) *last = base;
}
__global__ void __launch_bounds__(1024) wgm_k_in_places(int V, int *deg, const int *bases,
                                                        int *trow, int *wide) {
  __shared__ int warp_sum[32];
  int base = bases[blockIdx.x];
  for (int q = 0; q < 8; q++) {
    const long long i = (long long)blockIdx.x * WGM_IN_BLOCK + q * 1024 + threadIdx.x;
    const int x = i < V ? deg[i] : 0;
    int total;
    const int p = wgm_cta_scan(x, warp_sum, &total);
    if (i < V) {
      trow[i] = base + p;
      deg[i] = 0;
      if (x > WGM_BFS_UP_SCAN) wide[1 + atomicAdd(wide, 1)] = (int)i;
    }
    base += total;
  }
}
__global__ void __launch_bounds__(256) wgm_k_in_fill(int V, const int *row, const int *col,
                                                     const int *trow, int *at, int *tcol) {
  const int nw = gridDim.x * (blockDim.x >> 5), lane = wgm_lane();
  for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < (V + 31) / 32; k += nw) {
    const int v = 32 * k + lane;
    const int s = v < V ? row[v] : 0, d = v < V ? max(row[v + 1] - s, 0) : 0;
    const int incl = wgm_warp_incl_scan(d), total = __shfl_sync(WGM_FULL, incl, 31);
    const int off = incl - d;
    for (int w = 0; w < total; w += 32) {
      const int sl = w + lane, own = wgm_owner_of(off, min(sl, total - 1));
      const int e = __shfl_sync(WGM_FULL, s - off, own) + sl;
      if (sl >= total) continue;
      const int u = col[e];
      if ((unsigned)u < (unsigned)V) tcol[trow[u] + atomicAdd(&at[u], 1)] = 32 * k + own;
    }
  }
}

/* trow [V+1], tcol [E], wide [E / WGM_BFS_UP_SCAN + 2], scratch [V] from the
 * out-edges' first E columns. */
cudaError_t wgm_launch_in_edges(int V, long long E, const int *row, const int *col, int *trow,
                                int *tcol, int *wide, int *scratch, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(scratch, 0, (size_t)V * 4, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(wide, 0, 4, s);
  if (e != cudaSuccess) return e;
  wgm_k_in_count<<<1216, 256, 0, s>>>(V, E, col, scratch);
  const int nb = (V + WGM_IN_BLOCK - 1) / WGM_IN_BLOCK;
  int *sums = tcol; /* filled last */
  wgm_k_in_sums<<<nb, 1024, 0, s>>>(V, scratch, sums);
  wgm_k_in_bases<<<1, 1024, 0, s>>>(nb, sums, trow + V);
  wgm_k_in_places<<<nb, 1024, 0, s>>>(V, scratch, sums, trow, wide);
  wgm_k_in_fill<<<1216, 256, 0, s>>>(V, row, col, trow, scratch, tcol);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(1024) wgm_k_sssp(wgm_launch L, wgm_lonestar_args a) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_lonestar_step<true>(L, &c, a, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

__global__ void __launch_bounds__(1024) wgm_k_color(wgm_launch L, wgm_color_args a) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_phase_color(L, &c, a, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

/* 48 registers (eight spilled words): five 256-thread CTAs per SM.  RMAT-20: 0.228 ms,
 * against 0.235 with 64, 0.246 with 40 and 0.292 with 32 (more CTAs only
 * make the barrier dearer). */
__global__ void __maxnreg__(48) wgm_k_mis(wgm_launch L, wgm_mis_args a) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_phase_mis(L, &c, a, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

/* Pannotia colour in priority blocks (wgm_cb_look, wgm_cb_finish).  Dynamic
 * shared memory: wgm_color_blocks_smem_bytes (group 0 uses it). */
__global__ void __launch_bounds__(1024) wgm_k_color_blocks(wgm_launch L, wgm_color_args a,
                                                           wgm_color_blocks_args q) {
  WGM_PERSISTENT_PROLOGUE
  const wgm_split s(&c);
  int mx = 0;
  bool ok = true;
  for (int h = s.tid; h < a.hubs.H; h += s.nth) q.hub_max[h] = 0;
  if (c.id == 0 && threadIdx.x < 3)
    for (int k = 0; k < 3; k++) q.cnt[threadIdx.x * WGM_LINE + k] = 0;
  /* group 0 finishes blocks, the others look; a single group does both */
  const bool both = c.ngroups == 1;
  const int nw = blockDim.x >> 5;
  const int gw = both ? s.gw : s.gw - nw, NW = both ? nw : s.NW - nw;
  bool live = true;
  for (int b = 0; b <= q.NB; b++) {
    const bool look = b < q.NB && (both || c.id > 0);
    wgm_cb_first F;
    if (look) F = wgm_cb_prefetch(a, q, b, gw, NW);
    live = wgm_barrier(L, &c);
    if (!live) break;
    if (b > 0 && c.id == 0) {
      const int m = wgm_cb_finish(a.V, q.B, b - 1, q.colour, q.list, q.cnt, q.blk_hub, q.hub_rank,
                                  q.hub_max);
      if (m < 0 && threadIdx.x == 0) wgm_fail(L, WGM_DEV_BAD_INPUT, WGM_SITE_QUEUE, b - 1);
      mx = max(mx, m);
    }
    if (look) ok &= wgm_cb_look(a, q, b, gw, NW, F, &sm);
  }
  /* the largest colour is the reference's round count */
  if (c.id == 0) {
    mx = __reduce_max_sync(WGM_FULL, mx);
    if (s.lane == 0) atomicMax(&q.cnt[2], mx);
  }
  if (!__all_sync(WGM_FULL, ok) && s.lane == 0) wgm_fail(L, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, 0);
  if (live && wgm_barrier(L, &c)) {
    for (int k = s.tid; k < a.V; k += s.nth) a.color[__ldg(&q.ord[k]).x] = __ldcg(&q.colour[k]);
    if (c.id == 0 && threadIdx.x == 0 && a.rounds_out) *a.rounds_out = __ldcg(&q.cnt[2]);
  }
  WGM_PERSISTENT_EPILOGUE
}

size_t wgm_color_blocks_smem_bytes(int B) { return (2 * (size_t)B + 4) * 4; }

/* CTAs per SM of a launch with blocks of B vertices. */
cudaError_t wgm_color_blocks_per_sm(int block, int B, int *per_sm) {
  /* the limit is the kernel's, whoever launches it next: always the most */
  cudaError_t e = cudaFuncSetAttribute(wgm_k_color_blocks,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)wgm_color_blocks_smem_bytes(WGM_CB_MAX_B));
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, wgm_k_color_blocks, block,
                                                       wgm_color_blocks_smem_bytes(B));
}

cudaError_t wgm_launch_color_blocks(const wgm_launch &L, const wgm_color_args &a,
                                    const wgm_color_blocks_args &q, int grid, int block,
                                    cudaStream_t s) {
  wgm_k_color_blocks<<<grid, block, wgm_color_blocks_smem_bytes(q.B), s>>>(L, a, q);
  return cudaGetLastError();
}

/* Layout of the priority blocks: the rank order's vertex records, the
 * columns as ranks, how many late (cnt[2b]) and inner edges (cnt[2b+1])
 * each block would list, and the edges by the smaller degree of their ends
 * (hist, by wgm_degree_bucket). */
__global__ void __launch_bounds__(256) wgm_k_color_order(int V, const int *row, const int *order,
                                                         const int *hub_of, int4 *ord, int *rank) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < V; k += gridDim.x * blockDim.x) {
    const int v = order[k], s = row[v];
    ord[k] = make_int4(v, s, row[v + 1] - s, hub_of[k]);
    rank[v] = k;
  }
}
__global__ void __launch_bounds__(256) wgm_k_color_rank(int E, const int *col, const int *rank,
                                                        int *crank) {
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < E; e += gridDim.x * 256LL)
    crank[e] = __ldg(&rank[col[e]]);
}
__global__ void __launch_bounds__(256) wgm_k_color_count(int V, const int *crank, const int4 *ord,
                                                         int B, int *cnt,
                                                         unsigned long long *hist) {
  const int nw = gridDim.x * (blockDim.x >> 5), lane = wgm_lane();
  __shared__ int h[WGM_DEGREE_BUCKETS];
  if (threadIdx.x < WGM_DEGREE_BUCKETS) h[threadIdx.x] = 0;
  __syncthreads();
  for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < V; k += nw) {
    const int4 o = ord[k];
    const int b = k / B, lo = b * B;
    int n = 0, inner = 0;
    for (int x = lane; x < o.z && o.z != 1; x += 32) {
      const int r = crank[o.y + x];
      n += r < lo && r >= lo - B;
      inner += r < k && r >= lo;
      atomicAdd(&h[wgm_degree_bucket(min(o.z, __ldg(&ord[r].z)))], 1);
    }
    n = __reduce_add_sync(WGM_FULL, n);
    inner = __reduce_add_sync(WGM_FULL, inner);
    if (lane == 0 && n) atomicAdd(&cnt[2 * b], n);
    if (lane == 0 && inner) atomicAdd(&cnt[2 * b + 1], inner);
  }
  __syncthreads();
  if (threadIdx.x < WGM_DEGREE_BUCKETS && h[threadIdx.x])
    atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

cudaError_t wgm_launch_color_order(int V, int E, const int *row, const int *col, const int *order,
                                   const int *hub_of, int4 *ord, int *rank, int *crank,
                                   cudaStream_t s) {
  wgm_k_color_order<<<std::min((V + 255) / 256, 1216), 256, 0, s>>>(V, row, order, hub_of, ord,
                                                                    rank);
  wgm_k_color_rank<<<1216, 256, 0, s>>>(E, col, rank, crank);
  return cudaGetLastError();
}
cudaError_t wgm_launch_color_count(int V, const int *crank, const int4 *ord, int B, int *cnt,
                                   unsigned long long *hist, cudaStream_t s) {
  wgm_k_color_count<<<std::min((V + 7) / 8, 1216), 256, 0, s>>>(V, crank, ord, B, cnt, hist);
  return cudaGetLastError();
}

/* Pannotia colour without rounds (wgm_color_async_run): the counts of
 * wgm_phase_color between plain barriers, then the release loop, then one
 * barrier before the round count (the largest colour) is written.  Dynamic
 * shared memory: one release stack per warp. */
__global__ void __launch_bounds__(1024) wgm_k_color_async(wgm_launch L, wgm_color_args a,
                                                          wgm_color_async_args q) {
  WGM_PERSISTENT_PROLOGUE
  extern __shared__ wgm_ca_stack wgm_ca_stacks[];
  wgm_ca_stack *st = &wgm_ca_stacks[threadIdx.x >> 5];
  bool ok = true;
  wgm_color_async_init(&c, a, q);
  if (wgm_barrier(L, &c)) {
    wgm_step nx;
    wgm_phase_color(L, &c, a, &sm, wgm_step{3, 0}, &nx); /* larger out-neighbours */
    if (wgm_barrier(L, &c)) {
      ok = wgm_color_async_seed(&c, a, q, st);
      if (wgm_barrier(L, &c)) {
        ok &= wgm_color_async_run(L, a, q, st);
        if (!ok && threadIdx.x % 32 == 0) wgm_fail(L, WGM_DEV_OVERFLOW, WGM_SITE_QUEUE, 0);
        if (wgm_barrier(L, &c) && c.id == 0 && threadIdx.x == 0 && a.rounds_out)
          *a.rounds_out = __ldcg(&q.ctl[4 * WGM_LINE]);
      }
    }
  }
  WGM_PERSISTENT_EPILOGUE
}

size_t wgm_color_async_smem(int block) { return (size_t)(block / 32) * sizeof(wgm_ca_stack); }

cudaError_t wgm_color_async_per_sm(int block, int *per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, wgm_k_color_async, block,
                                                       wgm_color_async_smem(block));
}

cudaError_t wgm_launch_color_async(const wgm_launch &L, const wgm_color_args &a,
                                   const wgm_color_async_args &q, int grid, int block,
                                   cudaStream_t s) {
  wgm_k_color_async<<<grid, block, wgm_color_async_smem(block), s>>>(L, a, q);
  return cudaGetLastError();
}

/* Lonestar BFS on one CTA (wgm_bfs_cta): a plain one-CTA launch, no
 * discovery and no grid barrier.  Dynamic shared memory: the visited bits,
 * then the two frontier buffers of F vertices each. */
template <int W>
__global__ void __launch_bounds__(1024) wgm_k_bfs_cta(wgm_lonestar_args a, const int4 *ell,
                                                      int *spill, int spill_cap, int F,
                                                      int *status) {
  __shared__ int s_cnt[8];
  wgm_bfs_cta<W>(a, ell, spill, spill_cap, F, s_cnt);
  if (threadIdx.x == 0 && s_cnt[3] && status) *status = WGM_DEV_OVERFLOW;
}

/* The columns as W per vertex (wgm_bfs_cta): a column equal to the padding is
 * out of range and becomes another that is. */
template <int W>
__global__ void __launch_bounds__(256) wgm_k_bfs_ell(int V, const int *row, const int *col,
                                                     int *ell) {
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < (long long)V * W;
       i += gridDim.x * 256LL) {
    const int v = (int)(i / W), q = (int)(i % W), s = row[v];
    int u = WGM_BFS_PAD;
    if (q < row[v + 1] - s) {
      u = col[s + q];
      if (u == WGM_BFS_PAD) u = -1;
    }
    ell[i] = u;
  }
}

cudaError_t wgm_launch_bfs_ell(int W, int V, const int *row, const int *col, int *ell,
                               cudaStream_t s) {
  const int grid = (int)std::min<long long>(((long long)V * W + 255) / 256, 1216);
  if (W == 4)
    wgm_k_bfs_ell<4><<<grid, 256, 0, s>>>(V, row, col, ell);
  else
    wgm_k_bfs_ell<8><<<grid, 256, 0, s>>>(V, row, col, ell);
  return cudaGetLastError();
}

size_t wgm_bfs_cta_smem_bytes(int V, int F) {
  return (size_t)((V + 31) / 32) * 4 + (size_t)2 * F * 4;
}

cudaError_t wgm_launch_bfs_cta(const wgm_lonestar_args &a, int W, const int *ell, int *spill,
                               int spill_cap, int F, int *status, int block, cudaStream_t s) {
  auto *k = W == 4 ? wgm_k_bfs_cta<4> : W == 8 ? wgm_k_bfs_cta<8> : wgm_k_bfs_cta<0>;
  /* the limit is the kernel's, whoever launches it next: always the most */
  int dev = 0, most = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - 1024);
  if (e != cudaSuccess) return e;
  k<<<1, block, wgm_bfs_cta_smem_bytes(a.V, F), s>>>(a, reinterpret_cast<const int4 *>(ell), spill,
                                                     spill_cap, F, status);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(1024) wgm_k_psssp(wgm_launch L, wgm_psssp_args a) {
  WGM_PERSISTENT_PROLOGUE_TASKS
  WGM_DRIVE(wgm_phase_pannotia_sssp(L, &c, a, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

__global__ void __launch_bounds__(1024) wgm_k_pagerank(wgm_launch L, wgm_pr_args a) {
  WGM_PERSISTENT_PROLOGUE_TASKS
  WGM_DRIVE(wgm_phase_pagerank(L, &c, a, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

/* Dynamic shared memory that `per_sm` groups of `block` threads can each
 * have on an SM, in bytes (0: they do not fit with any). */
cudaError_t wgm_pagerank_smem(int block, int per_sm, int *bytes) {
  int dev = 0, sm_bytes = 0, most = 0, fit = 0;
  cudaFuncAttributes fa;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, wgm_k_pagerank);
  if (e != cudaSuccess) return e;
  most -= (int)fa.sharedSizeBytes;
  /* the limit is the kernel's, whoever launches it next: always the most */
  e = cudaFuncSetAttribute(wgm_k_pagerank, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e != cudaSuccess) return e;
  /* 1 KB of each group's share is the system's */
  int b = std::min(most, sm_bytes / per_sm - 1024 - (int)fa.sharedSizeBytes) & ~1023;
  if (b > 0) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, wgm_k_pagerank, block, b);
  *bytes = b > 0 && fit >= per_sm ? b : 0;
  return e;
}

/* Layout by rank: ranks, then columns and weights. */
__global__ void __launch_bounds__(256) wgm_k_rank_of(int V, const int *order, int *rank) {
  for (int k = blockIdx.x * 256 + threadIdx.x; k < V; k += gridDim.x * 256) rank[order[k]] = k;
}
__global__ void __launch_bounds__(256) wgm_k_rank_rows(wgm_rank_rows R, const int *row,
                                                       const int *col, const int *wt,
                                                       const int *rank, int *pcol, int *pwt,
                                                       int *wmin) {
  const int nw = gridDim.x * 8, lane = wgm_lane();
  int least = INT_MAX;
  /* parts of wide rows, then four rows at a time */
  const long long units = R.parts + (R.rows - R.wide + 3LL) / 4;
  for (long long unit = blockIdx.x * 8 + (threadIdx.x >> 5); unit < units; unit += nw) {
    int from = 0, to = 0, n = 0;
    if (unit < R.parts) {
      const int k = R.part_row[unit], off = (int)(unit - R.row_part[k]) * R.part_edges;
      if (lane == 0) {
        from = row[R.order[k]] + off;
        to = R.prow[k] + off;
        n = min(R.part_edges, R.prow[k + 1] - to);
      }
    } else {
      const long long k = R.wide + (unit - R.parts) * 4 + lane;
      if (lane < 4 && k < R.rows) {
        from = row[R.order[k]];
        to = R.prow[k];
        n = R.prow[k + 1] - to;
      }
    }
    const int incl = wgm_warp_incl_scan(n), total = __shfl_sync(WGM_FULL, incl, 31);
    const int off = incl - n;
    for (int w = 0; w < total; w += 128) {
      int c[4], x[4], at[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int sl = w + 32 * q + lane, own = wgm_owner_of(off, min(sl, total - 1));
        const int e = __shfl_sync(WGM_FULL, from - off, own) + sl;
        at[q] = __shfl_sync(WGM_FULL, to - off, own) + sl;
        c[q] = sl < total ? __ldcs(&col[e]) : -1;
        x[q] = wt && sl < total ? __ldcs(&wt[e]) : 0;
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (c[q] >= 0) {
          pcol[at[q]] = __ldg(&rank[c[q]]);
          if (wt) {
            pwt[at[q]] = x[q];
            /* a weight that can wrap a cost rules the test out, like a negative one */
            least = min(least, x[q] > INT_MAX - WGM_PANNOTIA_BIG ? -1 : x[q]);
          }
        }
    }
  }
  if (wt) {
    least = __reduce_min_sync(WGM_FULL, least);
    if (lane == 0) atomicMin(wmin, least);
  }
}
cudaError_t wgm_launch_rank_layout(int V, const wgm_rank_rows &R, const int *row, const int *col,
                                   const int *wt, int *rank, int *pcol, int *pwt, int *wmin,
                                   cudaStream_t s) {
  wgm_k_rank_of<<<std::min((V + 255) / 256, 1216), 256, 0, s>>>(V, R.order, rank);
  wgm_k_rank_rows<<<1216, 256, 0, s>>>(R, row, col, wt, rank, pcol, pwt, wmin);
  return cudaGetLastError();
}

/* os_freq (test_suite/os_freq/device/os_freq.cl:8-46): discovery, then
 * num_iterations x 10 barriers over every discovered CTA. */
__global__ void __launch_bounds__(1024) wgm_k_barrier_bench(wgm_launch L,
                                                            wgm_barrier_bench_args a) {
  __shared__ wgm_cta c;
  if (!wgm_discover(L, &c)) return;
  unsigned long long t0 = 0;
  for (int i = 0; i < a.iterations; i++) {
    for (int j = 0; j < 10; j++) {
      if (!wgm_barrier(L, &c)) return;
      if (i == 0 && j == 0) t0 = wgm_globaltimer();
    }
  }
  if (c.id == 0 && threadIdx.x == 0) {
    *a.t_first = t0;
    *a.t_last = wgm_globaltimer();
    *a.groups_out = c.ngroups;
  }
}

/* Standalone octree build (octree.cl:150-320 without a scheduler): init,
 * one barrier, then the task loop; nothing is offered to kill or fork. */
__global__ void __launch_bounds__(1024) wgm_k_octree(wgm_launch L, wgm_octree_args a) {
  WGM_PERSISTENT_PROLOGUE_TASKS
  wgm_octree_init(L, &c, a);
  if (wgm_barrier(L, &c)) wgm_octree_loop(L, &c, a, [](wgm_cta *) { return false; });
  WGM_PERSISTENT_EPILOGUE
}

__global__ void __launch_bounds__(1024) wgm_k_bc(wgm_launch L, wgm_bc_args a) {
  WGM_PERSISTENT_PROLOGUE
  WGM_DRIVE(wgm_phase_bc(L, &c, a, &sm, cur, nxt));
  WGM_PERSISTENT_EPILOGUE
}

/* Betweenness centrality, sources spread over CTAs (wgm_bc_cta_source):
 * a plain grid of resident CTAs, each with its own first source and the others
 * from a queue (one word after the sums), no discovery and no grid barrier. */
template <bool EVEN>
__global__ void __launch_bounds__(1024, 2) wgm_k_bc_cta(wgm_bc_args a, double *bc64, int few) {
  int *queue = reinterpret_cast<int *>(bc64 + a.V); /* sources, CTAs done */
  extern __shared__ int wgm_bc_dyn[];
  __shared__ int tab[32 * 32 * WGM_BC_K];
  __shared__ int s_cnt[9], s_src; /* wgm_bc_cta_source's counters */
  int *dist = wgm_bc_dyn;
  float *rho = reinterpret_cast<float *>(dist + a.V);
  float *sig = rho + a.V;
  int *order = reinterpret_cast<int *>(sig + a.V);
  int *ls = order + a.V;
  for (int src = blockIdx.x; src < a.num_sources;) {
    wgm_bc_cta_source<EVEN>(a, bc64, src, dist, rho, sig, order, ls, s_cnt, tab, few);
    if ((int)gridDim.x >= a.num_sources) break; /* a source each */
    if (threadIdx.x == 0) s_src = gridDim.x + atomicAdd(queue, 1);
    __syncthreads();
    src = s_src;
  }
  /* The last CTA to finish rounds the sums; the sources are all done then.  The
   * counter's own release and acquire order the sums: with a fence before and
   * one after it, a 15 x 8 grid took 53 us instead of 45. */
  __syncthreads();
  if (threadIdx.x == 0) {
    s_src = wgm_atom_add_acqrel_gpu(queue + 1, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_src) return;
  if (threadIdx.x == 0 && a.rounds_out) *a.rounds_out = a.num_sources;
  for (int i = threadIdx.x; i < a.V; i += blockDim.x) a.bc[i] = (float)__ldcg(&bc64[i]);
}

/* Standalone connect-four look-ahead (connect_four.cl:350-487 without a
 * scheduler). */
__global__ void __launch_bounds__(1024) wgm_k_c4(wgm_launch L, wgm_c4_args a) {
  WGM_PERSISTENT_PROLOGUE_TASKS
  wgm_c4_init(L, &c, a);
  if (wgm_barrier(L, &c)) wgm_c4_loop(L, &c, a, [](wgm_cta *) { return false; });
  WGM_PERSISTENT_EPILOGUE
}

const void *wgm_kernel_fn(int kid) {
  switch (kid) {
    case WGM_K_BFS: return (const void *)wgm_k_bfs;
    case WGM_K_SSSP: return (const void *)wgm_k_sssp;
    case WGM_K_COLOR: return (const void *)wgm_k_color;
    case WGM_K_BFS_TWO_WAY: return (const void *)wgm_k_bfs_two_way;
    case WGM_K_MIS: return (const void *)wgm_k_mis;
    case WGM_K_PSSSP: return (const void *)wgm_k_psssp;
    case WGM_K_PAGERANK: return (const void *)wgm_k_pagerank;
    case WGM_K_BARRIER_BENCH: return (const void *)wgm_k_barrier_bench;
    case WGM_K_OCTREE: return (const void *)wgm_k_octree;
    case WGM_K_C4: return (const void *)wgm_k_c4;
    case WGM_K_BC: return (const void *)wgm_k_bc;
    default: return nullptr;
  }
}

cudaError_t wgm_launch_lonestar(bool sssp, const wgm_launch &L, const wgm_lonestar_args &a,
                                int grid, int block, cudaStream_t s) {
  if (sssp)
    wgm_k_sssp<<<grid, block, 0, s>>>(L, a);
  else
    wgm_k_bfs<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_color(const wgm_launch &L, const wgm_color_args &a, int grid, int block,
                             cudaStream_t s) {
  wgm_k_color<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_mis(const wgm_launch &L, const wgm_mis_args &a, int grid, int block,
                           cudaStream_t s) {
  wgm_k_mis<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_psssp(const wgm_launch &L, const wgm_psssp_args &a, int grid, int block,
                             cudaStream_t s) {
  wgm_k_psssp<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_pagerank(const wgm_launch &L, const wgm_pr_args &a, int grid, int block,
                                cudaStream_t s) {
  wgm_k_pagerank<<<grid, block, (size_t)a.cached * 4, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_octree(const wgm_launch &L, const wgm_octree_args &a, int grid, int block,
                              cudaStream_t s) {
  wgm_k_octree<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_bc(const wgm_launch &L, const wgm_bc_args &a, int grid, int block,
                          cudaStream_t s) {
  wgm_k_bc<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_bc_cta(const wgm_bc_args &a, double *bc64, int edges, bool even, int block,
                              cudaStream_t s) {
  const size_t smem = (size_t)a.V * 20 + 16;
  const auto kernel = even ? wgm_k_bc_cta<true> : wgm_k_bc_cta<false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  int per_sm = 0, dev = 0, sms = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  e = cudaMemsetAsync(bc64, 0, (size_t)a.V * 8 + 8, s);
  if (e != cudaSuccess) return e;
  const int few = (int)min(32LL, max(1LL, 32LL * WGM_BC_K * a.V / max(edges, 1)));
  const int grid = max(1, min(per_sm * sms, a.num_sources));
  kernel<<<grid, block, smem, s>>>(a, bc64, few);
  return cudaGetLastError();
}
cudaError_t wgm_launch_c4(const wgm_launch &L, const wgm_c4_args &a, int grid, int block,
                          cudaStream_t s) {
  wgm_k_c4<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}
cudaError_t wgm_launch_barrier_bench(const wgm_launch &L, const wgm_barrier_bench_args &a,
                                     int grid, int block, cudaStream_t s) {
  wgm_k_barrier_bench<<<grid, block, 0, s>>>(L, a);
  return cudaGetLastError();
}

/* The barrier microbenchmark as a cluster grid: `clusters` clusters of
 * `csize` CTAs (WGM_BARRIER_CLUSTER needs whole clusters). */
cudaError_t wgm_barrier_bench_clusters(int csize, int block, int *clusters) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)csize, 1, 1);
  cfg.blockDim = dim3((unsigned)block, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(clusters, (void *)wgm_k_barrier_bench, &cfg);
}

cudaError_t wgm_launch_barrier_bench_cluster(const wgm_launch &L, const wgm_barrier_bench_args &a,
                                             int clusters, int csize, int block, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(clusters * csize), 1, 1);
  cfg.blockDim = dim3((unsigned)block, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, wgm_k_barrier_bench, L, a);
}
