// Cell graph and reverse Cuthill-McKee renumbering on the GPU.
//
// The reference relabels cells with ReverseCuthillMcKee (aquaflux/mesh/reorder.py:147-159):
// scipy.sparse.csgraph.reverse_cuthill_mckee(symmetric_mode=True) on the cell adjacency of the
// interior faces (cell_adjacency_coo, aquaflux/mesh/graph.py:29-56, coalesced to a sorted CSR).
// The permutation must be bit-identical, so this restates scipy's published algorithm exactly:
//   * seeds are taken in the order of numpy's argsort of the node degrees (the caller passes that
//     order, computed by the same numpy call on the host), skipping placed nodes -- one
//     breadth-first sweep per connected component;
//   * a sweep processes the current level's nodes in their placement order; each appends its
//     not-yet-placed neighbours, then sorts just those by degree with a stable insertion sort
//     (neighbours are visited in ascending index order, so the key is (degree, index));
//   * the Cuthill-McKee order is reversed at the end.
// A node adjacent to several nodes of a level is appended by the first of them in placement
// order.  Level-parallel form: every level's parents claim their unplaced neighbours with an
// atomicMin of the parent's position (placed nodes hold -1, below any position, so they are never
// claimed), each parent then collects the neighbours it won, sorts them, and writes them at its
// exclusive-scan offset -- exactly the sequential order.
//
// The levels are a chain: 382 of them for the 128^3 channel, a few thousand parents each, a dozen
// dependent memory reads.  Five launches and a host round trip a level made that 22 ms; k_rcm_sweep
// runs every level in one thread-block cluster (16 x 1024 threads, a parent a thread), whose
// hardware barrier costs a fraction of a launch and whose blocks pass the scan's totals through
// each other's shared memory: 4.9 ms.  It is bound by the scattered 4-byte accesses of the
// cluster's SMs (8 blocks reading each neighbour list and mark twice: 9.2 ms), hence 16 blocks and
// the neighbours kept between passes.
#include <algorithm>
#include <climits>
#include <vector>

#include "internal.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kMaxDegree = 64;  // per-node neighbour bound of the parent-local sort

__global__ void k_fill_int(long n, int* a, int v) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

// cnt[c + 1] += 1 for both cells of every interior pair (pairs outside [0, n) are skipped and
// flagged)
__global__ void k_graph_count(long np, int n, const int* own, const int* nb, int* cnt, int* bad) {
  long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const int a = own[p], b = nb[p];
  if (a < 0 || a >= n || b < 0 || b >= n || a == b) {
    atomicExch(bad, 1);
    return;
  }
  atomicAdd(&cnt[a + 1], 1);
  atomicAdd(&cnt[b + 1], 1);
}

// In-place inclusive scan of a[0..n): tiles of kTile entries by a block each, their totals by one
// block (k_scan_totals), the totals added (k_scan_add).  One block over all of it read 2M entries a
// chunk per thread, uncoalesced: 3.4 ms.
constexpr int kTile = 4096;
__device__ __forceinline__ int warp_scan(int x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) >= o) x += y;
  }
  return x;
}
// Inclusive scan over a block of 1024 threads; every thread gets the block's total.
__device__ __forceinline__ int block_scan(int x, int* total) {
  __shared__ int warps[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int incl = warp_scan(x);
  __syncthreads();  // (the shared totals of an earlier call have been read)
  if (lane == 31) warps[w] = incl;
  __syncthreads();
  if (w == 0) warps[lane] = warp_scan(warps[lane]);
  __syncthreads();
  *total = warps[31];
  return incl + (w > 0 ? warps[w - 1] : 0);
}
__global__ void __launch_bounds__(1024) k_scan_tiles(long n, int* a, int* totals) {
  const long i0 = (long)blockIdx.x * kTile + 4L * threadIdx.x;
  int v[4], s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s += i0 + k < n ? a[i0 + k] : 0;
    v[k] = s;
  }
  int total;
  const int off = block_scan(s, &total) - s;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (i0 + k < n) a[i0 + k] = v[k] + off;
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) k_scan_totals(int nt, int* totals) {
  int base = 0;
  for (int t0 = 0; t0 < nt; t0 += 1024) {
    const int t = t0 + threadIdx.x;
    int total;
    const int x = block_scan(t < nt ? totals[t] : 0, &total);
    if (t < nt) totals[t] = base + x;
    base += total;
  }
}
__global__ void __launch_bounds__(1024) k_scan_add(long n, int* a, const int* totals) {
  if (blockIdx.x == 0) return;
  const int off = totals[blockIdx.x - 1];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const long i = (long)blockIdx.x * kTile + 1024L * k + threadIdx.x;
    if (i < n) a[i] += off;
  }
}
// `totals` holds (n + kTile - 1) / kTile ints.
void scan(long n, int* a, int* totals, cudaStream_t s) {
  const int nt = (int)((n + kTile - 1) / kTile);
  k_scan_tiles<<<nt, 1024, 0, s>>>(n, a, totals);
  if (nt == 1) return;
  k_scan_totals<<<1, 1024, 0, s>>>(nt, totals);
  k_scan_add<<<nt, 1024, 0, s>>>(n, a, totals);
}

__global__ void k_graph_fill(long np, const int* own, const int* nb, const int* ptr0, int* cursor,
                             int* tmp) {
  long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const int a = own[p], b = nb[p];
  tmp[ptr0[a] + atomicAdd(&cursor[a], 1)] = b;
  tmp[ptr0[b] + atomicAdd(&cursor[b], 1)] = a;
}

// Sort each row's neighbours ascending (insertion sort) and count the distinct ones.
__global__ void k_graph_sort(int n, const int* ptr0, int* tmp, int* ucnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int b = ptr0[i], e = ptr0[i + 1];
  for (int p = b + 1; p < e; ++p) {
    const int v = tmp[p];
    int q = p - 1;
    while (q >= b && tmp[q] > v) {
      tmp[q + 1] = tmp[q];
      --q;
    }
    tmp[q + 1] = v;
  }
  int u = 0;
  for (int p = b; p < e; ++p) u += (p == b || tmp[p] != tmp[p - 1]) ? 1 : 0;
  ucnt[i + 1] = u;
}

__global__ void k_graph_compact(int n, const int* ptr0, const int* tmp, const int* ptr, int* idx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int w = ptr[i];
  for (int p = ptr0[i]; p < ptr0[i + 1]; ++p)
    if (p == ptr0[i] || tmp[p] != tmp[p - 1]) idx[w++] = tmp[p];
}

// The least node whose degree is negative or above kMaxDegree.
__global__ void k_rcm_check(int n, const int* ptr, int* worst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int d = ptr[i + 1] - ptr[i];
  if (d < 0 || d > kMaxDegree) atomicMin(worst, i);
}

constexpr int kCluster = 16;  // largest cluster; 8 (the portable size) where it does not fit
constexpr int kKept = 6;      // neighbours of a parent kept in registers between a level's passes

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

// Cuthill-McKee sweeps from `placed` placed nodes on: from node `seed` alone, or (seeds given) from
// every unplaced node of seeds in turn until all are placed.  order and mark change under the
// other blocks' hands, so they are read past the L1 cache.  result: placed nodes and -1, or the
// position of a seed out of range; -1 and the level's size where a level would place more nodes
// than are left (a row lists a node twice), before anything of it is written.
__global__ void __launch_bounds__(1024)
    k_rcm_sweep(int n, const int* __restrict__ ptr, const int* __restrict__ idx, int seed,
                const long* __restrict__ seeds, int placed, int* order, int* mark, int* result) {
  __shared__ int totals[2][kCluster];  // the blocks' counts of a round, sent by each of them
  __shared__ int found;
  unsigned rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int nc = (int)gridDim.x;  // the blocks of the one cluster
  const int t = threadIdx.x, gid = (int)rank * 1024 + t;
  const int NT = nc * 1024;
  int parity = 0, bad = 0;
  long next = 0;
  // value v of every block into all blocks' totals[parity]
  auto share = [&](int v) {
    if (t < nc) {
      const unsigned a = (unsigned)__cvta_generic_to_shared(&totals[parity][rank]);
      unsigned to;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(a), "r"(t));
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to), "r"(v) : "memory");
    }
    cluster_sync();
  };
  cluster_sync();
  while (placed < n) {
    if (seeds) {  // the first unplaced seed, NT at a time
      int at = INT_MAX;
      while (next < n) {
        if (t == 0) found = INT_MAX;
        __syncthreads();
        if (next + gid < n) {
          const long v = seeds[next + gid];
          if (v < 0 || v >= n || __ldcg(mark + v) != -1) atomicMin(&found, gid);
        }
        __syncthreads();
        share(found);
        at = INT_MAX;
        for (int k = 0; k < nc; ++k) at = min(at, totals[parity][k]);
        parity ^= 1;
        if (at != INT_MAX) break;
        next += NT;
      }
      if (at == INT_MAX) break;  // exhausted: not a permutation
      next += at;
      const long v = seeds[next];
      if (v < 0 || v >= n) {
        bad = 1;
        seed = (int)next;
        break;
      }
      seed = (int)v;
    }
    if (gid == 0) {
      order[placed] = seed;
      mark[seed] = -1;
    }
    cluster_sync();
    int ls = placed, le = placed + 1;
    while (ls < le) {
      // claim the unplaced neighbours; the last round's are kept in registers
      int b = 0, e = 0, nb[kKept];
      for (int p = ls + gid; p < le; p += NT) {
        const int i = __ldcg(order + p);
        b = ptr[i];
        e = ptr[i + 1];
#pragma unroll
        for (int k = 0; k < kKept; ++k)
          if (b + k < e) nb[k] = idx[b + k];
#pragma unroll
        for (int k = 0; k < kKept; ++k)
          if (b + k < e) atomicMin(&mark[nb[k]], p);
        for (int q = b + kKept; q < e; ++q) atomicMin(&mark[idx[q]], p);
      }
      cluster_sync();
      int base = le;
      for (int r0 = ls; r0 < le; r0 += NT) {
        const int p = r0 + gid;
        unsigned long long won = 0;  // bit k: neighbour b + k (kMaxDegree of them at most)
        if (p < le) {
          if (le - ls > NT) {  // several rounds: read again
            const int i = __ldcg(order + p);
            b = ptr[i];
            e = ptr[i + 1];
#pragma unroll
            for (int k = 0; k < kKept; ++k)
              if (b + k < e) nb[k] = idx[b + k];
          }
          int mk[kKept];
#pragma unroll
          for (int k = 0; k < kKept; ++k)
            if (b + k < e) mk[k] = __ldcg(mark + nb[k]);
#pragma unroll
          for (int k = 0; k < kKept; ++k)
            if (b + k < e && mk[k] == p) won |= 1ull << k;
          for (int q = b + kKept; q < e; ++q)
            if (__ldcg(mark + idx[q]) == p) won |= 1ull << (q - b);
        }
        const int c = __popcll(won);
        int total;
        int at = block_scan(c, &total) - c;
        share(total);
        int sum = 0;
        for (int k = 0; k < nc; ++k) {
          if (k < (int)rank) at += totals[parity][k];
          sum += totals[parity][k];
        }
        parity ^= 1;
        if (base + sum > n) {  // (the same in every block)
          bad = 2;
          seed = base + sum - le;
          break;
        }
        if (c > 0) {  // the neighbours won, by (degree, index), and mark them placed
          int kid[kMaxDegree], kdeg[kMaxDegree];
          int m = 0;
          for (; won; won &= won - 1) {
            const int j = idx[b + __ffsll((long long)won) - 1];
            const int d = ptr[j + 1] - ptr[j];
            int k = m++;
            while (k > 0 && d < kdeg[k - 1]) {  // stable: equal degrees keep ascending index order
              kid[k] = kid[k - 1];
              kdeg[k] = kdeg[k - 1];
              --k;
            }
            kid[k] = j;
            kdeg[k] = d;
          }
          for (int k = 0; k < m; ++k) {
            order[base + at + k] = kid[k];
            mark[kid[k]] = -1;
          }
        }
        base += sum;
      }
      cluster_sync();
      if (bad) break;
      ls = le;
      le = base;
    }
    if (bad) break;
    placed = le;
    if (!seeds) break;
  }
  if (gid == 0) {
    result[0] = bad == 2 ? -1 : placed;
    result[1] = bad ? seed : -1;
  }
  cluster_sync();  // no block leaves while another may still write to its shared memory
}

__global__ void k_rcm_perm(int n, const int* order, int* perm) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) perm[order[k]] = n - 1 - k;
}

int blocks_of(long n) { return (int)std::max(1L, (n + kThreads - 1) / kThreads); }

}  // namespace

extern "C" int fv_cell_graph(int n, long n_pairs, const int* owner, const int* neighbour,
                             int* indptr, int* indices, int* work, void* stream) {
  if (n <= 0 || n_pairs < 0 || !indptr || !work || (n_pairs > 0 && (!owner || !neighbour || !indices))) {
    fv_set_error("fv_cell_graph: bad arguments");
    return FV_ERR_ARG;
  }
  if (2 * n_pairs > INT_MAX) {
    fv_set_error("fv_cell_graph: too many pairs for int32 offsets");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  int* ptr0 = work;                 // n + 1
  int* cursor = ptr0 + n + 1;       // n
  int* bad = cursor + n;            // 1
  int* tmp = bad + 1;               // 2 n_pairs
  k_fill_int<<<blocks_of(2L * n + 2), kThreads, 0, s>>>(2L * n + 2, ptr0, 0);
  k_fill_int<<<blocks_of(n + 1), kThreads, 0, s>>>(n + 1, indptr, 0);
  if (n_pairs > 0) {
    k_graph_count<<<blocks_of(n_pairs), kThreads, 0, s>>>(n_pairs, n, owner, neighbour, ptr0, bad);
    int h_bad = 0;
    FV_CUDA_TRY(cudaMemcpyAsync(&h_bad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    FV_CUDA_TRY(cudaStreamSynchronize(s));
    if (h_bad) {
      fv_set_error("fv_cell_graph: a cell pair is out of range or joins a cell to itself");
      return FV_ERR_ARG;
    }
    scan(n + 1, ptr0, indptr + 1, s);  // (indptr's entries are written by k_graph_sort)
    k_graph_fill<<<blocks_of(n_pairs), kThreads, 0, s>>>(n_pairs, owner, neighbour, ptr0, cursor,
                                                         tmp);
    k_graph_sort<<<blocks_of(n), kThreads, 0, s>>>(n, ptr0, tmp, indptr);
    scan(n + 1, indptr, cursor, s);
    k_graph_compact<<<blocks_of(n), kThreads, 0, s>>>(n, ptr0, tmp, indptr, indices);
  }
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

extern "C" int fv_rcm_permutation(int n, const int* indptr, const int* indices,
                                  const long* seed_order, int* perm, int* work, void* stream) {
  if (n <= 0 || !indptr || !seed_order || !perm || !work) {
    fv_set_error("fv_rcm_permutation: bad arguments");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  int* order = work;        // n
  int* mark = order + n;    // n: -1 placed, INT_MAX unclaimed, else the claiming position
  int* result = mark + n;   // 2 (of n + 1)
  int h[2];
  k_fill_int<<<1, kThreads, 0, s>>>(1, result, INT_MAX);
  k_rcm_check<<<blocks_of(n), kThreads, 0, s>>>(n, indptr, result);
  FV_CUDA_TRY(cudaMemcpyAsync(h, result, sizeof(int), cudaMemcpyDeviceToHost, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  if (h[0] < n) {
    int be[2];
    const int i = h[0];
    FV_CUDA_TRY(cudaMemcpy(be, indptr + i, sizeof(be), cudaMemcpyDeviceToHost));
    fv_set_error("fv_rcm_permutation: node %d has degree %d (at most %d)", i, be[1] - be[0],
                 kMaxDegree);
    return FV_ERR_ARG;
  }
  auto bad_seed = [](long seed) {
    fv_set_error("fv_rcm_permutation: seed %ld out of range", seed);
    return FV_ERR_ARG;
  };
  if (seed_order[0] < 0 || seed_order[0] >= n) return bad_seed(seed_order[0]);
  long* seeds = nullptr;  // device copy of the seed order, for more than one component
  int blocks = kCluster;
  auto sweep = [&](int placed) -> int {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = blocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int fits = 0;
    if (blocks > 8 && (cudaFuncSetAttribute(k_rcm_sweep,
                                            cudaFuncAttributeNonPortableClusterSizeAllowed,
                                            1) != cudaSuccess ||
                       cudaOccupancyMaxActiveClusters(&fits, k_rcm_sweep, &cfg) != cudaSuccess ||
                       fits < 1)) {
      cudaGetLastError();
      blocks = 8;
      cfg.gridDim = dim3(blocks);
      at.val.clusterDim.x = blocks;
    }
    FV_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_rcm_sweep, n, indptr, indices, (int)seed_order[0],
                                   (const long*)seeds, placed, order, mark, result));
    FV_CUDA_TRY(cudaMemcpyAsync(h, result, sizeof(h), cudaMemcpyDeviceToHost, s));
    FV_CUDA_TRY(cudaStreamSynchronize(s));
    return FV_OK;
  };
  k_fill_int<<<blocks_of(n), kThreads, 0, s>>>(n, mark, INT_MAX);
  int rc = sweep(0);
  if (rc == FV_OK && h[0] >= 0 && h[0] < n) {  // the other components, from the seed order
    rc = cudaMalloc(&seeds, sizeof(long) * (size_t)n) == cudaSuccess &&
                 cudaMemcpyAsync(seeds, seed_order, sizeof(long) * (size_t)n,
                                 cudaMemcpyHostToDevice, s) == cudaSuccess
             ? sweep(h[0])
             : FV_ERR_CUDA;
  }
  cudaFree(seeds);
  if (rc != FV_OK) return rc;
  if (h[0] < 0) {
    fv_set_error("fv_rcm_permutation: inconsistent level size %d", h[1]);
    return FV_ERR_ARG;
  }
  if (h[1] >= 0) return bad_seed(seed_order[h[1]]);
  if (h[0] < n) {
    fv_set_error("fv_rcm_permutation: seed order is not a permutation");
    return FV_ERR_ARG;
  }
  k_rcm_perm<<<blocks_of(n), kThreads, 0, s>>>(n, order, perm);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}
