// Block-sparse (BSR) SpMV, zero-fill ILU(0) and deterministic reductions.
//
// ILU(0) restates aquaflux/solve/_ilu0.pyx (factor :68-121, solve :124-147, solve_transpose
// :150-178) for b x b dense blocks.  On a block-dense pattern, scalar IKJ ILU(0) over the
// block-expanded (cell-major interleaved) ordering is the same elimination as:
//   for each lower block (i, j), ascending j:   L_ij = A_ij U_jj^-1   (U_jj: upper triangle of the
//                                                factored diagonal block of row j)
//                                                A_ik -= L_ij A_jk   for k > j stored in both rows
//   then the in-place unit-lower / upper LU of A_ii and A_ik = L_ii^-1 A_ik for k > i,
// which is what one thread does per block row here.  Rows run in level-set order (a row's level
// is one more than the deepest row it depends on), so the factor and the triangular sweeps
// reproduce the sequential algorithm's dependencies exactly.  With b = 1 this is the reference's
// scalar CSR ILU(0).
#include <algorithm>
#include <climits>
#include <cstdio>
#include <type_traits>
#include <memory>
#include <vector>

#include "internal.cuh"

void fv_set_error_index(long i);

namespace {

constexpr int kThreads = 256;

// B contiguous values p[0 .. B) into registers with the widest vector loads the block size allows
// (p is aligned to B values: every block row segment and every cell segment is).
template <int B, class V>
__device__ __forceinline__ void load_seg(const V* __restrict__ p, V (&o)[B]) {
  if constexpr (std::is_same<V, double>::value && B % 2 == 0) {
#pragma unroll
    for (int k = 0; k < B / 2; ++k) {
      const double2 t = reinterpret_cast<const double2*>(p)[k];
      o[2 * k] = t.x;
      o[2 * k + 1] = t.y;
    }
  } else if constexpr (std::is_same<V, float>::value && B % 4 == 0) {
#pragma unroll
    for (int k = 0; k < B / 4; ++k) {
      const float4 t = reinterpret_cast<const float4*>(p)[k];
      o[4 * k] = t.x;
      o[4 * k + 1] = t.y;
      o[4 * k + 2] = t.z;
      o[4 * k + 3] = t.w;
    }
  } else if constexpr (std::is_same<V, float>::value && B % 2 == 0) {
#pragma unroll
    for (int k = 0; k < B / 2; ++k) {
      const float2 t = reinterpret_cast<const float2*>(p)[k];
      o[2 * k] = t.x;
      o[2 * k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < B; ++k) o[k] = p[k];
  }
}

// a * b + c with one rounding.
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Calls fn(std::integral_constant<int, B>) for the runtime block size b in 2 .. 8.
template <class Fn>
void with_block_size(int b, Fn&& fn) {
  switch (b) {
    case 2: fn(std::integral_constant<int, 2>{}); break;
    case 3: fn(std::integral_constant<int, 3>{}); break;
    case 4: fn(std::integral_constant<int, 4>{}); break;
    case 5: fn(std::integral_constant<int, 5>{}); break;
    case 6: fn(std::integral_constant<int, 6>{}); break;
    case 7: fn(std::integral_constant<int, 7>{}); break;
    default: fn(std::integral_constant<int, 8>{}); break;
  }
}


// ------------------------------------------------------------------------------ BSR SpMV
template <class V>
__global__ void k_bsr_spmv(int nbr, int b, const int* __restrict__ ptr, const int* __restrict__ idx,
                           const V* __restrict__ val, const V* __restrict__ x,
                           const V* __restrict__ rhs, V* __restrict__ y) {
  // one thread per scalar row: row r = (block row i, component a)
  long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (long)nbr * b) return;
  int i = (int)(r / b), a = (int)(r % b);
  V acc = 0;
  const long bb = (long)b * b;
  for (int q = ptr[i]; q < ptr[i + 1]; ++q) {
    const V* blk = val + (long)q * bb + (long)a * b;
    const V* xs = x + (long)idx[q] * b;
    for (int c = 0; c < b; ++c) acc += blk[c] * xs[c];
  }
  y[r] = rhs ? rhs[r] - acc : acc;
}

// The same product with a compile-time block size and vector loads of each row segment (every
// block row segment and x segment starts at a multiple of B values from 16-byte aligned bases).
// RES: y = rhs - A x, the product rounded before the difference, as two passes give it.
template <class V, int B, bool RES>
__global__ void k_bsr_spmv_b(int nbr, const int* __restrict__ ptr, const int* __restrict__ idx,
                             const V* __restrict__ val, const V* __restrict__ x,
                             const V* __restrict__ rhs, V* __restrict__ y) {
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (long)nbr * B) return;
  const int i = (int)(r / B), a = (int)(r % B);
  constexpr long BB = (long)B * B;
  V acc = 0;
  for (int q = ptr[i]; q < ptr[i + 1]; ++q) {
    V m[B], xs[B];
    load_seg<B>(val + (long)q * BB + (long)a * B, m);
    load_seg<B>(x + (long)idx[q] * B, xs);
#pragma unroll
    for (int c = 0; c < B; ++c) acc += m[c] * xs[c];
  }
  y[r] = RES ? rhs[r] - acc : acc;
}

// Transposed product through the precomputed transpose map: for block row j of A^T, gather
// blocks (i, j) of A (tptr/tidx list rows i, tblk the block index in A).
template <class V>
__global__ void k_bsr_spmv_t(int nbc, int b, const int* __restrict__ tptr, const int* __restrict__ tidx,
                             const int* __restrict__ tblk, const V* __restrict__ val,
                             const V* __restrict__ x, V* __restrict__ y) {
  long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (long)nbc * b) return;
  int j = (int)(r / b), a = (int)(r % b);
  V acc = 0;
  const long bb = (long)b * b;
  for (int q = tptr[j]; q < tptr[j + 1]; ++q) {
    const V* blk = val + (long)tblk[q] * bb;
    const V* xs = x + (long)tidx[q] * b;
    for (int c = 0; c < b; ++c) acc += blk[(long)c * b + a] * xs[c];
  }
  y[r] = acc;
}

// The same transposed product with a compile-time block size: the same products accumulated in
// the same order (bitwise the runtime-size kernel's result), the loops unrolled.
template <class V, int B>
__global__ void k_bsr_spmv_tb(int nbc, const int* __restrict__ tptr, const int* __restrict__ tidx,
                              const int* __restrict__ tblk, const V* __restrict__ val,
                              const V* __restrict__ x, V* __restrict__ y) {
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (long)nbc * B) return;
  const int j = (int)(r / B), a = (int)(r % B);
  constexpr long BB = (long)B * B;
  V acc = 0;
  for (int q = tptr[j]; q < tptr[j + 1]; ++q) {
    const V* blk = val + (long)tblk[q] * BB + a;
    V xs[B];
    load_seg<B>(x + (long)tidx[q] * B, xs);
#pragma unroll
    for (int c = 0; c < B; ++c) acc += blk[(long)c * B] * xs[c];
  }
  y[r] = acc;
}

// y = A^T x through a device transpose map, the compile-time-size kernel for b in 2 .. 8 (x
// 16-byte aligned: its segments are read with vector loads).
template <class V>
void launch_spmv_t(int n, int b, const int* tp, const int* ti, const int* tb, const V* values,
                   const V* x, V* y, cudaStream_t s) {
  const long rows = (long)n * b;
  if (b >= 2 && b <= 8 && (uintptr_t)x % 16 == 0)
    with_block_size(b, [&](auto B) {
      k_bsr_spmv_tb<V, B()><<<fv_blocks(rows, kThreads), kThreads, 0, s>>>(n, tp, ti, tb, values,
                                                                           x, y);
    });
  else
    k_bsr_spmv_t<V><<<fv_blocks(rows, kThreads), kThreads, 0, s>>>(n, b, tp, ti, tb, values, x, y);
}

// tval[q] = val[tblk[q]]^T: the blocks of A in the order of A^T's pattern, each transposed, so
// that row a of block q of A^T is contiguous (the transposed sweeps and products read it with
// the forward kernels' vector loads).
template <class V>
__global__ void k_transpose_blocks(long nnzb, int b, const int* __restrict__ tblk,
                                   const V* __restrict__ val, V* __restrict__ tval) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long bb = (long)b * b;
  if (t >= nnzb * bb) return;
  const long q = t / bb;
  const int e = (int)(t - q * bb), r = e / b, c = e - r * b;
  tval[t] = val[(long)tblk[q] * bb + (long)c * b + r];
}

// Host-built transpose of a BSR pattern (cached per pattern pointer for the SpMV entry points).
struct Transpose {
  std::vector<int> ptr, idx, blk;
};
void build_transpose(int nbr, int nbc, const int* ptr, const int* idx, Transpose* t) {
  t->ptr.assign(nbc + 1, 0);
  for (int i = 0; i < nbr; ++i)
    for (int q = ptr[i]; q < ptr[i + 1]; ++q) t->ptr[idx[q] + 1]++;
  for (int j = 0; j < nbc; ++j) t->ptr[j + 1] += t->ptr[j];
  t->idx.assign(t->ptr[nbc], 0);
  t->blk.assign(t->ptr[nbc], 0);
  std::vector<int> fill(t->ptr.begin(), t->ptr.end() - 1);
  for (int i = 0; i < nbr; ++i)
    for (int q = ptr[i]; q < ptr[i + 1]; ++q) {
      int s = fill[idx[q]]++;
      t->idx[s] = i;
      t->blk[s] = q;
    }
}

// ------------------------------------------------------------------------------ ILU(0)
template <class V>
struct IluView {
  int n, b;
  const int* ptr;
  const int* idx;
  const int* diag;  // block index of the diagonal block of each row
  V* val;
};

__device__ __forceinline__ void note_zero_pivot(unsigned long long* flag, int row, int col) {
  unsigned long long key = ((unsigned long long)(unsigned)row << 32) | (unsigned)col;
  atomicMin(flag, key);
}

// Factor the block rows of one level.  One thread per block row.
template <class V>
__global__ void k_ilu_factor_level(IluView<V> F, const int* rows, int count,
                                   unsigned long long* zero_flag) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t];
  const int b = F.b;
  const long bb = (long)b * b;
  const int rb = F.ptr[i], re = F.ptr[i + 1], di = F.diag[i];
  // lower blocks, ascending column
  for (int q = rb; q < di; ++q) {
    const int j = F.idx[q];
    V* Lij = F.val + (long)q * bb;
    const V* Ujj = F.val + (long)F.diag[j] * bb;
    // L_ij = A_ij U_jj^-1, column by column (scalar columns jb ascending)
    for (int cb = 0; cb < b; ++cb) {
      const V piv = Ujj[(long)cb * b + cb];
      if (piv == V(0)) note_zero_pivot(zero_flag, i * b, j * b + cb);
      for (int a = 0; a < b; ++a) {
        V l = Lij[(long)a * b + cb] / piv;
        Lij[(long)a * b + cb] = l;
        for (int c2 = cb + 1; c2 < b; ++c2) Lij[(long)a * b + c2] -= l * Ujj[(long)cb * b + c2];
      }
    }
    // A_ik -= L_ij A_jk for k > j present in both rows (merge of sorted column lists)
    int p = q + 1;
    for (int s = F.diag[j] + 1; s < F.ptr[j + 1]; ++s) {
      const int k = F.idx[s];
      while (p < re && F.idx[p] < k) ++p;
      if (p >= re) break;
      if (F.idx[p] != k) continue;
      V* Aik = F.val + (long)p * bb;
      const V* Ajk = F.val + (long)s * bb;
      for (int a = 0; a < b; ++a)
        for (int c = 0; c < b; ++c) {
          V acc = Aik[(long)a * b + c];
          for (int m = 0; m < b; ++m) acc -= Lij[(long)a * b + m] * Ajk[(long)m * b + c];
          Aik[(long)a * b + c] = acc;
        }
    }
  }
  // diagonal block: in-place LU (unit lower), and L_ii^-1 applied to the upper blocks
  V* D = F.val + (long)di * bb;
  for (int cb = 0; cb < b; ++cb) {
    const V piv = D[(long)cb * b + cb];
    for (int a = cb + 1; a < b; ++a) {
      if (piv == V(0)) note_zero_pivot(zero_flag, i * b + a, i * b + cb);
      V l = D[(long)a * b + cb] / piv;
      D[(long)a * b + cb] = l;
      for (int c = cb + 1; c < b; ++c) D[(long)a * b + c] -= l * D[(long)cb * b + c];
      for (int q = di + 1; q < re; ++q) {
        V* U = F.val + (long)q * bb;
        for (int c = 0; c < b; ++c) U[(long)a * b + c] -= l * U[(long)cb * b + c];
      }
    }
  }
}

// Forward sweep (L y = r, unit lower) for one level; y may be r.
template <class V>
__global__ void k_ilu_lower(IluView<V> F, const int* rows, int count, const V* r, V* y) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t], b = F.b;
  const long bb = (long)b * b;
  V acc[8];
  for (int a = 0; a < b; ++a) acc[a] = r[(long)i * b + a];
  for (int q = F.ptr[i]; q < F.diag[i]; ++q) {
    const V* L = F.val + (long)q * bb;
    const V* yj = y + (long)F.idx[q] * b;
    for (int a = 0; a < b; ++a)
      for (int c = 0; c < b; ++c) acc[a] -= L[(long)a * b + c] * yj[c];
  }
  const V* D = F.val + (long)F.diag[i] * bb;
  for (int a = 0; a < b; ++a) {
    V s = acc[a];
    for (int c = 0; c < a; ++c) s -= D[(long)a * b + c] * acc[c];
    acc[a] = s;
    y[(long)i * b + a] = s;
  }
}

// Backward sweep (U x = y) for one level; x holds y on entry.  Per scalar row the upper entries
// are consumed in ascending column order (in-block first, then the blocks k > i), as in
// aquaflux/solve/_ilu0.pyx:143-147.
template <class V>
__global__ void k_ilu_upper(IluView<V> F, const int* rows, int count, V* x) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t], b = F.b;
  const long bb = (long)b * b;
  const V* D = F.val + (long)F.diag[i] * bb;
  V* xi = x + (long)i * b;
  for (int a = b - 1; a >= 0; --a) {
    V s = xi[a];
    for (int c = a + 1; c < b; ++c) s -= D[(long)a * b + c] * xi[c];
    for (int q = F.diag[i] + 1; q < F.ptr[i + 1]; ++q) {
      const V* U = F.val + (long)q * bb + (long)a * b;
      const V* xk = x + (long)F.idx[q] * b;
      for (int c = 0; c < b; ++c) s -= U[c] * xk[c];
    }
    xi[a] = s / D[(long)a * b + a];
  }
}

// Transposed sweeps use the transpose map: tptr/tidx/tblk list, for block column i, the rows j
// and block indices of the stored blocks (j, i).
// U^T z = r: forward over block columns; z_i = U_ii^-T (r_i - sum_{j<i} U_ji^T z_j).
template <class V>
__global__ void k_ilu_upper_t(IluView<V> F, const int* tptr, const int* tidx, const int* tblk,
                              const int* rows, int count, const V* r, V* z) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t], b = F.b;
  const long bb = (long)b * b;
  V acc[8];
  for (int a = 0; a < b; ++a) acc[a] = r[(long)i * b + a];
  for (int q = tptr[i]; q < tptr[i + 1]; ++q) {
    const int j = tidx[q];
    if (j >= i) continue;
    const V* U = F.val + (long)tblk[q] * bb;  // block (j, i)
    const V* zj = z + (long)j * b;
    for (int a = 0; a < b; ++a)
      for (int c = 0; c < b; ++c) acc[a] -= U[(long)c * b + a] * zj[c];
  }
  const V* D = F.val + (long)F.diag[i] * bb;
  for (int a = 0; a < b; ++a) {
    V s = acc[a];
    for (int c = 0; c < a; ++c) s -= D[(long)c * b + a] * acc[c];
    s = s / D[(long)a * b + a];
    acc[a] = s;
    z[(long)i * b + a] = s;
  }
}

// L^T x = z: backward over block columns; x_i = L_ii^-T (z_i - sum_{k>i} L_ki^T x_k).  The
// contributions are taken in descending row order, the order of the reference's scatter form
// (aquaflux/solve/_ilu0.pyx:174-178).
template <class V>
__global__ void k_ilu_lower_t(IluView<V> F, const int* tptr, const int* tidx, const int* tblk,
                              const int* rows, int count, V* x) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t], b = F.b;
  const long bb = (long)b * b;
  const V* D = F.val + (long)F.diag[i] * bb;
  V* xi = x + (long)i * b;
  for (int a = b - 1; a >= 0; --a) {
    V s = xi[a];
    for (int q = tptr[i + 1] - 1; q >= tptr[i]; --q) {
      const int k = tidx[q];
      if (k <= i) continue;
      const V* L = F.val + (long)tblk[q] * bb;  // block (k, i)
      const V* xk = x + (long)k * b;
      for (int c = b - 1; c >= 0; --c) s -= L[(long)c * b + a] * xk[c];
    }
    for (int c = b - 1; c > a; --c) s -= D[(long)c * b + a] * xi[c];
    xi[a] = s;
  }
}

// ---- lane-group kernels: an 8-lane group per block row, lane a owns scalar row / column a of
// the block (b <= 8), so the b x b block work of a row runs on b lanes instead of one thread.
// Element-wise operation orders are those of the one-thread kernels above, except the forward
// solve's upper sweep, which subtracts the off-diagonal blocks before the in-block terms (the
// reference subtracts in ascending column order); b = 1 uses the one-thread kernels.
// A level's kernel is launched while the one before still runs (programmatic dependent launch): it
// lets the next one start, finds its rows and asks the L2 cache for their blocks, which no sweep
// writes, and only then waits for the level before.  Without that each level paid its launch and
// the memory latency of rows, offsets, columns and blocks in turn.
__device__ __forceinline__ void next_level_may_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_level_before() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
#define FV_LG 8
__device__ __forceinline__ unsigned lg_mask() { return 0xffu << ((threadIdx.x & 31) & ~(FV_LG - 1)); }

// Factor the block rows of one level, a group of FV_LG lanes per block row (lane a = row a of the
// block), with a compile-time block size: the row's lower block, the pivot row's diagonal block and
// each upper block it updates with are held in registers (vector loads), the diagonal block's pivot
// rows are shuffled from the lane that owns them.  Every entry sees the scalar elimination of
// k_ilu_factor_level in the same order, so the factors are bitwise the same.  For the wider levels
// (factor_wide), where rows enough are in flight and a fourth of a warp per row issues less.
template <class V, int B>
__global__ void k_ilu_factor_lgb(IluView<V> F, const int* rows, int count,
                                 V* rp, unsigned long long* zero_flag) {
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;  // whole groups exit together
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  const int ar = live ? a : 0;  // row index of the lane's (possibly unused) loads
  constexpr long BB = (long)B * B;
  const int re = F.ptr[i + 1], di = F.diag[i];
  for (int q = F.ptr[i]; q < di; ++q) {
    const int j = F.idx[q];
    V* Lij = F.val + (long)q * BB;
    const V* Ujj = F.val + (long)F.diag[j] * BB;
    V L[B], U[B * B];
    load_seg<B>(Lij + (long)ar * B, L);
#pragma unroll
    for (int r = 0; r < B; ++r) {
      V row[B];
      load_seg<B>(Ujj + (long)r * B, row);
#pragma unroll
      for (int c = 0; c < B; ++c) U[r * B + c] = row[c];
    }
#pragma unroll
    for (int cb = 0; cb < B; ++cb) {
      const V piv = U[cb * B + cb];
      if (piv == V(0) && a == 0) note_zero_pivot(zero_flag, i * B, j * B + cb);
      const V l = L[cb] / piv;
      L[cb] = l;
#pragma unroll
      for (int c2 = cb + 1; c2 < B; ++c2) L[c2] -= l * U[cb * B + c2];
    }
    if (live) {
#pragma unroll
      for (int c = 0; c < B; ++c) Lij[(long)a * B + c] = L[c];
    }
    // A_ik -= L_ij A_jk for k > j present in both rows (merge of sorted column lists)
    int p = q + 1;
    for (int s2 = F.diag[j] + 1; s2 < F.ptr[j + 1]; ++s2) {
      const int k = F.idx[s2];
      while (p < re && F.idx[p] < k) ++p;
      if (p >= re) break;
      if (F.idx[p] != k) continue;
      V* Aik = F.val + (long)p * BB + (long)ar * B;
      const V* Ajk = F.val + (long)s2 * BB;
      V A[B], M[B * B];
      load_seg<B>(Aik, A);
#pragma unroll
      for (int r = 0; r < B; ++r) {
        V row[B];
        load_seg<B>(Ajk + (long)r * B, row);
#pragma unroll
        for (int c = 0; c < B; ++c) M[r * B + c] = row[c];
      }
#pragma unroll
      for (int c = 0; c < B; ++c) {
        V acc = A[c];
#pragma unroll
        for (int mm = 0; mm < B; ++mm) acc -= L[mm] * M[mm * B + c];
        A[c] = acc;
      }
      if (live) {
#pragma unroll
        for (int c = 0; c < B; ++c) Aik[c] = A[c];
      }
    }
  }
  __syncwarp(mask);
  V* D = F.val + (long)di * BB;
  V Drow[B];
  load_seg<B>(D + (long)ar * B, Drow);
#pragma unroll
  for (int cb = 0; cb < B; ++cb) {
    // row cb of the diagonal block is final: lane cb's registers; of the upper blocks: in memory
    V prow[B];
#pragma unroll
    for (int c = 0; c < B; ++c) prow[c] = __shfl_sync(mask, Drow[c], cb, FV_LG);
    if (live && a > cb) {
      const V piv = prow[cb];
      if (piv == V(0)) note_zero_pivot(zero_flag, i * B + a, i * B + cb);
      const V l = Drow[cb] / piv;
      Drow[cb] = l;
#pragma unroll
      for (int c = cb + 1; c < B; ++c) Drow[c] -= l * prow[c];
      for (int q = di + 1; q < re; ++q) {
        V* Ub = F.val + (long)q * BB;
        V ua[B], uc[B];
        load_seg<B>(Ub + (long)a * B, ua);
        load_seg<B>(Ub + (long)cb * B, uc);
#pragma unroll
        for (int c = 0; c < B; ++c) ua[c] -= l * uc[c];
#pragma unroll
        for (int c = 0; c < B; ++c) Ub[(long)a * B + c] = ua[c];
      }
    }
    __syncwarp(mask);
  }
  if (live) {
    V piv = Drow[0];
#pragma unroll
    for (int c = 0; c < B; ++c) {
      D[(long)a * B + c] = Drow[c];
      if (c == a) piv = Drow[c];
    }
    if (rp) rp[(long)i * B + a] = V(1) / piv;  // (a level by warps follows)
  }
}

// ---- factorisation: a warp per block row, the row's blocks in shared memory.
// What bounds it is the chain along a row's lower blocks, not bytes: with 8 lanes a row and every
// block updated in place in global memory, each lower block cost five or six dependent memory round
// trips and a merge of two index lists (fp32, b = 6, 9-27 blocks a row: 100-185 us a level set
// whatever its width; fp64 cavity: 11.9 us a level set of 64 rows).  Here a row's blocks and columns
// are copied in once and back once; the lower blocks' rows j are looked up by 32 lanes at once; the
// columns of row j come in one load, each lane counting row i's columns below its own to find its
// place; what the pattern alone gives is found before the level before is waited for; the next row
// j is fetched and the matching blocks' columns are read before the chain of quotients, which hides
// them; and the matching blocks are updated side by side.  Pivots of finished rows come with their
// reciprocals (`rp`): a quotient is a product and a correction, not a division on the chain (fp64: 192 cycles
// for 321).
// Lanes: for b <= 4 one per block entry (16 to a block, two blocks at a time), which keeps the
// number of fp64 instructions, 64 cycles each, at one per elimination step; above, one per column
// (8 to a block, four blocks at a time).
// Every entry sees the scalar elimination of k_ilu_factor_level in the same order: bitwise the same.

// x / piv: in fp64 through the pivot's reciprocal (see upper_block_solve) where the quotient is far
// from under- and overflow (192 cycles of fp64 issue for a division's 321).
__device__ __forceinline__ bool mid_range(double q) {
  const int e = __double2hiint(q) & 0x7ff00000;
  return e > 0x10000000 && e < 0x70000000;
}
__device__ __forceinline__ double quotient(double x, double piv, double rpiv) {
  const double q = x * rpiv;
  if ((__double_as_longlong(x) << 1) == 0 && isfinite(rpiv)) return q;
  if (mid_range(q) && mid_range(x) && mid_range(rpiv)) return fma_rn(fma_rn(-q, piv, x), rpiv, q);
  return x / piv;
}
__device__ __forceinline__ float quotient(float x, float piv, float) { return x / piv; }

// Levels of at least this many rows take 8 lanes a row, whose time is a chain along a row's lower
// blocks while the lanes last; a warp a row shortens the chain and takes four times the lanes, so
// the line lies higher the longer the rows (`lower`: most lower blocks of a row in the level), and
// in a level of uneven rows, whose longest is the lanes' chain and whose mean the warps' work, by
// their ratio.  fp32, us a factor of four level sets, lane groups / warps, by lower blocks and rows:
//   b = 6    3:  5,000  98 /  99    6: 5,000 142 / 129, 8,191 162 / 187
//           16:  8,191 448 / 411, 12,000 490 / 562
//   b = 4    3:  5,000  78 /  81    6: 5,000 112 / 113, 8,191 116 / 125   16: 12,000 345 / 347
//   b = 2    3:  3,000  63 /  65    6: 8,192  97 / 100                    16: 12,000 270 / 255
//   b = 8   10:  8,191 306 / 354   16: 8,191 510 / 545
// and at 65,535 rows of 6 lower blocks 622 / 1,171, 342 / 737, 184 / 484 (80^3 grid in reverse
// Cuthill-McKee order, level sets of up to 4,800 rows of 3: b = 2 1,438 / 1,223, b = 4 1,979 / 1,714,
// b = 6 2,571 / 2,514; 96^3, 6,900 rows: 1,923 / 1,913, 2,619 / 2,715, 3,560 / 3,627).
// Rows scattered over the matrix (a grid's own order, where a level set is a diagonal) cost the lane
// groups' short reads more than the warps' long ones: 80^3 grid, level sets of up to 4,800 rows, us
// a factor with the line at 4,000 / 6,144: b = 2 1,466 / 1,216, b = 4 1,956 / 1,698, b = 6 2,614 /
// 2,521; 112^3, 9,408 rows, at 6,144 / 8,192 / 12,288: b = 3 3,191 / 3,137 / 3,307, b = 6 4,721 /
// 4,892 / 5,455.
constexpr int factor_wide(int b, int lower, bool scattered) {
  const int line = b <= 4   ? 512 * lower + 3400
                   : b <= 6 ? 256 * lower + 4100
                            : 128 * lower + 3600;
  return scattered ? std::max(line, b <= 4 ? 8192 : 6144) : line;
}
// fp64 issue is four times scarcer for a warp a row than for four rows a warp, so there the line is
// where the warps' rows fill the SMs' fp64 units; with a lane an entry (b <= 4) it lies higher (3D
// 48^3, 142 level sets of up to 1,728 rows: b = 6 lane groups 6.55 ms, warps 5.9 ms, warps below
// 1,024 rows 5.15; b = 4 3.91, 2.46, 2.79.  80^3, up to 4,800 rows, b = 6: 13.0, 20.7 and 11.6).
// And a level launched early is placed where it finds room, not where fp64 units are free: it pays
// only while a level has no more rows than there are SMs (64 x 64 cavity 793 us, 1026 without; the
// 48^3 b = 6 factor 8.4 ms with every level early, 6.2 with none).
// The warps' time goes by rounds of one warp on each of the 608 quarters of an SM, the lane groups'
// by the chain: with few lower blocks a round less.  Warps / lane groups, 12 level sets, by lower
// blocks:
//   b = 3   1,100 rows  2: 0.93, 3: 0.84   1,300  2: 1.09, 3: 1.08, 4: 0.95   1,900  4: 1.15, 6: 0.98
//   b = 6     600 rows  1: 0.87, 3: 0.69     800  1: 1.25, 2: 1.16, 3: 1.06, 6: 0.92
// (3: 48^3 grid in reverse Cuthill-McKee order, level sets of up to 1,728 rows, b = 4 2,522 us with
// all of them by warps, 2,670 from 1,217 rows on by lane groups).  Scattered, the same grid's own
// order, line at 1,024 / 2,048: b = 4 2,745 / 2,450.
constexpr int factor_wide64(int b, int lower, bool scattered) {
  constexpr int round = 4 * 152;
  if (b > 4) return scattered || lower >= 3 ? 1024 : round + 1;
  return scattered || lower >= 6 ? 2048 : (lower >= 3 ? 3 : 2) * round + 1;
}
constexpr int kEarly64 = 152;
constexpr size_t kFactorSmem = 96 * 1024;

// Shared memory of one warp: the matches of one lower block, the row's columns (padded to a
// multiple of four), the pivot row's diagonal block and reciprocals, the row's blocks.
template <class V>
__host__ __device__ constexpr size_t factor_warp_bytes(int cap, int bb) {
  return (32 * 8 + (size_t)(cap + 7) / 4 * 16 + 72 * sizeof(V) + (size_t)cap * bb * sizeof(V) + 15) /
         16 * 16;
}

template <class V, int B>
__global__ void __launch_bounds__(128) k_ilu_factor_w(IluView<V> F, const int* rows, int count,
                                                      int cap, V* rp,
                                                      unsigned long long* zero_flag) {
  constexpr int BB = B * B;
  constexpr bool EM = B <= 4;            // a lane per entry
  constexpr int SG = EM ? 16 : 8, NSG = 32 / SG;
  extern __shared__ __align__(16) unsigned char factor_smem[];
  next_level_may_start();
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x / 32) + warp;
  if (w >= count) return;  // whole warps exit together
  int2* match = (int2*)(factor_smem + (size_t)warp * factor_warp_bytes<V>(cap, BB));
  int* cols = (int*)(match + 32);
  V* Us = (V*)(cols + (cap + 7) / 4 * 4);
  V* blk = Us + 72;
  const int i = rows[w], rb = F.ptr[i], nb = F.ptr[i + 1] - rb, nl = F.diag[i] - rb;
  V* row = F.val + (long)rb * BB;
  for (int k = lane; k < nb + 4; k += 32) cols[k] = k < nb ? F.idx[rb + k] : 0x7fffffff;
#pragma unroll 4
  for (int k = lane; k < nb * BB; k += 32) blk[k] = row[k];
  const int e = lane & (SG - 1), sg = lane / SG;
  const unsigned sgmask = (SG == 16 ? 0xffffu : 0xffu) << (sg * SG);
  const bool live = e < (EM ? BB : B);
  const int el = live ? e : 0;
  const int a = EM ? el / B : el, c = EM ? el % B : el;  // EM: entry (a, c); else row a / column c
  __syncwarp();

  int jl = 0, dl = 0, rl = 0;  // lane's lower block: row j, its diagonal's position and its end
  // the coming lower block's row: columns (one a lane), diagonal block and reciprocals
  constexpr int PU = (BB + B + 31) / 32;
  int j = 0, dj = 0, ej = 0, kcol = -1;
  V pu[PU];
  auto place = [&](int q) {  // (the pattern only)
    if ((q & 31) == 0 && q + lane < nl) {
      jl = cols[q + lane];
      dl = F.diag[jl];
      rl = F.ptr[jl + 1];
    }
    j = __shfl_sync(0xffffffffu, jl, q & 31);
    dj = __shfl_sync(0xffffffffu, dl, q & 31);
    ej = __shfl_sync(0xffffffffu, rl, q & 31);
    kcol = dj + 1 + lane < ej ? F.idx[dj + 1 + lane] : -1;
  };
  auto fetch = [&] {
#pragma unroll
    for (int u = 0; u < PU; ++u) {
      const int k = u * 32 + lane;
      if (k < BB) pu[u] = F.val[(long)dj * BB + k];
      else if (k < BB + B) pu[u] = rp[(long)j * B + k - BB];
    }
  };
  // the lanes' columns of row j stored in row i too, as (position in row i, block of row j); their
  // number
  auto find = [&](int q, int key, int s) {
    int lo = 0;
    if (nb <= 64) {  // columns below the key, counted (no chain of dependent reads)
      for (int k = 0; k < nb; k += 4) {
        const int4 v = *reinterpret_cast<const int4*>(cols + k);
        lo += (v.x < key) + (v.y < key) + (v.z < key) + (v.w < key);
      }
    } else {
      int hi = nb;
      lo = q + 1;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid] < key) lo = mid + 1;
        else hi = mid;
      }
      __syncwarp();
    }
    const bool found = key >= 0 && lo < nb && cols[lo] == key;
    const unsigned mask = __ballot_sync(0xffffffffu, found);
    if (found) match[__popc(mask & ((1u << lane) - 1))] = make_int2(lo, s);
    __syncwarp();
    return __popc(mask);
  };
  auto column = [&](int t, int m, V (&Mc)[B]) {  // column c of match t's block of row j
    if (t < m) {
      const V* M = F.val + (long)match[t].y * BB + c;
#pragma unroll
      for (int k = 0; k < B; ++k) Mc[k] = M[k * B];
    }
  };
  auto update = [&](int t, int m, const V* Lq, const V (&Mc)[B]) {  // A_ik -= L_ij A_jk
    if (t >= m) return;
    V* A = blk + match[t].x * BB;
    if constexpr (EM) {
      V acc = A[el];
#pragma unroll
      for (int k = 0; k < B; ++k) acc -= Lq[a * B + k] * Mc[k];
      if (live) A[e] = acc;
    } else {
#pragma unroll
      for (int r = 0; r < B; ++r) {
        V acc = A[r * B + c], Lr[B];
        load_seg<B>(Lq + r * B, Lr);
#pragma unroll
        for (int k = 0; k < B; ++k) acc -= Lr[k] * Mc[k];
        if (live) A[r * B + c] = acc;
      }
    }
  };
  int m = 0;
  if (nl > 0) {
    place(0);
    m = find(0, kcol, dj + 1 + lane);
  }
  // only the pattern and the row itself, which no earlier level writes, were read so far
  wait_level_before();
  if (nl > 0) fetch();
  for (int q = 0; q < nl; ++q) {
    const int jq = j, s0 = dj + 1, eq = ej;
    V M0[B];
    column(sg, m, M0);
#pragma unroll
    for (int u = 0; u < PU; ++u)
      if (u * 32 + lane < BB + B) Us[u * 32 + lane] = pu[u];
    __syncwarp();
    if (q + 1 < nl) {
      place(q + 1);
      fetch();
    }
    // L_ij = A_ij U_jj^-1, scalar columns ascending
    V* Lq = blk + q * BB;
    if constexpr (EM) {
      V x = Lq[el];
#pragma unroll
      for (int cb = 0; cb < B; ++cb) {
        const V piv = Us[cb * B + cb];
        if (piv == V(0) && lane == 0) note_zero_pivot(zero_flag, i * B, jq * B + cb);
        if (c == cb) x = quotient(x, piv, Us[BB + cb]);
        const V l = __shfl_sync(0xffffffffu, x, a * B + cb, SG);
        if (cb < B - 1 && c > cb) x -= l * Us[cb * B + c];
      }
      __syncwarp();
      if (live && sg == 0) Lq[e] = x;
    } else {
      V L[B];
      load_seg<B>(Lq + a * B, L);
#pragma unroll
      for (int cb = 0; cb < B; ++cb) {
        V Ur[B];
        load_seg<B>(Us + cb * B, Ur);
        const V piv = Ur[cb];
        if (piv == V(0) && lane == 0) note_zero_pivot(zero_flag, i * B, jq * B + cb);
        const V l = quotient(L[cb], piv, Us[BB + cb]);
        L[cb] = l;
#pragma unroll
        for (int k = cb + 1; k < B; ++k) L[k] -= l * Ur[k];
      }
      __syncwarp();
      if (live && sg == 0) {
#pragma unroll
        for (int k = 0; k < B; ++k) Lq[a * B + k] = L[k];
      }
    }
    __syncwarp();
    update(sg, m, Lq, M0);
    for (int t = sg + NSG; t < m; t += NSG) {
      column(t, m, M0);
      update(t, m, Lq, M0);
    }
    __syncwarp();
    for (int s = s0 + 32; s < eq; s += 32) {  // more than 32 columns in row j
      const int more = find(q, s + lane < eq ? F.idx[s + lane] : -1, s + lane);
      for (int t = sg; t < more; t += NSG) {
        column(t, more, M0);
        update(t, more, Lq, M0);
      }
      __syncwarp();
    }
    if (q + 1 < nl) m = find(q + 1, kcol, dj + 1 + lane);
  }
  // the diagonal block: in-place LU (unit lower)
  V* D = blk + nl * BB;
  if constexpr (EM) {
    V x = D[el];
#pragma unroll
    for (int cb = 0; cb < B - 1; ++cb) {
      const V piv = __shfl_sync(0xffffffffu, x, cb * B + cb, SG);
      if (c == cb && a > cb && live && sg == 0) {
        if (piv == V(0)) note_zero_pivot(zero_flag, i * B + a, i * B + cb);
      }
      if (c == cb && a > cb) x = x / piv;
      const V l = __shfl_sync(0xffffffffu, x, a * B + cb, SG);
      const V p = __shfl_sync(0xffffffffu, x, cb * B + c, SG);
      if (a > cb && c > cb) x -= l * p;
    }
    __syncwarp();
    if (live && sg == 0) D[e] = x;
  } else {
    V x[B];
#pragma unroll
    for (int m = 0; m < B; ++m) x[m] = D[a * B + m];
#pragma unroll
    for (int cb = 0; cb < B - 1; ++cb) {
      V p[B];
#pragma unroll
      for (int m = cb; m < B; ++m) p[m] = __shfl_sync(0xffffffffu, x[m], cb, SG);
      if (a > cb) {
        if (p[cb] == V(0) && live && sg == 0) note_zero_pivot(zero_flag, i * B + a, i * B + cb);
        const V l = x[cb] / p[cb];
        x[cb] = l;
#pragma unroll
        for (int m = cb + 1; m < B; ++m) x[m] -= l * p[m];
      }
    }
    __syncwarp();
    if (live && sg == 0) {
#pragma unroll
      for (int m = 0; m < B; ++m) D[a * B + m] = x[m];
    }
  }
  __syncwarp();
  if (lane < B) rp[(long)i * B + lane] = V(1) / D[lane * B + lane];
  // the upper blocks: L_ii^-1 applied
  for (int t = nl + 1 + sg; t < nb; t += NSG) {
    V* U = blk + t * BB;
    if constexpr (EM) {
      V x = U[el];
#pragma unroll
      for (int cb = 0; cb < B - 1; ++cb) {
        const V uc = __shfl_sync(sgmask, x, cb * B + c, SG);
        if (a > cb) x -= D[a * B + cb] * uc;
      }
      if (live) U[e] = x;
    } else {
      V u[B];
#pragma unroll
      for (int r = 0; r < B; ++r) u[r] = U[r * B + c];
#pragma unroll
      for (int cb = 0; cb < B - 1; ++cb)
#pragma unroll
        for (int r = cb + 1; r < B; ++r) u[r] -= D[r * B + cb] * u[cb];
      if (live) {
#pragma unroll
        for (int r = 0; r < B; ++r) U[r * B + c] = u[r];
      }
    }
  }
  __syncwarp();
#pragma unroll 4
  for (int k = lane; k < nb * BB; k += 32) row[k] = blk[k];
}

// How the lane groups of a level read their rows (launch_apply_levels chooses):
//   kPlain   a launch after the other; the compiler's unrolling reads a few blocks ahead
//   kEarly   the same, launched before the level before has ended
//   kDeep    so too, two blocks at a time, the columns of eight by the group's lanes at once
//   kStream  a launch after the other, one block at a time: the fewest registers, the most warps
// Each asks the L2 cache for the row's first lines, or all of them (`ask` bytes), before its first
// read.
enum Read { kPlain, kEarly, kDeep, kStream };
__host__ __device__ constexpr bool early(int m) { return m == kEarly || m == kDeep; }

// acc minus the products of `count` blocks (positions q0, q0 + STEP, ...) with their columns'
// entries of x, in that order (and, STEP = -1, each block's entries from the last).
template <class V, int B, int STEP, int M>
__device__ __forceinline__ V subtract_blocks(V acc, const V* val, const int* idx, const V* x, int q0,
                                             int count, int a, bool live, unsigned mask) {
  constexpr long BB = (long)B * B;
  auto block = [&](const V (&L)[B], const V (&xj)[B]) {
#pragma unroll
    for (int c = 0; c < B; ++c) {
      const int e = STEP > 0 ? c : B - 1 - c;
      acc -= L[e] * xj[e];
    }
  };
  auto one = [&](int q) {
    V L[B], xj[B];
    load_seg<B>(val + (long)q * BB + (long)a * B, L);
    load_seg<B>(x + (long)idx[q] * B, xj);
    block(L, xj);
  };
  if constexpr (M == kDeep) {
    for (int k0 = 0; k0 < count; k0 += FV_LG) {
      const int col = k0 + a < count ? idx[q0 + STEP * (k0 + a)] : 0;
      for (int k = k0; k < count && k < k0 + FV_LG; k += 2) {
        V L[2][B], xj[2][B];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (live && k + u < count)
            load_seg<B>(val + (long)(q0 + STEP * (k + u)) * BB + (long)a * B, L[u]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = __shfl_sync(mask, col, k - k0 + u, FV_LG);
          if (live && k + u < count) load_seg<B>(x + (long)j * B, xj[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (live && k + u < count) block(L[u], xj[u]);
      }
    }
  } else if constexpr (M == kStream) {
    if (live)
#pragma unroll 1
      for (int k = 0; k < count; ++k) one(q0 + STEP * k);
  } else {
    if (live) {
      if (STEP > 0)
        for (int q = q0; q < q0 + count; ++q) one(q);
      else
        for (int q = q0; q > q0 - count; --q) one(q);
    }
  }
  return acc;
}

template <class V, int B>
__device__ __forceinline__ void ask_blocks(const V* val, int q0, int count, int a, int ask) {
  // lane a asks for the lines at a, a + 8, ... of the blocks' contiguous range, of its first `ask`
  // bytes
  const char* p = (const char*)(val + (long)q0 * B * B);
  const long end = min((long)count * B * B * (long)sizeof(V), (long)ask);
  for (long o = 128L * a; o < end; o += 128L * FV_LG)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

// Forward sweep of one level, a group of FV_LG lanes per block row (lane a = row a of the block).
template <class V, int B, int M>
__global__ void k_ilu_lower_lg(IluView<V> F, const int* rows, int count, int ask, const V* r,
                               V* y) {
  if (early(M)) next_level_may_start();
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  constexpr long BB = (long)B * B;
  const int q0 = F.ptr[i], di = F.diag[i];
  ask_blocks<V, B>(F.val, q0, di - q0 + 1, a, ask);
  if (early(M)) wait_level_before();
  V acc = live ? r[(long)i * B + a] : V(0);
  acc = subtract_blocks<V, B, 1, M>(acc, F.val, F.idx, y, q0, di - q0, a, live, mask);
  V D[B];
  if (live) load_seg<B>(F.val + (long)di * BB + (long)a * B, D);
#pragma unroll
  for (int c = 0; c < B; ++c) {
    const V vc = __shfl_sync(mask, acc, c, FV_LG);
    if (live && a > c) acc -= D[c] * vc;
  }
  if (live) y[(long)i * B + a] = acc;
}

// The in-block upper solve of one block row (lane a holds entry a of the row's right-hand side,
// D the lane's row of the diagonal block).  Every lane forms the correctly rounded reciprocal r
// of its own pivot d up front (all lanes at once), so the dependent chain needs no division: a
// division there runs on one lane in eight at each step (fp32: 87 us of a 155 us diagonal-only
// sweep of 1M block rows under ncu; fp64: the 128^3 fine-level solve 6.5 ms with divisions,
// GB300).  The quotient x / d is q = x r corrected once, q + (x - q d) r, with fused
// multiply-adds: by Markstein's theorem (IBM J. Res. Develop. 34(1), 1990) the correctly rounded
// quotient, outside the underflow range (pinned bitwise against IEEE division in both precisions
// by the sparse-solver tests).  A lane whose reciprocal overflows (fp32 pivot below ~3e-39)
// divides.
template <class V, int B>
__device__ __forceinline__ V upper_block_solve(V acc, const V (&D)[B], int a, bool live,
                                               unsigned mask) {
  V piv = V(1);
#pragma unroll
  for (int c = 0; c < B; ++c)
    if (a == c) piv = D[c];
  const V rpiv = V(1) / piv;
  const bool rfin = isfinite(rpiv);
#pragma unroll
  for (int c = B - 1; c >= 0; --c) {
    if (a == c) {
      if (rfin) {
        const V q = acc * rpiv;
        acc = fma_rn(fma_rn(-q, piv, acc), rpiv, q);
      } else {
        acc = acc / piv;
      }
    }
    const V vc = __shfl_sync(mask, acc, c, FV_LG);
    if (live && a < c) acc -= D[c] * vc;
  }
  return acc;
}

// Backward sweep of one level (U x = y).
template <class V, int B, int M>
__global__ void k_ilu_upper_lg(IluView<V> F, const int* rows, int count, int ask, V* x) {
  if (early(M)) next_level_may_start();
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  constexpr long BB = (long)B * B;
  const int di = F.diag[i], re = F.ptr[i + 1];
  ask_blocks<V, B>(F.val, di, re - di, a, ask);
  if (early(M)) wait_level_before();
  V acc = live ? x[(long)i * B + a] : V(0);
  acc = subtract_blocks<V, B, 1, M>(acc, F.val, F.idx, x, di + 1, re - di - 1, a, live, mask);
  V D[B];
  if (live) load_seg<B>(F.val + (long)di * BB + (long)a * B, D);
  acc = upper_block_solve<V, B>(acc, D, a, live, mask);
  if (live) x[(long)i * B + a] = acc;
}

// The last forward level followed by the first backward level on the same rows, one kernel: when
// those rows own no upper blocks (the second colour of a two-colour order), a row's backward step
// is the in-block upper solve of its own forward result, with the diagonal block already in
// registers.  The same operations in the same order as the two separate sweeps.
template <class V, int B, int M>
__global__ void k_ilu_lower_upper_lg(IluView<V> F, const int* rows, int count, int ask, const V* r,
                                     V* y) {
  if (early(M)) next_level_may_start();
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  constexpr long BB = (long)B * B;
  const int q0 = F.ptr[i], di = F.diag[i];
  ask_blocks<V, B>(F.val, q0, di - q0 + 1, a, ask);
  if (early(M)) wait_level_before();
  V acc = live ? r[(long)i * B + a] : V(0);
  acc = subtract_blocks<V, B, 1, M>(acc, F.val, F.idx, y, q0, di - q0, a, live, mask);
  V D[B];
  if (live) load_seg<B>(F.val + (long)di * BB + (long)a * B, D);
#pragma unroll
  for (int c = 0; c < B; ++c) {
    const V vc = __shfl_sync(mask, acc, c, FV_LG);
    if (live && a > c) acc -= D[c] * vc;
  }
  acc = upper_block_solve<V, B>(acc, D, a, live, mask);
  if (live) y[(long)i * B + a] = acc;
}

// The in-block lower solve of U^T's diagonal block D^T (lane a holds entry a of the right-hand
// side, Dc the lane's column of D: Dc[c] = D(c, a)): step c divides entry c by its pivot D(c, c),
// then every later entry a > c takes -D(c, a) times it.  The division is the reciprocal quotient
// of upper_block_solve (every lane's reciprocal formed up front, one fused correction: the
// correctly rounded quotient, the same value as the division).
template <class V, int B>
__device__ __forceinline__ V lower_t_block_solve(V acc, const V (&Dc)[B], int a, bool live,
                                                 unsigned mask) {
  V piv = V(1);
#pragma unroll
  for (int c = 0; c < B; ++c)
    if (a == c) piv = Dc[c];
  const V rpiv = V(1) / piv;
  const bool rfin = isfinite(rpiv);
#pragma unroll
  for (int c = 0; c < B; ++c) {
    if (a == c) {
      if (rfin) {
        const V q = acc * rpiv;
        acc = fma_rn(fma_rn(-q, piv, acc), rpiv, q);
      } else {
        acc = acc / piv;
      }
    }
    const V vc = __shfl_sync(mask, acc, c, FV_LG);
    if (live && a > c) acc -= Dc[c] * vc;
  }
  return acc;
}

// Forward sweep of one level of the transposed solve, U^T z = r: block row i of U^T takes the
// blocks (j, i) of U, j < i (positions tptr[i] .. tdiag[i] of the transpose, ascending j), row a
// of each transposed block (column a of the block of U) for lane a, then the in-block lower solve
// with D^T -- the operations and their order of the reference's transposed solve.
template <class V, int B, int M>
__global__ void k_ilu_upper_t_lg(IluView<V> F, const int* tptr, const int* tidx, const int* tdiag,
                                 const V* tval, const int* rows, int count, int ask, const V* r,
                                 V* z) {
  if (early(M)) next_level_may_start();
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  constexpr long BB = (long)B * B;
  const int q0 = tptr[i], di = tdiag[i];
  ask_blocks<V, B>(tval, q0, di - q0 + 1, a, ask);
  if (early(M)) wait_level_before();
  V acc = live ? r[(long)i * B + a] : V(0);
  acc = subtract_blocks<V, B, 1, M>(acc, tval, tidx, z, q0, di - q0, a, live, mask);
  V Dc[B];  // Dc[c] = D(c, a): row a of D^T
  if (live) load_seg<B>(tval + (long)di * BB + (long)a * B, Dc);
  else
#pragma unroll
    for (int c = 0; c < B; ++c) Dc[c] = V(0);
  acc = lower_t_block_solve<V, B>(acc, Dc, a, live, mask);
  if (live) z[(long)i * B + a] = acc;
}

// Backward sweep of one level of the transposed solve, L^T x = z (unit diagonal): the blocks
// (k, i) of L, k > i (positions tptr[i + 1] - 1 down to tdiag[i] + 1), then the in-block unit
// upper solve.
template <class V, int B, int M>
__global__ void k_ilu_lower_t_lg(IluView<V> F, const int* tptr, const int* tidx, const int* tdiag,
                                 const V* tval, const int* rows, int count, int ask, V* x) {
  if (early(M)) next_level_may_start();
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / FV_LG;
  const int a = threadIdx.x & (FV_LG - 1);
  if (gid >= count) return;
  const unsigned mask = lg_mask();
  const int i = rows[gid];
  const bool live = a < B;
  constexpr long BB = (long)B * B;
  const int di = tdiag[i], last = tptr[i + 1] - 1;
  ask_blocks<V, B>(tval, di, last - di + 1, a, ask);
  if (early(M)) wait_level_before();
  V acc = live ? x[(long)i * B + a] : V(0);
  acc = subtract_blocks<V, B, -1, M>(acc, tval, tidx, x, last, last - di, a, live, mask);
  V Dc[B];
  if (live) load_seg<B>(tval + (long)di * BB + (long)a * B, Dc);
  else
#pragma unroll
    for (int c = 0; c < B; ++c) Dc[c] = V(0);
#pragma unroll
  for (int c = B - 1; c >= 0; --c) {
    const V vc = __shfl_sync(mask, acc, c, FV_LG);
    if (live && a < c) acc -= Dc[c] * vc;
  }
  if (live) x[(long)i * B + a] = acc;
}

// ---- fp32 levels of few rows: a warp per block row, its blocks in shared memory.
// Such a level's time is its longest row's chain, and a coarse Galerkin row holds 15 to 40 blocks:
// with 8 lanes a row the chain paid a memory latency or two every few blocks (10 level sets of 720
// rows: 6 us each).  Here a row's columns, blocks, diagonal block and, going forward, right-hand side
// are in place before the level before is waited for; all its x entries then come in one round of
// loads, a block's by a lane, and what is left is the subtractions one after the other: 2 us a level
// set.  fp32 V-cycle of the 128 x 96 x 96 channel 2083 -> 1868 us, of 40^3 cells 607 -> 345.
// The line (sweep_rows) lies where the lanes run out instead of a row's chain.  A warp's time over the
// lane groups', level sets of rows of 2 / 13 blocks before the diagonal one, forward:
//   from L2      b = 2  3,500 rows 0.86 / 0.85, 5,500 1.03 / 0.92, 8,000 1.44 / 1.25
//                b = 4  3,500 rows 0.92 / 0.84, 5,500 1.03 / 0.78, 8,000 1.44
//                b = 5  2,000 rows 0.88 / 0.92, 3,500 1.08 / 1.06
//                b = 8  2,000 rows 0.94, 3,500 1.04, 5,500 0.99
//   from memory  b = 4  3,500 rows 0.78 / 0.63, 5,500 0.98 / 0.76, 8,000 1.66 / 1.26
//                b = 5  5,500 rows 1.03 / 1.06, 8,000 1.08 / 1.14, of scattered rows 0.79 / 0.89
//                b = 7  3,500 rows 0.90 / 0.86, 5,500 1.06 / 1.00, 8,000 1.19 / 1.13, scattered 1.08 / 0.89
//                b = 8  3,500 rows 0.94 / 0.86, 5,500 1.02 / 0.97, 8,000 1.45 / 1.40
// Scattered rows (a grid's own order) cost the lane groups more: solves on a 96^3 grid, lines at 4,608
// and at 8,192 rows, b = 2 1,216 / 1,105 us; at 6,144 and 8,192, b = 6 1,523 / 1,452, b = 4 1,382 / 1,407,
// and at 5,120 and 8,192, b = 8 1,829 / 2,045.
// The operations and their order are the lane-group kernels'.
enum { kLower, kLowerUpper, kUpper, kUpperT, kLowerT };
constexpr int sweep_rows(int b, long traffic, bool scattered) {
  constexpr int l2[9] = {0, 0, 4608, 4608, 5120, 2560, 5120, 1536, 4096};
  constexpr int memory[9] = {0, 0, 6144, 8192, 6144, 8192, 6144, 7168, 5120};
  constexpr int l2_far[9] = {0, 0, 7168, 7168, 6144, 3584, 7168, 3072, 4096};
  constexpr int memory_far[9] = {0, 0, 7168, 8192, 6144, 8192, 7168, 8192, 5120};
  if (scattered) return traffic >= 160000000 ? memory_far[b] : l2_far[b];
  return traffic >= 160000000 ? memory[b] : l2[b];
}

constexpr int kSweepBlocks = 32;  // blocks in shared memory at a time: a column a lane
template <int B>
__host__ __device__ constexpr int sweep_warp_entries(int cap) {
  return (cap * B * (B + 1) + 3) / 4 * 4;
}

// x is written by other blocks while this one runs: read past the L1 cache
template <int B>
__device__ __forceinline__ void load_x(const float* p, float (&o)[B]) {
  if constexpr (B % 4 == 0) {
#pragma unroll
    for (int k = 0; k < B / 4; ++k) {
      const float4 t = __ldcg(reinterpret_cast<const float4*>(p) + k);
      o[4 * k] = t.x;
      o[4 * k + 1] = t.y;
      o[4 * k + 2] = t.z;
      o[4 * k + 3] = t.w;
    }
  } else if constexpr (B % 2 == 0) {
#pragma unroll
    for (int k = 0; k < B / 2; ++k) {
      const float2 t = __ldcg(reinterpret_cast<const float2*>(p) + k);
      o[2 * k] = t.x;
      o[2 * k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < B; ++k) o[k] = __ldcg(p + k);
  }
}

// ptr / idx / diag / val: the factor's, or the transpose map's and its transposed blocks; cap: the
// most blocks of a row beside its diagonal, at most kSweepBlocks.
template <int B, int MODE>
__global__ void __launch_bounds__(128) k_ilu_sweep_w(const int* ptr, const int* idx,
                                                     const int* diag, const float* val,
                                                     const int* rows, int count, int cap,
                                                     const float* r, float* x) {
  constexpr int BB = B * B;
  constexpr bool kAfter = MODE == kUpper || MODE == kLowerT;  // the blocks after the diagonal one
  constexpr bool kDown = MODE == kLowerT;                     // from the last
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  next_level_may_start();
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x / 32) + warp;
  if (w >= count) return;  // whole warps exit together
  float* blk = (float*)sweep_smem + (long)warp * sweep_warp_entries<B>(cap);
  float* xs = blk + cap * BB;
  const int i = rows[w], di = diag[i];
  const int first = kAfter ? di + 1 : ptr[i], n = (kAfter ? ptr[i + 1] : di) - first;
  const int a = lane & (FV_LG - 1), al = a < B ? a : 0;
  const bool live = a < B;
  int col = 0;
  // blocks k0 .. k0 + m of the row's order, and the lane's column
  auto stage = [&](int k0, int m) {
    const int q = kDown ? first + n - k0 - m : first + k0;
    if (lane < m) col = idx[kDown ? q + m - 1 - lane : q + lane];
    const float* p = val + (long)q * BB;
    if constexpr (BB % 4 == 0) {
#pragma unroll 4
      for (int e = lane; e < m * (BB / 4); e += 32)
        reinterpret_cast<float4*>(blk)[e] = reinterpret_cast<const float4*>(p)[e];
    } else {
#pragma unroll 4
      for (int e = lane; e < m * BB; e += 32) blk[e] = p[e];
    }
  };
  stage(0, min(n, cap));
  float D[B], acc = 0.0f;
  load_seg<B>(val + (long)di * BB + al * B, D);
  if (!kAfter) acc = __ldcg(r + (long)i * B + al);
  wait_level_before();
  if (kAfter) acc = __ldcg(x + (long)i * B + al);
  for (int k0 = 0; k0 < n; k0 += cap) {
    const int m = min(n - k0, cap);
    if (k0) {
      __syncwarp();  // (the blocks before have been used)
      stage(k0, m);
    }
    if (lane < m) {
      float t[B];
      load_x<B>(x + (long)col * B, t);
#pragma unroll
      for (int c = 0; c < B; ++c) xs[lane * B + c] = t[c];
    }
    __syncwarp();
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      float L[B], xj[B];
      load_seg<B>(blk + (kDown ? m - 1 - k : k) * BB + al * B, L);
      load_seg<B>(xs + k * B, xj);
#pragma unroll
      for (int c = 0; c < B; ++c) {
        const int e = kDown ? B - 1 - c : c;
        acc -= L[e] * xj[e];
      }
    }
  }
  const unsigned mask = 0xffffffffu;
  if constexpr (MODE == kLower || MODE == kLowerUpper) {
#pragma unroll
    for (int c = 0; c < B; ++c) {
      const float vc = __shfl_sync(mask, acc, c, FV_LG);
      if (live && a > c) acc -= D[c] * vc;
    }
  }
  if constexpr (MODE == kUpper || MODE == kLowerUpper)
    acc = upper_block_solve<float, B>(acc, D, a, live, mask);
  if constexpr (MODE == kUpperT) acc = lower_t_block_solve<float, B>(acc, D, a, live, mask);
  if constexpr (MODE == kLowerT) {
#pragma unroll
    for (int c = B - 1; c >= 0; --c) {
      const float vc = __shfl_sync(mask, acc, c, FV_LG);
      if (live && a < c) acc -= D[c] * vc;
    }
  }
  if (lane < B) x[(long)i * B + lane] = acc;
}

// fp32 y = A x or, RES, rhs - A x of few block rows: a warp per row as above, which pays the
// memory's latency once a row instead of once a block; k_bsr_spmv_b's operations in its order.
// b = 6, coarse Galerkin rows: 5,370 of them, 17 blocks a row, 26 at most, 15.0 -> 8.3 us (7.5 ->
// 6.5 from L2), 212 of them 13.6 -> 4.3 (6.0 -> 2.8).
// The other kernel's time is its longest row's chain, this one's the warps' work as soon as they no
// longer run side by side: its line is in rows of the longest's length (warp_product).  This one's
// time over the other's, from L2 / from memory:
//   b = 2  grids of 5 blocks a row  3,025 rows 0.89 / 0.96, 5,184 0.95 / 0.98, 6,400 1.03 / 0.80
//          7  3,375 rows 0.88 / 0.74, 5,832 0.96 / 0.92, 8,000 1.24 / 1.00;  27  8,000 1.00 / 0.79
//   b = 4  5  2,025 rows 0.88 / 1.00, 4,096 0.98 / 1.00, 6,400 1.12 / 0.97
//          7  2,744 rows 0.96 / 0.98, 4,096 1.05 / 0.80, 5,832 1.10 / 0.80
//         27  4,096 rows 0.83 / 0.60, 5,832 0.96 / 0.74, 8,000 1.26 / 0.87
//             (20, at random columns, from L2: 3,000 rows 0.89, 5,000 1.12)
//   b = 6  5  2,025 rows 0.83 / 0.82, 4,096 1.01 / 0.80, 6,400 1.39 / 1.00
//          7  2,744 rows 0.94 / 0.80, 4,096 1.08 / 0.81, 6,859 1.40 / 1.03
//         27  3,375 rows 0.89 / 0.60, 4,913 1.11 / 0.70, 5,832 1.22 / 0.81
//   b = 8  5  2,025 rows 0.95 / 0.80, 4,096 1.45 / 1.23;  7  2,197 rows 1.03 / 0.81, 4,096 1.52 / 1.20
//         27  2,197 rows 0.97 / 0.66, 4,096 1.47 / 0.90, 4,913 1.91 / 1.09
// traffic: the bytes between two products (0: not known, as from L2).
inline bool warp_product(int rows, int b, long nnzb, int longest, long traffic) {
  if (traffic >= 100000000) return rows < (b == 8 ? 3584 : b == 7 ? 4608 : 6144);
  constexpr int few[9] = {0, 0, 5000, 2500, 3000, 2500, 3000, 1800, 2000};  // blocks a row: below 7,
  constexpr int some[9] = {0, 0, 6000, 3600, 3700, 3200, 3400, 2300, 1900};  // to 13,
  constexpr int many[9] = {0, 0, 6500, 5500, 4600, 4400, 3900, 3000, 2000};  // more
  if (nnzb <= 0) return rows < few[b];  // (unknown)
  if (longest <= 0) longest = (int)((nnzb + rows - 1) / rows);
  const int line = longest < 7 ? few[b] : longest < 14 ? some[b] : many[b];
  return nnzb < (long)line * longest;
}
template <int B, bool RES>
__global__ void __launch_bounds__(128) k_bsr_spmv_w(int nbr, const int* __restrict__ ptr,
                                                    const int* __restrict__ idx,
                                                    const float* __restrict__ val,
                                                    const float* __restrict__ x,
                                                    const float* __restrict__ rhs, float* y) {
  constexpr int BB = B * B;
  __shared__ __align__(16) float smem[4 * sweep_warp_entries<B>(kSweepBlocks)];
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + warp;
  if (i >= nbr) return;  // whole warps exit together
  float* blk = smem + warp * sweep_warp_entries<B>(kSweepBlocks);
  float* xs = blk + kSweepBlocks * BB;
  const int q0 = ptr[i], n = ptr[i + 1] - q0, al = lane < B ? lane : 0;
  const float own = RES ? rhs[(long)i * B + al] : 0.0f;
  float acc = 0.0f;
  for (int k0 = 0; k0 < n; k0 += kSweepBlocks) {
    const int m = min(n - k0, kSweepBlocks);
    __syncwarp();  // (the blocks before have been used)
    const float* p = val + (long)(q0 + k0) * BB;
    if constexpr (BB % 4 == 0) {
#pragma unroll 4
      for (int e = lane; e < m * (BB / 4); e += 32)
        reinterpret_cast<float4*>(blk)[e] = reinterpret_cast<const float4*>(p)[e];
    } else {
#pragma unroll 4
      for (int e = lane; e < m * BB; e += 32) blk[e] = p[e];
    }
    if (lane < m) {
      float t[B];
      load_seg<B>(x + (long)idx[q0 + k0 + lane] * B, t);
#pragma unroll
      for (int c = 0; c < B; ++c) xs[lane * B + c] = t[c];
    }
    __syncwarp();
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      float L[B], xj[B];
      load_seg<B>(blk + k * BB + al * B, L);
      load_seg<B>(xs + k * B, xj);
#pragma unroll
      for (int c = 0; c < B; ++c) acc += L[c] * xj[c];
    }
  }
  if (lane < B) y[(long)i * B + lane] = RES ? own - acc : acc;
}

// What a caller knows of a product's pattern and use: its blocks, the longest row's, and the bytes
// that pass between two products (0: not known).
struct ProductHint {
  long nnzb = 0;
  int longest = 0;
  long traffic = 0;
};

// y = A x, or rhs - A x with RES, where the alignment allows vector loads (2 <= b <= 8)
template <class V, bool RES>
void launch_spmv_b(int nbr, int b, const ProductHint& hint, const int* indptr, const int* indices,
                   const V* values, const V* x, const V* rhs, V* y, cudaStream_t s) {
  with_block_size(b, [&](auto B) {
    if constexpr (sizeof(V) == 4) {
      if (warp_product(nbr, b, hint.nnzb, hint.longest, hint.traffic)) {
        k_bsr_spmv_w<B(), RES><<<fv_blocks(nbr, 4), 128, 0, s>>>(nbr, indptr, indices, values, x,
                                                                 rhs, y);
        return;
      }
    }
    k_bsr_spmv_b<V, B(), RES><<<fv_blocks((long)nbr * b, kThreads), kThreads, 0, s>>>(
        nbr, indptr, indices, values, x, rhs, y);
  });
}

#include "ilu_narrow.inc.cuh"

template <class V>
__global__ void k_copy(long n, const V* a, V* b) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}
__global__ void k_to_f32(long n, const double* a, float* b) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

// ------------------------------------------------------------------------------ reductions
constexpr int kRedBlocks = 304;  // 2 x 152 SMs, fixed so the summation order never changes
__global__ void k_dot_partial(long n, const double* x, const double* y, double* part) {
  __shared__ double sh[kThreads];
  double s = 0.0;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    s += x[i] * y[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}
__global__ void k_dot_final(int nparts, const double* part, double* out) {
  __shared__ double sh[kThreads];
  double s = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

double* g_dot_parts = nullptr;

}  // namespace

// ------------------------------------------------------------------------------ FvIlu0
struct FvIlu0 {
  int n = 0, b = 0, nnzb = 0, precision = 64;
  int *ptr = nullptr, *idx = nullptr, *diag = nullptr;
  int *tptr = nullptr, *tidx = nullptr, *tblk = nullptr;
  int* tdiag = nullptr;   // position of the diagonal block in each row of the transpose
  void* val = nullptr;
  void* rp = nullptr;     // (n * b) reciprocals of the factor's pivots
  int row_cap = 0;        // most blocks in a row
  std::vector<int> lv_cap, lv_low;  // ... of each forward level, and most lower blocks
  std::vector<long> lv_sum;         // ... and its lower blocks together
  std::vector<char> lv_scattered;   // ... and whether its rows do not lie beside each other
  bool scattered = false;           // most rows are in such a level
  cudaStream_t side = nullptr;  // of fv_ilu0_factor_start
  bool open = false;            // started, not finished: the factor belongs to `side`
  cudaEvent_t side_event = nullptr;
  void* tval = nullptr;   // (b > 1) the factor's blocks transposed, in the transpose's order
  unsigned long long* zero_flag = nullptr;
  // level sets: rows grouped by level (device), level boundaries (host)
  int* rows_fwd = nullptr;   // L / factor order
  int* rows_bwd = nullptr;   // U order (from the last row)
  int* rows_tfwd = nullptr;  // U^T order
  int* rows_tbwd = nullptr;  // L^T order
  std::vector<int> lv_fwd, lv_bwd, lv_tfwd, lv_tbwd;
  void* work = nullptr;                      // (n * b) vector the captured sweeps run on
  long traffic = 0;  // bytes read between two reads of a block (fv_ilu0_set_traffic)
  // (b > 1) narrow level sets: the forward / transposed solve as one launch (ilu_narrow.inc.cuh)
  struct Run {
    int4* row = nullptr;    // 2n rows in level order, forward sweep then backward
    int4* col = nullptr;
    int* bounds = nullptr;  // nlev + 1 offsets into row / col
    void* rec = nullptr;    // records, renewed by each factorisation
    int nlev = 0, nlev_fwd = 0, widest = 0;
    int k = 0;              // blocks in a record, at most
    int most = 0;           // off-diagonal blocks of a row in a sweep, at most
  } run[2];
  bool fuse_fb = false;  // the last forward level's rows are the first backward level's (fused)
  cudaGraphExec_t apply_exec[2] = {nullptr, nullptr};  // forward / transposed solve
  cudaGraphExec_t factor_exec = nullptr;
  // host copy of the pattern (shared by clones): the transposed-solve structures are built on
  // first use
  std::shared_ptr<const std::vector<int>> h_ptr, h_idx, h_diag;
};

namespace {

// Level sets of a dependency DAG given as "row i depends on rows deps(i)".
template <class DepFn>
void levels(int n, bool ascending, DepFn deps, std::vector<int>* rows, std::vector<int>* bounds) {
  std::vector<int> lev(n, 0);
  int maxl = 0;
  if (ascending) {
    for (int i = 0; i < n; ++i) {
      int l = 0;
      deps(i, [&](int j) { l = std::max(l, lev[j] + 1); });
      lev[i] = l;
      maxl = std::max(maxl, l);
    }
  } else {
    for (int i = n - 1; i >= 0; --i) {
      int l = 0;
      deps(i, [&](int j) { l = std::max(l, lev[j] + 1); });
      lev[i] = l;
      maxl = std::max(maxl, l);
    }
  }
  bounds->assign(maxl + 2, 0);
  for (int i = 0; i < n; ++i) (*bounds)[lev[i] + 1]++;
  for (int l = 0; l <= maxl; ++l) (*bounds)[l + 1] += (*bounds)[l];
  rows->assign(n, 0);
  std::vector<int> fill(bounds->begin(), bounds->end() - 1);
  for (int i = 0; i < n; ++i) (*rows)[fill[lev[i]]++] = i;
}

template <class V>
IluView<V> view(FvIlu0* f) {
  return IluView<V>{f->n, f->b, f->ptr, f->idx, f->diag, (V*)f->val};
}

int upload_bytes(const void* h, size_t bytes, void** d, cudaStream_t s) {
  FV_CUDA_TRY(cudaMalloc(d, std::max<size_t>(1, bytes)));
  if (bytes) FV_CUDA_TRY(cudaMemcpyAsync(*d, h, bytes, cudaMemcpyHostToDevice, s));
  return FV_OK;
}

int widest(const std::vector<int>& bounds) {
  int w = 0;
  for (size_t l = 0; l + 1 < bounds.size(); ++l) w = std::max(w, bounds[l + 1] - bounds[l]);
  return w;
}

// The one-launch form of a solve (k_ilu_run), when every level set fits one block and the vector
// its shared memory (here in single precision; checked for the factor's in pack_run).  Above that a
// level has the rows to fill more SMs than one, a launch each: a 16-block cluster that runs levels
// of 700 rows, the vector in global memory, took 135 us a solve against 114 (128 x 96 x 96 channel,
// 20 levels, 15-27 blocks a row).  `row` gives a forward (0) /
// backward (1) row as RunView::row; a backward row's blocks are taken upwards (step 1) or down.
template <class RowFn>
int build_run(FvIlu0* f, int t, const std::vector<int>& fwd, const std::vector<int>& lv_fwd,
              const std::vector<int>& bwd, const std::vector<int>& lv_bwd, const int* idx,
              int back_step, RowFn row, cudaStream_t s) {
  const int nf = (int)lv_fwd.size() - 1, nb = (int)lv_bwd.size() - 1;
  FvIlu0::Run& run = f->run[t];
  run.widest = std::max(widest(lv_fwd), widest(lv_bwd));
  if (!run_block_size(f->b, sizeof(float)) || run.widest > run_capacity(f->b) ||
      run_smem_bytes(f->n, f->b, nf + nb, sizeof(float)) > kRunSmem)
    return FV_OK;
  std::vector<int4> rows, cols;
  for (int back = 0; back < 2; ++back)
    for (int i : back ? bwd : fwd) {
      const int4 d = row(back, i);
      int c[kRunBlocks] = {0, 0, 0, 0};
      for (int q = 0; q < kRunBlocks && q < d.y; ++q)
        c[q] = idx[d.z + (back ? back_step : 1) * q] * f->b;
      rows.push_back(d);
      cols.push_back(make_int4(c[0], c[1], c[2], c[3]));
      run.k = std::max(run.k, std::min(d.y, kRunBlocks));
      run.most = std::max(run.most, d.y);
    }
  std::vector<int> bounds(lv_fwd);
  for (int l = 1; l <= nb; ++l) bounds.push_back(f->n + lv_bwd[l]);
  run.nlev = nf + nb;
  run.nlev_fwd = nf;
  if (upload_bytes(rows.data(), sizeof(int4) * rows.size(), (void**)&run.row, s) ||
      upload_bytes(cols.data(), sizeof(int4) * cols.size(), (void**)&run.col, s) ||
      upload_bytes(bounds.data(), sizeof(int) * bounds.size(), (void**)&run.bounds, s))
    return FV_ERR_CUDA;
  FV_CUDA_TRY(cudaStreamSynchronize(s));  // the host copies end with this call
  return FV_OK;
}

// The records of a one-launch solve from the present factor.
template <class V>
int pack_run(FvIlu0* f, int t, cudaStream_t s) {
  FvIlu0::Run& run = f->run[t];
  // fp32 rows of more blocks than the records hold go by k_ilu_sweep_w, which has all of them in
  // place (212 coarse rows of 20 to 40 blocks: 22 us a solve, 40 us by k_ilu_run)
  if (!run.row || !run_block_size(f->b, sizeof(V)) ||
      (sizeof(V) == 8 && 2L * f->n > (long)run_mean64(f->b, run.most, t != 0) * run.nlev) ||
      run_smem_bytes(f->n, f->b, run.nlev, sizeof(V)) > kRunSmem ||
      (sizeof(V) == 4 && f->row_cap > 2 * kRunBlocks + 1))
    return FV_OK;
  const long lanes = 2L * f->n * run_lanes(f->b);
  if (!run.rec) FV_CUDA_TRY(cudaMalloc(&run.rec, sizeof(V) * lanes * run_entries(f->b, run.k)));
  k_run_pack<V><<<fv_blocks(lanes, kThreads), kThreads, 0, s>>>(
      f->n, f->b, run.k, t != 0, run.row, t ? (const V*)f->tval : (const V*)f->val, (V*)run.rec);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

inline bool runs(const FvIlu0* f, int t) { return f->run[t].rec != nullptr; }

template <class V>
int launch_run(FvIlu0* f, int t, const V* r, V* x, cudaStream_t s) {
  const FvIlu0::Run& run = f->run[t];
  const RunView<V> R{f->n,   run.nlev, run.nlev_fwd,        run.k,
                     run.bounds, run.row, run.col,          (const V*)run.rec,
                     t ? f->tidx : f->idx, t ? (const V*)f->tval : (const V*)f->val};
  int rc = FV_OK;
  with_block_size(f->b, [&](auto B) {
    rc = launch_run_b<V, B()>(R, run.widest, t != 0, r, x, s);
  });
  return rc;
}

// A level's kernel; `after` says that the launch before it on the stream is a level's too.
template <class K, class... Args>
void launch_level(K kern, int grid, cudaStream_t s, bool after, int threads, size_t smem,
                  Args... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = after ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, args...);
}

// Launch the level sequence of the factorization / a solve on `s` (captured into a graph once).
template <class V>
void launch_factor_levels(FvIlu0* f, cudaStream_t s) {
  IluView<V> F = view<V>(f);
  const int bb = f->b * f->b;
  auto lane_groups = [&](size_t l) {
    const int cnt = f->lv_fwd[l + 1] - f->lv_fwd[l], low = f->lv_low[l];
    if (factor_warp_bytes<V>(f->lv_cap[l], bb) > kFactorSmem) return true;
    const bool far = f->lv_scattered[l];
    if (sizeof(V) == 8) return cnt >= factor_wide64(f->b, low, far);
    const long line = factor_wide(f->b, low, far);
    return low ? f->lv_sum[l] >= line * low : cnt >= line;
  };
  bool warps = false;  // a level takes warps, which read the pivots' reciprocals
  for (size_t l = 0; l + 1 < f->lv_fwd.size(); ++l) warps = warps || !lane_groups(l);
  bool after = false;  // the launch before on `s` lets this one start early
  for (size_t l = 0; l + 1 < f->lv_fwd.size(); ++l) {
    const int cnt = f->lv_fwd[l + 1] - f->lv_fwd[l];
    if (cnt == 0) continue;
    const bool early = after && (sizeof(V) == 4 || cnt <= kEarly64);
    after = false;
    if (f->b == 1) {
      k_ilu_factor_level<V><<<fv_blocks(cnt, 128), 128, 0, s>>>(F, f->rows_fwd + f->lv_fwd[l], cnt,
                                                                f->zero_flag);
      continue;
    }
    // a level with a row of hundreds of blocks takes lane groups too, which hold no row, and keeps
    // the other levels to itself (96 x 96 grid, fp64: b = 6 3.1 ms, 4.1 with the first cell coupled
    // to 400 more and 34.9 with every level at a thread a row then; b = 8 4.8, 6.5, 87)
    if (lane_groups(l)) {
      with_block_size(f->b, [&](auto B) {
        k_ilu_factor_lgb<V, B()><<<fv_blocks((long)cnt * FV_LG, 128), 128, 0, s>>>(
            F, f->rows_fwd + f->lv_fwd[l], cnt, warps ? (V*)f->rp : nullptr, f->zero_flag);
      });
      continue;
    }
    const size_t wb = factor_warp_bytes<V>(f->lv_cap[l], bb);
    // a level that leaves SMs idle: a warp per block, so that no two share an SM's fp64 issue
    const int warps = cnt <= 4 * 152 || 4 * wb > kFactorSmem ? 1 : 4;
    with_block_size(f->b, [&](auto B) {
      auto kern = k_ilu_factor_w<V, B()>;
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFactorSmem);
      launch_level(kern, fv_blocks(cnt, warps), s, early, 32 * warps, warps * wb, F,
                   (const int*)f->rows_fwd + f->lv_fwd[l], cnt, f->lv_cap[l], (V*)f->rp,
                   f->zero_flag);
    });
    after = sizeof(V) == 4 || cnt <= kEarly64;
  }
}

// How a level's lane groups read, by rows and block size, and by the bytes that pass between two
// solves (traffic): from about the L2 cache's 126 MB on, its blocks come from memory.
// * A level of few rows is its rows' chain of latencies: the next one is launched early.  fp64 to
//   1,024 rows (above, its blocks would be placed around a level that fp64 issue still binds: 6,000
//   rows 1.1 to 1.4 times the time), fp32 to 32,768, odd block sizes, whose loads are scalar, to
//   8,192.  kEarly / kPlain / the form with neither request nor early launch, 6 level sets, fp64,
//   us: 512 rows, 14 blocks, b = 3 92 / 99 / 99.5, b = 6 134 / 146 / 144; 97 rows, 2 blocks, b = 4
//   58 / 64 / 65.
// * From memory: two blocks at a time and all of a row's lines asked for (V-cycle of 64^3 cells,
//   fp64, b = 6, its small levels 3,240 -> 3,150 us; fp32 80^3, levels of 14,000 rows 966 -> 943,
//   22 x 96 x 21, a cycle of 113 MB, levels of 22,000 289 -> 283; but 128 x 96 x 96, 30,000 rows
//   1,747 / 1,740, and from L2 4 to 28 % slower for b of 2, 3, 5 and 7).
//   fp32 of odd b so, over kPlain's time, from memory: 9,000 to 14,000 rows of 2 blocks before the
//   diagonal one b = 3 0.79 to 0.90, b = 5 0.85 to 1.06, b = 7 0.97 to 1.09, of 13 blocks 0.99 to
//   1.25; 20,000 rows 0.83 to 1.02; 28,000 0.83 to 1.28, 40,000 and 60,000 0.96 to 1.14 (solves on
//   a 150^3 grid, b = 3, transposed, 3,008 -> 2,666 us, b = 5 3,593 -> 3,344).
//   So, too, the transposed fp64 levels of few short rows of b = 2 and 3 (300 x 200 cells, b = 3, a
//   transposed V-cycle 6,016 -> 5,830 us; 29 blocks a row, b = 3, 511 rows 97 us, kEarly 86).
// * The cache is asked for a row's first KB, a line a lane; for all of a row where it is long in
//   bytes and from memory or early (V-cycles, fp64, b = 6: 50^3 2,067 -> 2,024 us, 24^3 680 -> 661;
//   late and from L2 6,000 rows of 14 blocks 1 to 9 % slower).
// * The widest are bound by bytes and want warps in flight (590,000 rows, b = 6: 120 us one block
//   at a time, 180-220 with the registers of a deeper read; 500,000 rows, b = 4 0.78 of kPlain's
//   time, b = 6 0.92), but for the block sizes with scalar or 8-byte loads, which the compiler's
//   unrolling serves better (b = 2, 16 blocks 71 / 83 us at 131,072 rows).
inline int level_read(bool fp32, int b, int rows, int longest, long traffic, bool transposed) {
  const bool wide_loads = b % 2 == 0 && b > 2;
  if (!fp32) {
    if (rows < 512 && (wide_loads ? traffic >= 160000000 : transposed && b <= 3 && longest <= 16))
      return kDeep;
    return rows <= 1024 ? kEarly : kPlain;
  }
  if (rows < 8192) return kEarly;
  if (rows >= 65536) return wide_loads ? kStream : kPlain;
  if (b % 2 != 0)
    return traffic >= 160000000 && rows < 24576 && (rows >= 16384 || (b < 7 && longest <= 9))
               ? kDeep : kPlain;
  if (traffic >= 100000000 && wide_loads && rows < 24576) return kDeep;
  return rows < 32768 ? kEarly : wide_loads ? kStream : kPlain;
}

template <class V>
void launch_apply_levels(FvIlu0* f, int transpose, const V* r, V* x, cudaStream_t s) {
  IluView<V> F = view<V>(f);
  const bool lg = f->b > 1;
  bool after = false;  // the launch before on `s` is a level of this solve
  auto levels_of = [&](const std::vector<int>& lv, const int* order, size_t first, auto&& one) {
    for (size_t l = first; l + 1 < lv.size(); ++l) {
      const int cnt = lv[l + 1] - lv[l];
      if (!cnt) continue;
      one(l, order + lv[l], cnt);
      after = true;
    }
  };
  // the lane-group kernels of a level, by block size and reading
  auto lane_groups = [&](int cnt, auto&& launch) {
    const int grid = fv_blocks((long)cnt * FV_LG, 128);
    const int read = level_read(sizeof(V) == 4, f->b, cnt, f->row_cap, f->traffic, transpose != 0);
    const bool all = read == kDeep ||
                     (sizeof(V) == 8 && (read == kEarly || f->traffic >= 160000000));
    const int ask = all ? INT_MAX : 1024;
    with_block_size(f->b, [&](auto B) {
      if (read == kPlain) launch(B, std::integral_constant<int, kPlain>{}, grid, ask);
      if (read == kEarly) launch(B, std::integral_constant<int, kEarly>{}, grid, ask);
      if constexpr (sizeof(V) == 8 ? B() % 2 == 0 || B() == 3 : B() != 2)
        if (read == kDeep) launch(B, std::integral_constant<int, kDeep>{}, grid, ask);
      if constexpr (B() % 2 == 0 && B() > 2 && sizeof(V) == 4)
        if (read == kStream) launch(B, std::integral_constant<int, kStream>{}, grid, ask);
    });
  };
  // an fp32 level of few rows by k_ilu_sweep_w; false: not one
  auto warp_rows = [&](auto mode, const int* rows, int cnt) {
    if constexpr (sizeof(V) == 4) {
      if (cnt >= sweep_rows(f->b, f->traffic, f->scattered)) return false;
      const bool T = mode() == kUpperT || mode() == kLowerT;
      const int cap = std::max(1, std::min(f->row_cap - 1, kSweepBlocks));
      with_block_size(f->b, [&](auto B) {
        launch_level(k_ilu_sweep_w<B(), mode()>, fv_blocks(cnt, 4), s, after, 128,
                     4 * sizeof(float) * sweep_warp_entries<B()>(cap), T ? (const int*)f->tptr : F.ptr,
                     T ? (const int*)f->tidx : F.idx, T ? (const int*)f->tdiag : F.diag,
                     T ? (const float*)f->tval : (const float*)F.val, rows, cnt, cap, r, x);
      });
      return true;
    } else {
      return false;
    }
  };
  const V* tval = (const V*)f->tval;
  if (!transpose) {
    const size_t last = f->lv_fwd.size() - 2;
    levels_of(f->lv_fwd, f->rows_fwd, 0, [&](size_t l, const int* rows, int cnt) {
      if (!lg) {
        k_ilu_lower<V><<<fv_blocks(cnt, 128), 128, 0, s>>>(F, rows, cnt, r, x);
        return;
      }
      if (f->fuse_fb && l == last ? warp_rows(std::integral_constant<int, kLowerUpper>{}, rows, cnt)
                                  : warp_rows(std::integral_constant<int, kLower>{}, rows, cnt))
        return;
      lane_groups(cnt, [&](auto B, auto M, int grid, int ask) {
        if (f->fuse_fb && l == last)
          launch_level(k_ilu_lower_upper_lg<V, B(), M()>, grid, s, after && early(M()), 128, 0,
                       F, rows, cnt, ask, r, x);
        else
          launch_level(k_ilu_lower_lg<V, B(), M()>, grid, s, after && early(M()), 128, 0,
                       F, rows, cnt, ask, r, x);
      });
    });
    levels_of(f->lv_bwd, f->rows_bwd, f->fuse_fb ? 1 : 0, [&](size_t, const int* rows, int cnt) {
      if (!lg) {
        k_ilu_upper<V><<<fv_blocks(cnt, 128), 128, 0, s>>>(F, rows, cnt, x);
        return;
      }
      if (warp_rows(std::integral_constant<int, kUpper>{}, rows, cnt)) return;
      lane_groups(cnt, [&](auto B, auto M, int grid, int ask) {
        launch_level(k_ilu_upper_lg<V, B(), M()>, grid, s, after && early(M()), 128, 0,
                     F, rows, cnt, ask, x);
      });
    });
  } else {
    levels_of(f->lv_tfwd, f->rows_tfwd, 0, [&](size_t, const int* rows, int cnt) {
      if (!lg) {
        k_ilu_upper_t<V><<<fv_blocks(cnt, 128), 128, 0, s>>>(F, f->tptr, f->tidx, f->tblk, rows,
                                                             cnt, r, x);
        return;
      }
      if (warp_rows(std::integral_constant<int, kUpperT>{}, rows, cnt)) return;
      lane_groups(cnt, [&](auto B, auto M, int grid, int ask) {
        launch_level(k_ilu_upper_t_lg<V, B(), M()>, grid, s, after && early(M()), 128, 0,
                     F, f->tptr, f->tidx, f->tdiag, tval, rows, cnt, ask, r, x);
      });
    });
    levels_of(f->lv_tbwd, f->rows_tbwd, 0, [&](size_t, const int* rows, int cnt) {
      if (!lg) {
        k_ilu_lower_t<V><<<fv_blocks(cnt, 128), 128, 0, s>>>(F, f->tptr, f->tidx, f->tblk, rows,
                                                             cnt, x);
        return;
      }
      if (warp_rows(std::integral_constant<int, kLowerT>{}, rows, cnt)) return;
      lane_groups(cnt, [&](auto B, auto M, int grid, int ask) {
        launch_level(k_ilu_lower_t_lg<V, B(), M()>, grid, s, after && early(M()), 128, 0,
                     F, f->tptr, f->tidx, f->tdiag, tval, rows, cnt, ask, x);
      });
    });
  }
}

// Capture `body` (a sequence of launches on a stream) into an executable graph, on a private
// stream in thread-local capture mode so that a caller's own capture is unaffected.
template <class Body>
int capture(Body body, cudaGraphExec_t* out) {
  cudaStream_t cs;
  FV_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    body(cs);
    e = cudaStreamEndCapture(cs, &g);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(cs);
  if (e != cudaSuccess) {
    fv_set_error("ILU(0) graph capture failed: %s", cudaGetErrorString(e));
    return FV_ERR_CUDA;
  }
  return FV_OK;
}

template <class V>
int ilu_factor_start(FvIlu0* f, cudaStream_t s) {
  FV_CUDA_TRY(cudaMemsetAsync(f->zero_flag, 0xff, sizeof(unsigned long long), s));
  if (!f->factor_exec) {
    int rc = capture([&](cudaStream_t cs) { launch_factor_levels<V>(f, cs); }, &f->factor_exec);
    if (rc != FV_OK) return rc;
  }
  FV_CUDA_TRY(cudaGraphLaunch(f->factor_exec, s));
  if (f->tval) {  // a transposed solve was asked for: keep its transposed blocks current
    const long nv = (long)f->nnzb * f->b * f->b;
    k_transpose_blocks<V><<<fv_blocks(nv, kThreads), kThreads, 0, s>>>(f->nnzb, f->b, f->tblk,
                                                                      (const V*)f->val,
                                                                      (V*)f->tval);
  }
  for (int t = 0; t < 2; ++t)
    if (t == 0 || f->tval) {
      int rc = pack_run<V>(f, t, s);
      if (rc != FV_OK) return rc;
    }
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

int ilu_factor_finish(FvIlu0* f, cudaStream_t s) {
  unsigned long long flag;
  FV_CUDA_TRY(cudaMemcpyAsync(&flag, f->zero_flag, sizeof(flag), cudaMemcpyDeviceToHost, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  if (flag != ~0ull) {
    long col = (long)(flag & 0xffffffffull);
    fv_set_error_index(col);
    fv_set_error(
        "ILU(0) met an exactly zero pivot at row %ld; the operator needs a different ordering or "
        "an explicit shift, neither of which this routine applies silently.",
        col);
    return FV_ERR_ZERO_PIVOT;
  }
  return FV_OK;
}

int upload(const std::vector<int>& h, int** d, cudaStream_t s);

// The transposed-solve structures (the pattern's transpose and the level sets of U^T and L^T),
// built the first time a transposed solve is asked for.
int ensure_transpose(FvIlu0* f, cudaStream_t s) {
  if (f->tptr) return FV_OK;
  const int n = f->n;
  Transpose T;
  build_transpose(n, n, f->h_ptr->data(), f->h_idx->data(), &T);
  std::vector<int> rows, rows_fwd;
  levels(n, true, [&](int i, auto&& use) {  // U^T: column i depends on rows j < i with (j, i)
    for (int q = T.ptr[i]; q < T.ptr[i + 1]; ++q)
      if (T.idx[q] < i) use(T.idx[q]);
  }, &rows, &f->lv_tfwd);
  if (upload(rows, &f->rows_tfwd, s)) return FV_ERR_CUDA;
  rows_fwd = rows;
  levels(n, false, [&](int i, auto&& use) {  // L^T: column i depends on rows k > i with (k, i)
    for (int q = T.ptr[i]; q < T.ptr[i + 1]; ++q)
      if (T.idx[q] > i) use(T.idx[q]);
  }, &rows, &f->lv_tbwd);
  if (upload(rows, &f->rows_tbwd, s)) return FV_ERR_CUDA;
  if (upload(T.ptr, &f->tptr, s) || upload(T.idx, &f->tidx, s) || upload(T.blk, &f->tblk, s))
    return FV_ERR_CUDA;
  if (f->b > 1) {  // the lane-group sweeps read the factor's blocks transposed
    std::vector<int> td(n, -1);
    for (int i = 0; i < n; ++i)
      for (int q = T.ptr[i]; q < T.ptr[i + 1]; ++q)
        if (T.idx[q] == i) td[i] = q;
    if (upload(td, &f->tdiag, s)) return FV_ERR_CUDA;
    int rc = build_run(f, 1, rows_fwd, f->lv_tfwd, rows, f->lv_tbwd, T.idx.data(), -1,
                       [&](int back, int i) {
      return back ? make_int4(i, T.ptr[i + 1] - 1 - td[i], T.ptr[i + 1] - 1, td[i])
                  : make_int4(i, td[i] - T.ptr[i], T.ptr[i], td[i]);
    }, s);
    if (rc != FV_OK) return rc;
    const long nv = (long)f->nnzb * f->b * f->b;
    const size_t vs = f->precision == 64 ? sizeof(double) : sizeof(float);
    FV_CUDA_TRY(cudaMalloc(&f->tval, vs * (size_t)nv));
    if (f->precision == 64)
      k_transpose_blocks<double><<<fv_blocks(nv, kThreads), kThreads, 0, s>>>(
          f->nnzb, f->b, f->tblk, (const double*)f->val, (double*)f->tval);
    else
      k_transpose_blocks<float><<<fv_blocks(nv, kThreads), kThreads, 0, s>>>(
          f->nnzb, f->b, f->tblk, (const float*)f->val, (float*)f->tval);
    FV_CUDA_TRY(cudaGetLastError());
    rc = f->precision == 64 ? pack_run<double>(f, 1, s) : pack_run<float>(f, 1, s);
    if (rc != FV_OK) return rc;
  }
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  return FV_OK;
}

template <class V>
int ilu_apply(FvIlu0* f, const V* r, V* x, int transpose, cudaStream_t s) {
  const long n = (long)f->n * f->b;
  V* w = (V*)f->work;
  const int t = transpose ? 1 : 0;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FV_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  if (cap != cudaStreamCaptureStatusNone) {
    // inside a caller's stream capture (a whole V-cycle as one graph): the level kernels go
    // straight into the caller's graph; nothing is allocated or built here
    if (t && !f->tptr) {
      fv_set_error("fv_ilu0_apply: the transposed-solve structures are built by a transposed "
                   "solve outside stream capture first");
      return FV_ERR_ARG;
    }
    if ((uintptr_t)x % 16 != 0) {  // the level kernels read x's block segments as vectors
      fv_set_error("fv_ilu0_apply: under stream capture x must be 16-byte aligned");
      return FV_ERR_ARG;
    }
    if (runs(f, t)) return launch_run<V>(f, t, r, x, s);
    launch_apply_levels<V>(f, t, r, x, s);
    FV_CUDA_TRY(cudaGetLastError());
    return FV_OK;
  }
  if (t) {
    int rc = ensure_transpose(f, s);
    if (rc != FV_OK) return rc;
  }
  if (runs(f, t)) return launch_run<V>(f, t, r, x, s);
  if (!f->apply_exec[t]) {
    int rc = capture([&](cudaStream_t cs) { launch_apply_levels<V>(f, t, w, w, cs); },
                     &f->apply_exec[t]);
    if (rc != FV_OK) return rc;
  }
  FV_CUDA_TRY(cudaMemcpyAsync(w, r, sizeof(V) * n, cudaMemcpyDeviceToDevice, s));
  FV_CUDA_TRY(cudaGraphLaunch(f->apply_exec[t], s));
  FV_CUDA_TRY(cudaMemcpyAsync(x, w, sizeof(V) * n, cudaMemcpyDeviceToDevice, s));
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

int upload(const std::vector<int>& h, int** d, cudaStream_t s) {
  FV_CUDA_TRY(cudaMalloc(d, sizeof(int) * std::max<size_t>(1, h.size())));
  if (!h.empty())
    FV_CUDA_TRY(cudaMemcpyAsync(*d, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice, s));
  return FV_OK;
}

}  // namespace

extern "C" int fv_ilu0_create(int n, int b, const int* indptr, const int* indices, int precision,
                              void* stream, FvIlu0** out) {
  if (!out || n <= 0 || b <= 0 || b > 8 || !indptr || !indices ||
      (precision != 32 && precision != 64)) {
    fv_set_error("fv_ilu0_create: bad arguments (1 <= b <= 8, precision 32 or 64)");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int nnzb = indptr[n];
  std::vector<int> diag(n, -1);
  for (int i = 0; i < n; ++i) {
    for (int q = indptr[i]; q < indptr[i + 1]; ++q) {
      if (indices[q] < 0 || indices[q] >= n || (q > indptr[i] && indices[q] <= indices[q - 1])) {
        fv_set_error("fv_ilu0_create: row %d has unsorted or out-of-range column indices", i);
        return FV_ERR_ARG;
      }
      if (indices[q] == i) diag[i] = q;
    }
  }
  // reference message: aquaflux/solve/_ilu0.pyx:56-63 (the first rows missing a diagonal)
  std::vector<int> missing;
  for (int i = 0; i < n; ++i)
    if (diag[i] < 0) missing.push_back(i);
  if (!missing.empty()) {
    char buf[256];
    int len = snprintf(buf, sizeof(buf), "rows [");
    for (size_t k = 0; k < missing.size() && k < 5; ++k)
      len += snprintf(buf + len, sizeof(buf) - len, "%s%d", k ? ", " : "", missing[k] * b);
    snprintf(buf + len, sizeof(buf) - len, "]%s", missing.size() > 5 ? " \xe2\x80\xa6" : "");
    fv_set_error_index((long)missing[0] * b);
    fv_set_error("%s store no diagonal entry; ILU(0) eliminates in place and cannot introduce one.",
                 buf);
    return FV_ERR_NO_DIAG;
  }
  FvIlu0* f = new FvIlu0();
  f->n = n;
  f->b = b;
  f->nnzb = nnzb;
  f->precision = precision;
  f->traffic = (long)nnzb * b * b * (precision / 8);
  for (int i = 0; i < n; ++i) f->row_cap = std::max(f->row_cap, indptr[i + 1] - indptr[i]);
  std::vector<int> rows;
  levels(n, true, [&](int i, auto&& use) {
    for (int q = indptr[i]; q < diag[i]; ++q) use(indices[q]);
  }, &rows, &f->lv_fwd);
  if (upload(rows, &f->rows_fwd, s)) return FV_ERR_CUDA;
  const std::vector<int> rows_fwd(rows);
  const size_t nf = f->lv_fwd.size();
  f->lv_cap.assign(nf - 1, 0);
  f->lv_low.assign(nf - 1, 0);
  f->lv_sum.assign(nf - 1, 0);
  f->lv_scattered.assign(nf - 1, 0);
  int far = 0;
  for (size_t l = 0; l + 1 < nf; ++l) {
    int jumps = 0;
    for (int k = f->lv_fwd[l]; k < f->lv_fwd[l + 1]; ++k) {
      const int i = rows[k];
      jumps += k > f->lv_fwd[l] && rows[k - 1] != i - 1;
      f->lv_cap[l] = std::max(f->lv_cap[l], indptr[i + 1] - indptr[i]);
      f->lv_low[l] = std::max(f->lv_low[l], diag[i] - indptr[i]);
      f->lv_sum[l] += diag[i] - indptr[i];
    }
    f->lv_scattered[l] = jumps > (f->lv_fwd[l + 1] - f->lv_fwd[l]) / 8;
    if (f->lv_scattered[l]) far += f->lv_fwd[l + 1] - f->lv_fwd[l];
  }
  f->scattered = far > n / 2;
  std::vector<int> fwd_last(rows.begin() + f->lv_fwd[nf - 2], rows.begin() + f->lv_fwd[nf - 1]);
  levels(n, false, [&](int i, auto&& use) {
    for (int q = diag[i] + 1; q < indptr[i + 1]; ++q) use(indices[q]);
  }, &rows, &f->lv_bwd);
  if (upload(rows, &f->rows_bwd, s)) return FV_ERR_CUDA;
  // fused last forward / first backward level when they hold the same rows (the first backward
  // level's rows own no upper blocks by construction)
  std::vector<int> bwd_first(rows.begin() + f->lv_bwd[0], rows.begin() + f->lv_bwd[1]);
  std::sort(fwd_last.begin(), fwd_last.end());
  std::sort(bwd_first.begin(), bwd_first.end());
  f->fuse_fb = b > 1 && nf > 2 && f->lv_bwd.size() > 2 && fwd_last == bwd_first;
  int rc = build_run(f, 0, rows_fwd, f->lv_fwd, rows, f->lv_bwd, indices, 1, [&](int back, int i) {
    return back ? make_int4(i, indptr[i + 1] - 1 - diag[i], diag[i] + 1, diag[i])
                : make_int4(i, diag[i] - indptr[i], indptr[i], diag[i]);
  }, s);
  if (rc != FV_OK) return rc;
  f->h_ptr = std::make_shared<const std::vector<int>>(indptr, indptr + n + 1);
  f->h_idx = std::make_shared<const std::vector<int>>(indices, indices + nnzb);
  f->h_diag = std::make_shared<const std::vector<int>>(diag);
  if (upload(*f->h_ptr, &f->ptr, s) || upload(*f->h_idx, &f->idx, s) || upload(diag, &f->diag, s))
    return FV_ERR_CUDA;
  size_t vs = precision == 64 ? sizeof(double) : sizeof(float);
  FV_CUDA_TRY(cudaMalloc(&f->val, vs * (size_t)nnzb * b * b));
  FV_CUDA_TRY(cudaMalloc(&f->rp, vs * (size_t)n * b));
  FV_CUDA_TRY(cudaMalloc(&f->zero_flag, sizeof(unsigned long long)));
  FV_CUDA_TRY(cudaMalloc(&f->work, vs * (size_t)n * b));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  *out = f;
  return FV_OK;
}

extern "C" int fv_ilu0_destroy(FvIlu0* f) {
  if (!f) return FV_OK;
  if (f->open) cudaStreamSynchronize(f->side);
  if (f->side) cudaStreamDestroy(f->side);
  if (f->side_event) cudaEventDestroy(f->side_event);
  cudaFree(f->ptr);
  cudaFree(f->idx);
  cudaFree(f->diag);
  cudaFree(f->tptr);
  cudaFree(f->tidx);
  cudaFree(f->tblk);
  cudaFree(f->tdiag);
  cudaFree(f->val);
  cudaFree(f->rp);
  cudaFree(f->tval);
  cudaFree(f->zero_flag);
  cudaFree(f->rows_fwd);
  cudaFree(f->rows_bwd);
  cudaFree(f->rows_tfwd);
  cudaFree(f->rows_tbwd);
  cudaFree(f->work);
  for (const FvIlu0::Run& r : f->run) {
    cudaFree(r.row);
    cudaFree(r.col);
    cudaFree(r.bounds);
    cudaFree(r.rec);
  }
  for (cudaGraphExec_t e : f->apply_exec)
    if (e) cudaGraphExecDestroy(e);
  if (f->factor_exec) cudaGraphExecDestroy(f->factor_exec);
  delete f;
  return FV_OK;
}

namespace {
// Device copy of n ints (nothing when the source is absent).
int copy_ints(const int* src, size_t n, int** dst, cudaStream_t s) {
  if (!src) return FV_OK;
  FV_CUDA_TRY(cudaMalloc(dst, sizeof(int) * std::max<size_t>(1, n)));
  FV_CUDA_TRY(cudaMemcpyAsync(*dst, src, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
  return FV_OK;
}
}  // namespace

extern "C" int fv_ilu0_clone(const FvIlu0* src, int precision, void* stream, FvIlu0** out) {
  if (!src || !out || (precision != 0 && precision != 32 && precision != 64)) {
    fv_set_error("fv_ilu0_clone: bad arguments (precision 0, 32 or 64)");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  FvIlu0* f = new FvIlu0();
  f->n = src->n;
  f->b = src->b;
  f->nnzb = src->nnzb;
  f->precision = precision;
  f->row_cap = src->row_cap;
  f->traffic = (long)src->nnzb * src->b * src->b * (precision / 8);
  f->lv_cap = src->lv_cap;
  f->lv_low = src->lv_low;
  f->lv_sum = src->lv_sum;
  f->lv_scattered = src->lv_scattered;
  f->scattered = src->scattered;
  f->lv_fwd = src->lv_fwd;
  f->lv_bwd = src->lv_bwd;
  f->lv_tfwd = src->lv_tfwd;
  f->lv_tbwd = src->lv_tbwd;
  f->fuse_fb = src->fuse_fb;
  f->h_ptr = src->h_ptr;
  f->h_idx = src->h_idx;
  f->h_diag = src->h_diag;
  const size_t n = src->n, nnzb = src->nnzb;
  int rc = FV_OK;
  rc |= copy_ints(src->ptr, n + 1, &f->ptr, s);
  rc |= copy_ints(src->idx, nnzb, &f->idx, s);
  rc |= copy_ints(src->diag, n, &f->diag, s);
  rc |= copy_ints(src->rows_fwd, n, &f->rows_fwd, s);
  rc |= copy_ints(src->rows_bwd, n, &f->rows_bwd, s);
  if (src->tptr) {
    rc |= copy_ints(src->tptr, n + 1, &f->tptr, s);
    rc |= copy_ints(src->tidx, nnzb, &f->tidx, s);
    rc |= copy_ints(src->tblk, nnzb, &f->tblk, s);
    rc |= copy_ints(src->rows_tfwd, n, &f->rows_tfwd, s);
    rc |= copy_ints(src->rows_tbwd, n, &f->rows_tbwd, s);
    rc |= copy_ints(src->tdiag, n, &f->tdiag, s);
  }
  for (int t = 0; t < 2; ++t) {
    const FvIlu0::Run& r = src->run[t];
    if (!r.row) continue;
    f->run[t] = r;
    f->run[t].row = f->run[t].col = nullptr;
    f->run[t].bounds = nullptr;
    f->run[t].rec = nullptr;
    rc |= copy_ints((const int*)r.row, 8 * n, (int**)&f->run[t].row, s);
    rc |= copy_ints((const int*)r.col, 8 * n, (int**)&f->run[t].col, s);
    rc |= copy_ints(r.bounds, r.nlev + 1, &f->run[t].bounds, s);
  }
  if (rc == FV_OK && precision != 0) {
    const size_t vs = precision == 64 ? sizeof(double) : sizeof(float);
    if (cudaMalloc(&f->val, vs * nnzb * f->b * f->b) != cudaSuccess ||
        cudaMalloc(&f->rp, vs * n * f->b) != cudaSuccess ||
        cudaMalloc(&f->zero_flag, sizeof(unsigned long long)) != cudaSuccess ||
        cudaMalloc(&f->work, vs * n * f->b) != cudaSuccess)
      rc = FV_ERR_CUDA;
    // the transposed blocks, filled by the clone's factorisations
    if (rc == FV_OK && f->tdiag && cudaMalloc(&f->tval, vs * nnzb * f->b * f->b) != cudaSuccess)
      rc = FV_ERR_CUDA;
  }
  if (rc == FV_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = FV_ERR_CUDA;
  if (rc != FV_OK) {
    fv_set_error("fv_ilu0_clone: device allocation or copy failed");
    fv_ilu0_destroy(f);
    return FV_ERR_CUDA;
  }
  *out = f;
  return FV_OK;
}

namespace {
int factor_start(FvIlu0* f, const void* values, int values_f64, cudaStream_t s) {
  const long n = (long)f->nnzb * f->b * f->b;
  if (f->precision == 64) {
    FV_CUDA_TRY(cudaMemcpyAsync(f->val, values, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    return ilu_factor_start<double>(f, s);
  }
  if (values_f64)
    k_to_f32<<<fv_blocks(n, kThreads), kThreads, 0, s>>>(n, (const double*)values, (float*)f->val);
  else
    FV_CUDA_TRY(cudaMemcpyAsync(f->val, values, sizeof(float) * n, cudaMemcpyDeviceToDevice, s));
  return ilu_factor_start<float>(f, s);
}

// A factorisation started and not finished runs on its own stream: nothing else may use the factor.
bool refuse_open(const FvIlu0* f, const char* what) {
  if (f->open) fv_set_error("%s: fv_ilu0_factor_finish has to follow fv_ilu0_factor_start first", what);
  return f->open;
}
}  // namespace

extern "C" int fv_ilu0_factor(FvIlu0* f, const void* values, int values_f64, void* stream) {
  if (!f || !values || !f->val) {
    fv_set_error("fv_ilu0_factor: bad arguments");
    return FV_ERR_ARG;
  }
  if (refuse_open(f, "fv_ilu0_factor")) return FV_ERR_ARG;
  const int rc = factor_start(f, values, values_f64, (cudaStream_t)stream);
  return rc == FV_OK ? ilu_factor_finish(f, (cudaStream_t)stream) : rc;
}

extern "C" int fv_ilu0_factor_start(FvIlu0* f, const void* values, int values_f64, int urgent,
                                    void* stream) {
  if (!f || !values || !f->val) {
    fv_set_error("fv_ilu0_factor_start: bad arguments");
    return FV_ERR_ARG;
  }
  if (refuse_open(f, "fv_ilu0_factor_start")) return FV_ERR_ARG;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FV_CUDA_TRY(cudaStreamIsCapturing((cudaStream_t)stream, &cap));
  if (cap != cudaStreamCaptureStatusNone) {
    fv_set_error("fv_ilu0_factor_start: a factorisation cannot be captured (its zero pivots are read "
                 "by the host)");
    return FV_ERR_CUDA;
  }
  if (!f->side) {
    int least = 0, greatest = 0;
    FV_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    if (!f->side_event)
      FV_CUDA_TRY(cudaEventCreateWithFlags(&f->side_event, cudaEventDisableTiming));
    FV_CUDA_TRY(cudaStreamCreateWithPriority(&f->side, cudaStreamNonBlocking,
                                             urgent ? greatest : least));
  }
  FV_CUDA_TRY(cudaEventRecord(f->side_event, (cudaStream_t)stream));
  FV_CUDA_TRY(cudaStreamWaitEvent(f->side, f->side_event, 0));
  const int rc = factor_start(f, values, values_f64, f->side);
  f->open = rc == FV_OK;
  if (rc != FV_OK) cudaStreamSynchronize(f->side);  // what was queued reads the caller's values
  return rc;
}

extern "C" int fv_ilu0_factor_finish(FvIlu0* f, void* stream) {
  if (!f || !f->open) {
    fv_set_error("fv_ilu0_factor_finish: no factorisation was started");
    return FV_ERR_ARG;
  }
  f->open = false;
  FV_CUDA_TRY(cudaEventRecord(f->side_event, f->side));
  FV_CUDA_TRY(cudaStreamWaitEvent((cudaStream_t)stream, f->side_event, 0));
  return ilu_factor_finish(f, f->side);
}

extern "C" int fv_ilu0_apply(FvIlu0* f, const void* r, void* x, int transpose, void* stream) {
  if (!f || !r || !x || !f->val) {
    fv_set_error("fv_ilu0_apply: bad arguments");
    return FV_ERR_ARG;
  }
  if (refuse_open(f, "fv_ilu0_apply")) return FV_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (f->precision == 64) return ilu_apply<double>(f, (const double*)r, (double*)x, transpose, s);
  return ilu_apply<float>(f, (const float*)r, (float*)x, transpose, s);
}

extern "C" int fv_ilu0_set_traffic(FvIlu0* f, long bytes) {
  if (!f || bytes < 0) {
    fv_set_error("fv_ilu0_set_traffic: bad arguments");
    return FV_ERR_ARG;
  }
  if (f->traffic == bytes) return FV_OK;
  f->traffic = bytes;
  for (cudaGraphExec_t& e : f->apply_exec) {  // captured with the other kernels
    if (e) cudaGraphExecDestroy(e);
    e = nullptr;
  }
  return FV_OK;
}

extern "C" int fv_ilu0_factor_values(const FvIlu0* f, void* out, void* stream) {
  if (!f || !out || !f->val) {
    fv_set_error("fv_ilu0_factor_values: bad arguments");
    return FV_ERR_ARG;
  }
  if (refuse_open(f, "fv_ilu0_factor_values")) return FV_ERR_ARG;
  size_t vs = f->precision == 64 ? sizeof(double) : sizeof(float);
  FV_CUDA_TRY(cudaMemcpyAsync(out, f->val, vs * (size_t)f->nnzb * f->b * f->b,
                              cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
  return FV_OK;
}

// ------------------------------------------------------------------------------ shifted operator
namespace {
// Diagonal of every dof (cell i, field a) after the shift, and its equilibration factor.
__global__ void k_shift_diag(int n, int b, const int* __restrict__ ptr, const int* __restrict__ idx,
                             const double* __restrict__ val, const double* __restrict__ shift,
                             double* diag_cm, double* scale_cm, double* scale_fm, int* missing) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)n * b) return;
  const int i = (int)(t / b), a = (int)(t % b);
  int dq = -1;
  for (int q = ptr[i]; q < ptr[i + 1]; ++q)
    if (idx[q] == i) {
      dq = q;
      break;
    }
  if (dq < 0) {
    atomicMin(missing, i);
    return;
  }
  double d = val[((long)dq * b + a) * b + a];
  if (shift) d = d + shift[(long)a * n + i];
  diag_cm[t] = d;
  if (scale_cm) {
    double m = fabs(d);
    if (m == 0.0) m = 1.0;
    const double sc = 1.0 / sqrt(m);
    scale_cm[t] = sc;
    if (scale_fm) scale_fm[(long)a * n + i] = sc;
  }
}

// out[q][a][c] = ((v + shift on the diagonal) * s_row) * s_col, one thread per scalar row (i, a).
template <class Out>
__global__ void k_shift_scale(int n, int b, const int* __restrict__ ptr, const int* __restrict__ idx,
                              const double* __restrict__ val, const double* __restrict__ diag_cm,
                              const double* __restrict__ scale_cm, Out* __restrict__ out) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)n * b) return;
  const int i = (int)(t / b), a = (int)(t % b);
  const double sr = scale_cm ? scale_cm[t] : 1.0;
  for (int q = ptr[i]; q < ptr[i + 1]; ++q) {
    const int j = idx[q];
    const long base = ((long)q * b + a) * b;
    for (int c = 0; c < b; ++c) {
      double v = (j == i && c == a) ? diag_cm[t] : val[base + c];
      if (scale_cm) {
        v = v * sr;
        v = v * scale_cm[(long)j * b + c];
      }
      out[base + c] = (Out)v;
    }
  }
}
}  // namespace

extern "C" int fv_bsr_shift_equilibrate(int n, int b, const int* indptr, const int* indices,
                                        const double* values, const double* shift, int equilibrate,
                                        double* scale_fm, double* work, void* out, int out_f64,
                                        void* stream) {
  if (n <= 0 || b <= 0 || !indptr || !indices || !values || !work || !out) {
    fv_set_error("fv_bsr_shift_equilibrate: bad arguments");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const long m = (long)n * b;
  double* diag_cm = work;
  double* scale_cm = equilibrate ? work + m : nullptr;
  int* missing = reinterpret_cast<int*>(work + 2 * m);
  const int init = 0x7fffffff;
  FV_CUDA_TRY(cudaMemcpyAsync(missing, &init, sizeof(int), cudaMemcpyHostToDevice, s));
  k_shift_diag<<<fv_blocks(m, kThreads), kThreads, 0, s>>>(n, b, indptr, indices, values, shift,
                                                           diag_cm, scale_cm, scale_fm, missing);
  if (out_f64)
    k_shift_scale<double><<<fv_blocks(m, kThreads), kThreads, 0, s>>>(
        n, b, indptr, indices, values, diag_cm, scale_cm, (double*)out);
  else
    k_shift_scale<float><<<fv_blocks(m, kThreads), kThreads, 0, s>>>(
        n, b, indptr, indices, values, diag_cm, scale_cm, (float*)out);
  FV_CUDA_TRY(cudaGetLastError());
  int miss = 0;
  FV_CUDA_TRY(cudaMemcpyAsync(&miss, missing, sizeof(int), cudaMemcpyDeviceToHost, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  if (miss != init) {
    fv_set_error_index(miss);
    fv_set_error("fv_bsr_shift_equilibrate: block row %d stores no diagonal block; the shift has "
                 "nowhere to go", miss);
    return FV_ERR_NO_DIAG;
  }
  return FV_OK;
}

// ------------------------------------------------------------------------------ SpMV entry points
namespace {
template <class V>
int spmv(int nbr, int b, const int* indptr, const int* indices, const V* values, const V* x, V* y,
         int transpose, cudaStream_t s) {
  if (nbr <= 0 || b <= 0 || !indptr || !indices || !values || !x || !y) {
    fv_set_error("fv_bsr_spmv: bad arguments");
    return FV_ERR_ARG;
  }
  const long rows = (long)nbr * b;
  if (!transpose) {
    const bool aligned = ((uintptr_t)values % 16 == 0) && ((uintptr_t)x % 16 == 0);
    if (aligned && b >= 2 && b <= 8)
      launch_spmv_b<V, false>(nbr, b, {}, indptr, indices, values, x, (const V*)nullptr, y, s);
    else
      k_bsr_spmv<V><<<fv_blocks(rows, kThreads), kThreads, 0, s>>>(nbr, b, indptr, indices,
                                                                   values, x, nullptr, y);
    FV_CUDA_TRY(cudaGetLastError());
    return FV_OK;
  }
  // transposed product: build the transpose map of the (device) pattern on the host once per call
  std::vector<int> hp(nbr + 1);
  FV_CUDA_TRY(cudaMemcpyAsync(hp.data(), indptr, sizeof(int) * (nbr + 1), cudaMemcpyDeviceToHost, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  for (int i = 0; i < nbr; ++i)
    if (hp[i] > hp[i + 1] || hp[0] != 0) {
      fv_set_error("fv_bsr_spmv: indptr is not a non-decreasing offset list from 0");
      return FV_ERR_ARG;
    }
  std::vector<int> hi(hp[nbr]);
  FV_CUDA_TRY(cudaMemcpy(hi.data(), indices, sizeof(int) * hp[nbr], cudaMemcpyDeviceToHost));
  for (int q = 0; q < hp[nbr]; ++q)
    if (hi[q] < 0 || hi[q] >= nbr) {
      fv_set_error("fv_bsr_spmv: column index %d at block %d out of range [0, %d)", hi[q], q, nbr);
      return FV_ERR_ARG;
    }
  Transpose T;
  build_transpose(nbr, nbr, hp.data(), hi.data(), &T);
  int *tp = nullptr, *ti = nullptr, *tb = nullptr;
  if (upload(T.ptr, &tp, s) || upload(T.idx, &ti, s) || upload(T.blk, &tb, s)) {
    cudaFree(tp);
    cudaFree(ti);
    cudaFree(tb);
    return FV_ERR_CUDA;
  }
  launch_spmv_t<V>(nbr, b, tp, ti, tb, values, x, y, s);
  FV_CUDA_TRY(cudaGetLastError());
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  cudaFree(tp);
  cudaFree(ti);
  cudaFree(tb);
  return FV_OK;
}
}  // namespace

// Transpose map of a square BSR pattern (host): for block row j of A^T the rows i of A with a
// block (i, j) (tptr / tidx) and that block's index in A (tblk).  tptr n + 1; tidx, tblk nnzb.
extern "C" int fv_bsr_transpose_map(int n, const int* indptr, const int* indices, int* tptr,
                                    int* tidx, int* tblk) {
  if (n <= 0 || !indptr || !indices || !tptr || !tidx || !tblk) {
    fv_set_error("fv_bsr_transpose_map: bad arguments");
    return FV_ERR_ARG;
  }
  if (!fv_offsets_ok("fv_bsr_transpose_map", n, indptr)) return FV_ERR_ARG;
  for (int q = 0; q < indptr[n]; ++q)
    if (indices[q] < 0 || indices[q] >= n) {
      fv_set_error("fv_bsr_transpose_map: column index out of range");
      return FV_ERR_ARG;
    }
  Transpose T;
  build_transpose(n, n, indptr, indices, &T);
  std::copy(T.ptr.begin(), T.ptr.end(), tptr);
  std::copy(T.idx.begin(), T.idx.end(), tidx);
  std::copy(T.blk.begin(), T.blk.end(), tblk);
  return FV_OK;
}

// y = A^T x through a transpose map from fv_bsr_transpose_map (device arrays; no allocation).
extern "C" int fv_bsr_spmv_t_mapped(int n, int b, const int* tptr, const int* tidx,
                                    const int* tblk, const void* values, const void* x, void* y,
                                    int f64, void* stream) {
  if (n <= 0 || b <= 0 || !tptr || !tidx || !tblk || !values || !x || !y) {
    fv_set_error("fv_bsr_spmv_t_mapped: bad arguments");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (f64)
    launch_spmv_t<double>(n, b, tptr, tidx, tblk, (const double*)values, (const double*)x,
                          (double*)y, s);
  else
    launch_spmv_t<float>(n, b, tptr, tidx, tblk, (const float*)values, (const float*)x, (float*)y,
                         s);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

extern "C" int fv_bsr_transpose_blocks(long nnzb, int b, const int* tblk, const void* values,
                                       void* tvalues, int f64, void* stream) {
  if (nnzb <= 0 || b <= 0 || !tblk || !values || !tvalues) {
    fv_set_error("fv_bsr_transpose_blocks: bad arguments");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const long nv = nnzb * b * b;
  if (f64)
    k_transpose_blocks<double><<<fv_blocks(nv, kThreads), kThreads, 0, s>>>(
        nnzb, b, tblk, (const double*)values, (double*)tvalues);
  else
    k_transpose_blocks<float><<<fv_blocks(nv, kThreads), kThreads, 0, s>>>(
        nnzb, b, tblk, (const float*)values, (float*)tvalues);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

extern "C" int fv_bsr_spmv_f64(int nbr, int b, const int* indptr, const int* indices,
                               const double* values, const double* x, double* y, int transpose,
                               void* stream) {
  return spmv<double>(nbr, b, indptr, indices, values, x, y, transpose, (cudaStream_t)stream);
}
extern "C" int fv_bsr_spmv_f32(int nbr, int b, const int* indptr, const int* indices,
                               const float* values, const float* x, float* y, int transpose,
                               void* stream) {
  return spmv<float>(nbr, b, indptr, indices, values, x, y, transpose, (cudaStream_t)stream);
}

namespace {
template <class V>
int bsr_product(const char* name, bool need_rhs, int nbr, int b, const ProductHint& hint,
                const int* indptr, const int* indices, const V* values, const V* x, const V* rhs,
                V* y, void* stream) {
  if (nbr <= 0 || b <= 0 || hint.nnzb < 0 || !indptr || !indices || !values || !x || !y ||
      (need_rhs && !rhs)) {
    fv_set_error("%s: bad arguments", name);
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (((uintptr_t)values | (uintptr_t)x) % 16 == 0 && b >= 2 && b <= 8) {
    if (rhs)
      launch_spmv_b<V, true>(nbr, b, hint, indptr, indices, values, x, rhs, y, s);
    else
      launch_spmv_b<V, false>(nbr, b, hint, indptr, indices, values, x, rhs, y, s);
  } else {
    k_bsr_spmv<V><<<fv_blocks((long)nbr * b, kThreads), kThreads, 0, s>>>(nbr, b, indptr, indices,
                                                                         values, x, rhs, y);
  }
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}
}  // namespace

extern "C" int fv_bsr_residual_f64(int nbr, int b, const int* indptr, const int* indices,
                                   const double* values, const double* x, const double* rhs,
                                   double* r, void* stream) {
  return bsr_product<double>("fv_bsr_residual", true, nbr, b, {}, indptr, indices, values, x, rhs, r,
                             stream);
}
extern "C" int fv_bsr_residual_f32(int nbr, int b, const int* indptr, const int* indices,
                                   const float* values, const float* x, const float* rhs, float* r,
                                   void* stream) {
  return bsr_product<float>("fv_bsr_residual", true, nbr, b, {}, indptr, indices, values, x, rhs, r,
                            stream);
}
extern "C" int fv_bsr_product_f64(int nbr, int b, long nnzb, int longest, long traffic,
                                  const int* indptr, const int* indices, const double* values,
                                  const double* x, const double* rhs, double* y, void* stream) {
  return bsr_product<double>("fv_bsr_product", false, nbr, b, {nnzb, longest, traffic}, indptr,
                             indices, values, x, rhs, y, stream);
}
extern "C" int fv_bsr_product_f32(int nbr, int b, long nnzb, int longest, long traffic,
                                  const int* indptr, const int* indices, const float* values,
                                  const float* x, const float* rhs, float* y, void* stream) {
  return bsr_product<float>("fv_bsr_product", false, nbr, b, {nnzb, longest, traffic}, indptr,
                            indices, values, x, rhs, y, stream);
}

// out[i] = sum over fields q and cells c in [seg[i], seg[i + 1]) of a[q nc + c] b[q nc + c]: one
// block per segment, fixed summation order.
__global__ void k_segment_dot(const int* seg, int nfld, int nc, const double* a, const double* b,
                              double* out) {
  __shared__ double red[256];
  const int i = blockIdx.x;
  const int lo = seg[i], hi = seg[i + 1];
  double acc = 0.0;
  for (int q = 0; q < nfld; ++q)
    for (int c = lo + threadIdx.x; c < hi; c += blockDim.x)
      acc += a[(long)q * nc + c] * b[(long)q * nc + c];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[i] = red[0];
}

extern "C" int fv_segment_dot(int n_seg, const int* seg, int nfld, int nc, const double* a,
                              const double* b, double* out, void* stream) {
  if (n_seg <= 0 || nfld <= 0 || nc <= 0 || !seg || !a || !b || !out) {
    fv_set_error("fv_segment_dot: bad arguments");
    return FV_ERR_ARG;
  }
  k_segment_dot<<<n_seg, 256, 0, (cudaStream_t)stream>>>(seg, nfld, nc, a, b, out);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

extern "C" int fv_dot_f64(long n, const double* x, const double* y, double* out, void* stream) {
  if (n < 0 || !x || !y || !out) {
    fv_set_error("fv_dot_f64: bad arguments");
    return FV_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (!g_dot_parts) FV_CUDA_TRY(cudaMalloc(&g_dot_parts, sizeof(double) * kRedBlocks));
  k_dot_partial<<<kRedBlocks, kThreads, 0, s>>>(n, x, y, g_dot_parts);
  k_dot_final<<<1, kThreads, 0, s>>>(kRedBlocks, g_dot_parts, out);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}
