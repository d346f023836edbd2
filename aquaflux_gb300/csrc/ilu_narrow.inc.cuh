// Triangular solves of an ILU(0) factor whose level sets are narrow: both sweeps in one launch.
//
// Included by sparse.cu inside its anonymous namespace.
//
// A level set of a small or banded operator holds a few dozen block rows, so a launch per level is
// all latency: 2.9 us (fp64, forward) and 3.6 us (backward) a level on the 64 x 64 cavity, whose
// 127 level sets of at most 64 rows made a solve 0.83 ms, for a few hundred bytes a row.
// Here one block runs every level, the vector in its shared memory, a block barrier between
// levels.  What bounds it then is fp64 issue and the instructions around it: an fp64 instruction
// holds a quarter of an SM for 64 cycles whatever its active lanes (measured; its latency is no
// longer), so
//   * rows take 4 lanes for b <= 4;
//   * the fp64 forward solve uses fused multiply-subtracts, and a diagonal block whose upper part
//     is divided by its pivots at the factorisation, so that all quotients of a row are taken at
//     once: 8 and 11 fp64 instructions a level (b = 3, two blocks) for 18 and 30;
//   * a row's operands are packed at the factorisation, in level order and lane by lane
//     (k_run_pack): a record is read at constant offsets from one address, a level ahead.
// Measured on that cavity: a forward solve 0.83 -> 0.185 ms, a transposed one 0.86 -> 0.34 ms.  A
// cluster of 2, 4 or 8 blocks exchanging entries with st.async divides the fp64 work but pays a
// remote store's latency a level: 0.28 ms at every size.
//
// fp32 solves and the fp64 transposed solve see the operations of the launch-per-level kernels in
// their order: bitwise the same.

constexpr int kRunThreads = 384;   // largest block (168 registers a thread)
constexpr int kRunBlocks = 4;      // off-diagonal blocks of a row in its record; more are read in place
constexpr size_t kRunSmem = 220 * 1024;

__host__ __device__ constexpr int run_lanes(int b) { return b <= 4 ? 4 : 8; }
// Block sizes whose operands, two levels of them, stay in a thread's registers.
__host__ __device__ constexpr bool run_block_size(int b, size_t vs) {
  return b >= 2 && b <= (vs == 8 ? 4 : 6);
}
// Rows a level may hold: one per lane group of the block.
inline int run_capacity(int b) { return kRunThreads / run_lanes(b); }
// ... and in fp64 the rows they may hold in the mean, `most` blocks in a row, for one block's fp64
// units not to take longer than a launch per level: soonest in the transposed solve, with twice the
// operations of the fused forward one.  Time in one launch over that of a launch per level (60 level
// sets; the launches take 0.34 ms for 2 blocks a row of b = 3, 0.62 for 8), by blocks a row and rows:
//   transposed  b = 3    2: 64 0.80, 88 1.03    4: 48 0.92, 56 1.03    8: 40 0.99, 48 1.07   20: 24 1.08
//               b = 4    2: 64 0.97, 72 1.09    4: 40 0.98, 48 1.09    8: 32 0.94, 40 1.05   20: 24 1.05
//               b = 2    2: 96 0.90             4: 64 0.96, 72 1.03    8: 48 0.92, 56 1.05   20: 24 1.03
//   forward     b = 4    2: 96 0.71             4: 80 1.00, 88 1.09    8: 80 0.97, 88 1.04   20: 88 0.97
//   and below 1 for b = 2 and 3 throughout
// (in the mean: 90 x 90 cells, level sets of 1 to 90 rows, b = 3 615 us transposed, 991 by launches).
inline int run_mean64(int b, int most, bool transposed) {
  if (!transposed) return b == 4 && most >= 4 ? 80 : run_capacity(b);
  constexpr int few[5] = {240, 240, 200, 152, 104};
  return 16 + (most <= 4 ? few[most] : std::max(0, 120 - 5 * most)) / b;
}
// Entries of a record per lane: the diagonal block's row, the pivot's reciprocal, `k` blocks' rows.
__host__ __device__ constexpr int run_entries(int b, int k) { return b + 1 + k * b; }

// One solve in level order, the forward sweep's rows then the backward sweep's: `bounds` the level
// offsets, `row` (row, off-diagonal blocks, first one's position, diagonal block's position),
// `col` the rows' first kRunBlocks columns (times b), `rec` their records.
template <class V>
struct RunView {
  int n, nlev, nlev_fwd, k;  // k: blocks per record
  const int* bounds;
  const int4* row;
  const int4* col;
  const V* rec;
  const int* idx;
  const V* val;
};

// acc - l * x: one rounding in the fp64 forward solve (half the fp64 instructions of two).
template <bool FUSED, class V>
__device__ __forceinline__ V msub(V acc, V l, V x) {
  if constexpr (FUSED) return fma_rn(-l, x, acc);
  else return acc - l * x;
}

// The quotient of upper_block_solve (see there): correctly rounded from the pivot's reciprocal.
template <class V>
__device__ __forceinline__ V pivot_quotient(V acc, V piv, V rpiv) {
  if (isfinite(rpiv)) {
    const V q = acc * rpiv;
    return fma_rn(fma_rn(-q, piv, acc), rpiv, q);
  }
  return acc / piv;
}

// A quotient by a pivot that may stand in a record: between 2^-256 and 2^256.
__device__ __forceinline__ bool scalable(double q) {
  const int e = (__double2hiint(q) >> 20 & 0x7ff) - 1023;
  return e >= -256 && e < 256;
}
__device__ __forceinline__ bool finite_hi(double x) {  // no fp64 comparison
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// The records of a solve from the factor's blocks (val: transposed blocks for the transposed solve,
// whose backward sweep takes a row's blocks from the last one down). A row of the fp64 forward
// solve whose pivot's reciprocal or scaled entries would be large or small enough for a product
// with them to leave the range of doubles stays as it is, marked by a NaN for the reciprocal, and
// is divided last.
template <class V>
__global__ void k_run_pack(int n, int b, int k, bool transposed, const int4* row, const V* val,
                           V* rec) {
  const int lg = run_lanes(b);
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int s = (int)(t / lg), a = (int)(t % lg);
  if (s >= 2 * n || a >= b) return;
  const int4 d = row[s];
  const int step = transposed && s >= n ? -1 : 1;
  V* o = rec + (long)s * run_entries(b, k) * lg + a;
  const V* D = val + ((long)d.w * b + a) * b;
  const V piv = D[a];
  V rpiv = V(1) / piv;
  bool scaled = sizeof(V) == 8 && !transposed;
  if (scaled) {
    scaled = scalable(rpiv);
    for (int c = a + 1; c < b; ++c) scaled = scaled && (D[c] == V(0) || scalable(D[c] / piv));
    if (!scaled) rpiv = (V)__longlong_as_double(0x7ff8000000000000LL);
  }
  for (int c = 0; c < b; ++c) o[(long)c * lg] = scaled && c > a ? D[c] / piv : D[c];
  o[(long)b * lg] = rpiv;
  for (int q = 0; q < k && q < d.y; ++q) {
    const V* L = val + ((long)(d.z + step * q) * b + a) * b;
    for (int c = 0; c < b; ++c) o[(long)(b + 1 + q * b + c) * lg] = L[c];
  }
}

// A row's operands, held a level ahead.
template <class V, int B, int K>
struct RunRow {
  int4 row, col;  // row.x < 0: this group has no row in the level
  V D[B], rpiv, L[K][B];
};

// Level l's operands of this thread's group; l <= nlev, the level past the last being empty.
template <class V, int B, int K>
__device__ __forceinline__ void run_fetch(const RunView<V>& R, const int* bounds, int l,
                                          RunRow<V, B, K>& w) {
  constexpr int LG = run_lanes(B);
  const int a = threadIdx.x & (LG - 1), s = bounds[l] + threadIdx.x / LG;
  w.row = make_int4(-1, 0, 0, 0);
  if (s >= bounds[l + 1]) return;
  w.row = R.row[s];
  w.col = R.col[s];
  const V* p = R.rec + (long)s * (run_entries(B, R.k) * LG) + (a < B ? a : 0);
#pragma unroll
  for (int c = 0; c < B; ++c) w.D[c] = p[c * LG];
  w.rpiv = p[B * LG];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (k < R.k) {
#pragma unroll
      for (int c = 0; c < B; ++c) w.L[k][c] = p[(B + 1 + k * B + c) * LG];
    }
}

// One level: the rows' entries of xs from those of the levels before.
template <class V, int B, int K, bool T>
__device__ __forceinline__ void run_level(const RunView<V>& R, int l, const RunRow<V, B, K>& w,
                                          V* xs) {
  constexpr int LG = run_lanes(B);
  constexpr bool kFused = sizeof(V) == 8 && !T;  // fp64 forward solve
  const int a = threadIdx.x & (LG - 1), ar = a < B ? a : 0;
  const bool live = a < B;
  const bool back = l >= R.nlev_fwd, down = T && back;
  const bool on = w.row.x >= 0;
  if (!__any_sync(0xffffffffu, on)) return;
  const int nq = on ? w.row.y : 0;
  const int me = on ? w.row.x * B + ar : 0;
  V acc = xs[me];
  V xj[K][B];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (k < R.k) {
      const int j = k >= nq ? 0 : k == 0 ? w.col.x : k == 1 ? w.col.y : k == 2 ? w.col.z : w.col.w;
#pragma unroll
      for (int c = 0; c < B; ++c) xj[k][c] = xs[j + c];
    }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (__any_sync(0xffffffffu, k < nq)) {
      V s = acc;
      if (down) {
#pragma unroll
        for (int c = B - 1; c >= 0; --c) s = msub<kFused>(s, w.L[k][c], xj[k][c]);
      } else {
#pragma unroll
        for (int c = 0; c < B; ++c) s = msub<kFused>(s, w.L[k][c], xj[k][c]);
      }
      if (k < nq) acc = s;
    }
  if constexpr (K == kRunBlocks) {
    for (int k0 = kRunBlocks; k0 < nq; k0 += 2) {
      V L[2][B];
      int col[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (k0 + k < nq) {
          const int q = down ? w.row.z - k0 - k : w.row.z + k0 + k;
          col[k] = R.idx[q] * B;
          load_seg<B>(R.val + ((long)q * B + ar) * B, L[k]);
        }
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (k0 + k < nq) {
          if (down) {
#pragma unroll
            for (int c = B - 1; c >= 0; --c) acc = msub<kFused>(acc, L[k][c], xs[col[k] + c]);
          } else {
#pragma unroll
            for (int c = 0; c < B; ++c) acc = msub<kFused>(acc, L[k][c], xs[col[k] + c]);
          }
        }
    }
    __syncwarp();
  }
  // the diagonal block: L (unit lower) and U forward and back, U^T (lower) and L^T (unit upper)
  // for the transpose
  V piv = V(1);
#pragma unroll
  for (int c = 0; c < B; ++c)
    if (a == c) piv = w.D[c];
  if (!back) {
#pragma unroll
    for (int c = 0; c < B; ++c) {
      if (T && a == c) acc = pivot_quotient(acc, piv, w.rpiv);
      if (c < B - 1) {
        const V vc = __shfl_sync(0xffffffffu, acc, c, LG);
        if (live && a > c) acc = msub<kFused>(acc, w.D[c], vc);
      }
    }
  } else {
    bool scaled = true;
    if constexpr (kFused) {
      scaled = finite_hi(w.rpiv);
      if (scaled) {
        const V q = acc * w.rpiv;
        acc = fma_rn(fma_rn(-q, piv, acc), w.rpiv, q);
      }
    }
    if (kFused && __any_sync(0xffffffffu, on && live && !scaled)) {
      // a row left unscaled (k_run_pack) takes the launch-per-level kernel's operations
#pragma unroll
      for (int c = B - 1; c >= 0; --c) {
        if (a == c && !scaled) acc = acc / piv;
        const V vc = __shfl_sync(0xffffffffu, acc, c, LG);
        if (live && a < c) acc = scaled ? msub<kFused>(acc, w.D[c], vc) : acc - w.D[c] * vc;
      }
    } else {
#pragma unroll
      for (int c = B - 1; c >= 0; --c) {
        if (!T && !kFused && a == c) acc = pivot_quotient(acc, piv, w.rpiv);
        if (c > 0) {
          const V vc = __shfl_sync(0xffffffffu, acc, c, LG);
          if (live && a < c) acc = msub<kFused>(acc, w.D[c], vc);
        }
      }
    }
  }
  if (on && live) xs[me] = acc;
}

// K blocks per record (R.k <= K).
template <class V, int B, int K, bool T>
__global__ void __launch_bounds__(kRunThreads) k_ilu_run(RunView<V> R, const V* r, V* x) {
  constexpr int LG = run_lanes(B);
  extern __shared__ __align__(16) unsigned char run_smem[];
  int* bounds = (int*)run_smem;
  V* xs = (V*)(run_smem + ((R.nlev + 2) * 4 + 15) / 16 * 16);
  const int t = threadIdx.x, nt = blockDim.x;
  for (int l = t; l < R.nlev + 2; l += nt) bounds[l] = R.bounds[l <= R.nlev ? l : R.nlev];
  const long nx = (long)R.n * B;
  constexpr int kVec = 16 / (int)sizeof(V);
  if ((uintptr_t)r % 16 == 0) {
    const long nv = nx / kVec;
#pragma unroll 8
    for (long k = t; k < nv; k += nt)
      reinterpret_cast<uint4*>(xs)[k] = reinterpret_cast<const uint4*>(r)[k];
    for (long k = nv * kVec + t; k < nx; k += nt) xs[k] = r[k];
  } else {
#pragma unroll 8
    for (long k = t; k < nx; k += nt) xs[k] = r[k];
  }
  __syncthreads();

  RunRow<V, B, K> w0, w1;
  run_fetch<V, B, K>(R, bounds, 0, w0);
  for (int l = 0; l < R.nlev; l += 2) {
    run_fetch<V, B, K>(R, bounds, l + 1, w1);
    run_level<V, B, K, T>(R, l, w0, xs);
    __syncthreads();
    if (l + 1 == R.nlev) break;
    run_fetch<V, B, K>(R, bounds, l + 2, w0);
    run_level<V, B, K, T>(R, l + 1, w1, xs);
    __syncthreads();
  }
  if ((uintptr_t)x % 16 == 0) {
    const long nv = nx / kVec;
#pragma unroll 4
    for (long k = t; k < nv; k += nt)
      reinterpret_cast<uint4*>(x)[k] = reinterpret_cast<const uint4*>(xs)[k];
    for (long k = nv * kVec + t; k < nx; k += nt) x[k] = xs[k];
  } else {
    for (long k = t; k < nx; k += nt) x[k] = xs[k];
  }
}

// Shared memory of a solve: level bounds, the vector.
inline size_t run_smem_bytes(long n, int b, int nlev, size_t vs) {
  return ((size_t)(nlev + 2) * 4 + 15) / 16 * 16 + (size_t)n * b * vs;
}

template <class V, int B>
int launch_run_b(const RunView<V>& R, int widest, bool transpose, const V* r, V* x,
                 cudaStream_t s) {
  if constexpr (run_block_size(B, sizeof(V))) {
    const size_t smem = run_smem_bytes(R.n, B, R.nlev, sizeof(V));
    const int threads = std::max(256, (widest * run_lanes(B) + 31) / 32 * 32);
    // two blocks a row are what a 2D mesh has; fewer registers, fewer instructions than four
    auto kern = R.k <= 2 ? (transpose ? k_ilu_run<V, B, 2, true> : k_ilu_run<V, B, 2, false>)
                         : (transpose ? k_ilu_run<V, B, kRunBlocks, true>
                                      : k_ilu_run<V, B, kRunBlocks, false>);
    // the limit belongs to the function, which other threads launch with other sizes: one value
    FV_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kRunSmem));
    kern<<<1, threads, smem, s>>>(R, r, x);
    FV_CUDA_TRY(cudaGetLastError());
  }
  return FV_OK;
}
