// General row-major matrix product on the CUDA cores:
//   out[m][n] = alpha * A[m][k] B[k][n] + bias[m] + (accumulate ? out : 0).
// Used for the FP64 verification path (dense LinearMatrix at d = 50, full mass
// matrices, full-covariance Normal priors) and for FP32 products (full mass
// matrices, the elastic model's blob projections).  The FP32 production
// contraction of the dense LinearMatrix runs on the tensor cores (dense_tc.cu).
// gemm_kernel: FP64, any shape, and FP32 rows too long for 32-bit offsets;
// gemv_kernel: FP64, few columns; gemm_f32_kernel: FP32.
#include "common.cuh"
#include "gemm_shape.cuh"

namespace hmc {
namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// blockIdx.z selects the k range [z * k_chunk, (z + 1) * k_chunk); with
// `partial` set, the raw sums of that range go to partial[z][m][n] and the
// epilogue is left to splitk_reduce_kernel.
template <typename T>
__global__ void __launch_bounds__(256) gemm_kernel(int64_t M, int64_t N, int64_t K, T alpha, const T* __restrict__ A,
                                                   const T* __restrict__ B, const T* __restrict__ bias, T bias_scale,
                                                   const T* __restrict__ row_scale, T* out, int accumulate,
                                                   int64_t k_chunk, T* partial) {
  __shared__ T As[BK][BM + 1];
  __shared__ T Bs[BK][BN + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int64_t row0 = (int64_t)blockIdx.y * BM, col0 = (int64_t)blockIdx.x * BN;
  T acc[TM][TN];
#pragma unroll
  for (int a = 0; a < TM; ++a)
#pragma unroll
    for (int b = 0; b < TN; ++b) acc[a][b] = (T)0;

  const int64_t kb = (int64_t)blockIdx.z * k_chunk;
  const int64_t ke = kb + k_chunk < K ? kb + k_chunk : K;
  for (int64_t k0 = kb; k0 < ke; k0 += BK) {
    // A tile: BM x BK, 1024 elements, 4 per thread.
    for (int e = threadIdx.x; e < BM * BK; e += 256) {
      const int r = e / BK, kk = e % BK;
      const int64_t gr = row0 + r, gk = k0 + kk;
      As[kk][r] = (gr < M && gk < ke) ? A[gr * K + gk] : (T)0;
    }
    for (int e = threadIdx.x; e < BK * BN; e += 256) {
      const int kk = e / BN, cc = e % BN;
      const int64_t gk = k0 + kk, gc = col0 + cc;
      Bs[kk][cc] = (gk < ke && gc < N) ? B[gk * N + gc] : (T)0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      T a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] += a[i] * b[j];
    }
    __syncthreads();
  }
  if (partial) {
    T* p = partial + (int64_t)blockIdx.z * M * N;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t r = row0 + ty + 16 * i;
      if (r >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int64_t c = col0 + tx + 16 * j;
        if (c < N) p[r * N + c] = acc[i][j];
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t r = row0 + ty + 16 * i;
    if (r >= M) continue;
    const T bv = bias ? bias_scale * bias[r] : (T)0;
    const T rs = row_scale ? row_scale[r] : (T)1;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int64_t c = col0 + tx + 16 * j;
      if (c >= N) continue;
      T v = alpha * acc[i][j] + bv;
      if (row_scale) v *= rs;
      if (accumulate) v += out[r * N + c];
      out[r * N + c] = v;
    }
  }
}

// out = alpha * sum_z partial[z] (+ out), summed in z order.
template <typename T>
__global__ void splitk_reduce_kernel(int64_t mn, int splits, T alpha, const T* __restrict__ partial, T* out,
                                     int accumulate) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < mn; e += (int64_t)gridDim.x * blockDim.x) {
    T s = (T)0;
    for (int z = 0; z < splits; ++z) s += partial[(int64_t)z * mn + e];
    s *= alpha;
    out[e] = accumulate ? out[e] + s : s;
  }
}

// The FP32 product.  A thread owns RPT rows x 4 columns of the output, CX
// threads a block's columns and THREADS / CX groups its rows; k runs in chunks of
// 16 that are loaded one chunk ahead, and a thread reads its rows and columns
// with RPT + 4 16-byte loads per 16 RPT multiply-adds (the tile kernel above:
// eight 4-byte loads per 16, and a block that waits for every chunk's loads).
// Every output is one chain of fused multiply-adds in ascending k, as there, so
// results do not change.  What bounds it is instruction issue; a block is four
// warps, one per scheduler, and the rows per thread are those that leave the
// matrix the least padding: 129 x 129 against 8192 columns, the full mass matrix
// of a source location, took 26 us (192 padded rows) and takes 13.
constexpr int KC = 16;
template <int CX, int RPT, int THREADS, bool B16>
__global__ void __launch_bounds__(THREADS, 3)
    gemm_f32_kernel(int64_t M, int64_t N, int64_t K, float alpha, const float* __restrict__ A,
                    const float* __restrict__ B, const float* __restrict__ bias, float bias_scale,
                    const float* __restrict__ row_scale, float* out, int accumulate, int64_t k_chunk, float* partial) {
  constexpr int CT = CX * 4;
  constexpr int PITCH = KC + 4;  // the row groups of a warp read different banks
  constexpr int ALOADS = KC * RPT / CX;                         // per thread
  constexpr int BLOADS = (KC * (B16 ? CX : CT) + THREADS - 1) / THREADS;
  constexpr int threads = THREADS, groups = threads / CX, rows = groups * RPT;
  constexpr int buffer = rows * PITCH + KC * CT;  // floats: A chunk [row][k], then B chunk [k][column]
  __shared__ __align__(16) float sm[2 * buffer];
  const int tx = threadIdx.x % CX, ty = threadIdx.x / CX;
  const int64_t row0 = (int64_t)blockIdx.y * rows, col0 = (int64_t)blockIdx.x * CT;
  const int64_t kb = (int64_t)blockIdx.z * k_chunk;
  const int64_t ke = kb + k_chunk < K ? kb + k_chunk : K;

  // The next chunk travels in registers while this one is multiplied.  Rows and
  // columns past the matrix repeat its last ones (their sums are not stored), so
  // only the last chunk of k checks bounds.
  float ar[ALOADS], br[B16 ? 4 * BLOADS : BLOADS];
  constexpr int lstep = threads / KC;
  const int lr = threadIdx.x / KC, lk = threadIdx.x % KC;
  uint32_t aoff[ALOADS];  // (f32_offsets_fit)
#pragma unroll
  for (int i = 0; i < ALOADS; ++i) {
    const int64_t r = lr + i * lstep, last = M - 1 - row0;
    aoff[i] = (uint32_t)((r < last ? r : last) * K) + (uint32_t)lk;
  }
  const float* const abase = A + row0 * K;
  auto fetch = [&](int64_t k0) {
    const float* a = abase + k0;
    if (k0 + KC <= ke) {
#pragma unroll
      for (int i = 0; i < ALOADS; ++i) ar[i] = a[aoff[i]];
    } else {
#pragma unroll
      for (int i = 0; i < ALOADS; ++i) ar[i] = k0 + lk < ke ? a[aoff[i]] : 0.f;
    }
    const float* b = B + k0 * N + col0;
    if constexpr (B16) {
#pragma unroll
      for (int i = 0; i < BLOADS; ++i) {
        const int e = threadIdx.x + i * threads;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < KC * CX && k0 + e / CX < ke && col0 + e % CX * 4 < N) v = *(const float4*)(b + e / CX * N + e % CX * 4);
        br[4 * i] = v.x, br[4 * i + 1] = v.y, br[4 * i + 2] = v.z, br[4 * i + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < BLOADS; ++i) {
        const int e = threadIdx.x + i * threads;
        br[i] = e < KC * CT && k0 + e / CT < ke && col0 + e % CT < N ? b[e / CT * N + e % CT] : 0.f;
      }
    }
  };
  auto put = [&](float* As) {
    float* const Bs = As + rows * PITCH;
#pragma unroll
    for (int i = 0; i < ALOADS; ++i) As[(lr + i * lstep) * PITCH + lk] = ar[i];
    if constexpr (B16) {
#pragma unroll
      for (int i = 0; i < BLOADS; ++i) {
        const int e = threadIdx.x + i * threads;
        if (e < KC * CX) *(float4*)(Bs + e * 4) = make_float4(br[4 * i], br[4 * i + 1], br[4 * i + 2], br[4 * i + 3]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < BLOADS; ++i) {
        const int e = threadIdx.x + i * threads;
        if (e < KC * CT) Bs[e] = br[i];
      }
    }
  };

  float acc[RPT][4];
#pragma unroll
  for (int i = 0; i < RPT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  int now = 0;
  if (kb < ke) {
    fetch(kb);
    put(sm);
    __syncthreads();
  }
  for (int64_t k0 = kb; k0 < ke; k0 += KC) {
    const bool more = k0 + KC < ke;
    if (more) fetch(k0 + KC);
    const float* As = sm + now * buffer;
    const float* b = As + rows * PITCH + tx * 4;
#pragma unroll
    for (int kk = 0; kk < KC; kk += 4) {
      float4 av[RPT];
#pragma unroll
      for (int i = 0; i < RPT; ++i) av[i] = *(const float4*)(As + (ty + i * groups) * PITCH + kk);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 bv = *(const float4*)(b + (kk + q) * CT);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const float x = q == 0 ? av[i].x : q == 1 ? av[i].y : q == 2 ? av[i].z : av[i].w;
          acc[i][0] = fmaf(x, bv.x, acc[i][0]);
          acc[i][1] = fmaf(x, bv.y, acc[i][1]);
          acc[i][2] = fmaf(x, bv.z, acc[i][2]);
          acc[i][3] = fmaf(x, bv.w, acc[i][3]);
        }
      }
    }
    now ^= 1;
    if (more) put(sm + now * buffer);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int64_t r = row0 + ty + i * groups;
    if (r >= M) continue;
    const float bv = bias && !partial ? bias_scale * bias[r] : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t c = col0 + tx * 4 + j;
      if (c >= N) continue;
      if (partial) {
        partial[((int64_t)blockIdx.z * M + r) * N + c] = acc[i][j];
        continue;
      }
      float v = alpha * acc[i][j] + bv;
      if (row_scale) v *= row_scale[r];
      if (accumulate) v += out[r * N + c];
      out[r * N + c] = v;
    }
  }
}

using F32Kernel = void (*)(int64_t, int64_t, int64_t, float, const float*, const float*, const float*, float, const float*,
                           float*, int, int64_t, float*);
template <int CX, int RPT, int THREADS>
F32Kernel f32_kernel(bool b16) {
  return b16 ? gemm_f32_kernel<CX, RPT, THREADS, true> : gemm_f32_kernel<CX, RPT, THREADS, false>;
}
int gemm_f32(unsigned splits, int64_t m, int64_t n, int64_t k, float alpha, const void* A, const void* B,
             const void* bias, float bias_scale, const void* row_scale, void* out, int accumulate, int64_t k_chunk,
             void* partial, cudaStream_t st) {
  const bool b16 = n % 4 == 0 && ((uintptr_t)B & 15) == 0;
  const bool few = n <= F32_FEW_COLUMNS;
  const int rpt = few ? f32_offsets_fit(F32_FEW_ROWS, k) : f32_rows_per_thread(m, n, k);
  if (rpt == 0) {
    const dim3 tiles((unsigned)((n + BN - 1) / BN), (unsigned)((m + BM - 1) / BM), splits);
    gemm_kernel<float><<<tiles, 256, 0, st>>>(m, n, k, alpha, (const float*)A, (const float*)B, (const float*)bias,
                                              bias_scale, (const float*)row_scale, (float*)out, accumulate, k_chunk,
                                              (float*)partial);
    return check_launch("gemm_kernel");
  }
  F32Kernel kern;
  int rows, columns, threads;
  if (few) {
    // one model or a few chains: a thread per row, no columns of padding
    // (14000 x 60, one column: 11.2 us with 64-column tiles, 3.3 us)
    kern = f32_kernel<1, 1, 64>(b16);
    rows = F32_FEW_ROWS, columns = F32_FEW_COLUMNS, threads = 64;
  } else {
    kern = rpt == 9   ? f32_kernel<8, 9, 128>(b16)
           : rpt == 8 ? f32_kernel<8, 8, 128>(b16)
           : rpt == 6 ? f32_kernel<8, 6, 128>(b16)
           : rpt == 4 ? f32_kernel<8, 4, 128>(b16)
                      : f32_kernel<8, 2, 128>(b16);
    rows = 16 * rpt, columns = 32, threads = 128;
  }
  const dim3 grid((unsigned)((n + columns - 1) / columns), (unsigned)((m + rows - 1) / rows), splits);
  kern<<<grid, threads, 0, st>>>(m, n, k, alpha, (const float*)A, (const float*)B, (const float*)bias, bias_scale,
                                 (const float*)row_scale, (float*)out, accumulate, k_chunk, (float*)partial);
  return check_launch("gemm_f32_kernel");
}

// The same product for a handful of FP64 columns (one model, a few chains): a
// warp per row of A and NC columns, its lanes striding over k, so every row
// of A streams coalesced and 1000 rows occupy the chip, where the tile kernel
// above has 16 blocks that multiply 64-column tiles of padding.  d = 1000, one
// column, matrix from HBM: 14.2 us against 1180 us with the tile kernel; d = 50:
// 4.2 us against 75 us.
constexpr int GEMV_WARPS = 4;
template <typename T, int NC>
__global__ void __launch_bounds__(32 * GEMV_WARPS) gemv_kernel(int64_t M, int64_t N, int64_t K, T alpha,
                                                               const T* __restrict__ A, const T* __restrict__ B,
                                                               const T* __restrict__ bias, T bias_scale,
                                                               const T* __restrict__ row_scale, T* out,
                                                               int accumulate) {
  const int lane = threadIdx.x & 31;
  const int64_t r = blockIdx.x * (int64_t)GEMV_WARPS + (threadIdx.x >> 5);
  const int64_t c0 = blockIdx.y * (int64_t)NC;
  if (r >= M) return;
  const T* __restrict__ a = A + r * K;
  const T* __restrict__ b = B + c0;
  T acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = (T)0;
#pragma unroll 8
  for (int64_t k = lane; k < K; k += 32) {
    const T av = a[k];
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (NC == 1 || c0 + c < N) acc[c] += av * b[k * N + c];
  }
#pragma unroll
  for (int c = 0; c < NC; ++c)
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  T mine = acc[0];  // lane c finishes column c
#pragma unroll
  for (int c = 1; c < NC; ++c) mine = lane == c ? acc[c] : mine;
  if (lane >= NC || c0 + lane >= N) return;
  T v = alpha * mine + (bias ? bias_scale * bias[r] : (T)0);
  if (row_scale) v *= row_scale[r];
  T* o = out + r * N + c0 + lane;
  *o = accumulate ? *o + v : v;
}

template <typename T, int NC>
int gemv(int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B, const void* bias,
         double bias_scale, const void* row_scale, void* out, int accumulate, cudaStream_t st) {
  const dim3 grid((unsigned)((m + GEMV_WARPS - 1) / GEMV_WARPS), (unsigned)((n + NC - 1) / NC));
  gemv_kernel<T, NC><<<grid, 32 * GEMV_WARPS, 0, st>>>(m, n, k, (T)alpha, (const T*)A, (const T*)B, (const T*)bias,
                                                       (T)bias_scale, (const T*)row_scale, (T*)out, accumulate);
  return check_launch("gemv_kernel");
}

}  // namespace

// out = (alpha * A B + bias_scale * bias[m]) * row_scale[m] + (accumulate ? out : 0)
int gemm_ex(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B, const void* bias,
            double bias_scale, const void* row_scale, void* out, int accumulate, cudaStream_t stream) {
  HMC_REQUIRE(m >= 0 && n >= 0 && k >= 0, "hmc_gemm: negative size");
  if (m == 0 || n == 0) return HMC_OK;
  HMC_REQUIRE(A && B && out, "hmc_gemm: null operand");
  HMC_REQUIRE((n + BN - 1) / BN <= 0x7FFFFFFF && (m + BM - 1) / BM <= GRID_ROWS, "hmc_gemm: matrix too large");
  const dim3 grid((unsigned)((n + BN - 1) / BN), (unsigned)((m + BM - 1) / BM));
  const int64_t kc = k > 0 ? k : 1;
  // (FP64 only: FP32 sums keep their order in k)
  if (dtype == HMC_F64 && f64_by_rows(m, n, k)) {
    if (n == 1) return gemv<double, 1>(m, n, k, alpha, A, B, bias, bias_scale, row_scale, out, accumulate, stream);
    if (n <= 4) return gemv<double, 4>(m, n, k, alpha, A, B, bias, bias_scale, row_scale, out, accumulate, stream);
    return gemv<double, 8>(m, n, k, alpha, A, B, bias, bias_scale, row_scale, out, accumulate, stream);
  }
  if (dtype == HMC_F32)
    return gemm_f32(1, m, n, k, (float)alpha, A, B, bias, (float)bias_scale, row_scale, out, accumulate,
                    kc, nullptr, stream);
  if (dtype == HMC_F64)
    gemm_kernel<double><<<grid, 256, 0, stream>>>(m, n, k, alpha, (const double*)A, (const double*)B,
                                                   (const double*)bias, bias_scale, (const double*)row_scale,
                                                   (double*)out, accumulate, kc, nullptr);
  else
    return fail(HMC_ERR_INVALID_ARG, "hmc_gemm: unknown dtype %d", dtype);
  return check_launch("gemm_kernel");
}

int gemm_splitk(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B, void* out,
                int accumulate, void* work, int64_t work_elems, cudaStream_t stream) {
  HMC_REQUIRE(m >= 0 && n >= 0 && k >= 0, "hmc_gemm_splitk: negative size");
  if (m == 0 || n == 0) return HMC_OK;
  HMC_REQUIRE(A && B && out && work, "hmc_gemm_splitk: null operand");
  HMC_REQUIRE(work_elems >= m * n, "hmc_gemm_splitk: work holds fewer than m * n elements");
  HMC_REQUIRE(dtype == HMC_F32 || dtype == HMC_F64, "hmc_gemm_splitk: unknown dtype %d", dtype);
  HMC_REQUIRE((m + BM - 1) / BM <= GRID_ROWS, "hmc_gemm_splitk: matrix too large");
  const int64_t tiles = ((n + BN - 1) / BN) * ((m + BM - 1) / BM);
  // about four CTAs per SM in total, at least 256 k per split
  int64_t splits = (4 * 152 + tiles - 1) / tiles;
  const int64_t by_k = (k + 255) / 256;
  const int64_t by_work = work_elems / (m * n);
  splits = splits < by_k ? splits : by_k;
  splits = splits < by_work ? splits : by_work;
  splits = splits < 65535 ? splits : 65535;
  splits = splits > 1 ? splits : 1;
  int64_t chunk = k > 0 ? (k + splits - 1) / splits : 1;
  chunk = (chunk + BK - 1) / BK * BK;
  splits = k > 0 ? (k + chunk - 1) / chunk : 1;
  const dim3 grid((unsigned)((n + BN - 1) / BN), (unsigned)((m + BM - 1) / BM), (unsigned)splits);
  const unsigned rblocks = blocks_for(m * n, 256) < 152u * 8u ? blocks_for(m * n, 256) : 152u * 8u;
  if (dtype == HMC_F32) {
    HMC_TRY(gemm_f32((unsigned)splits, m, n, k, 1.f, A, B, nullptr, 0.f, nullptr, nullptr, 0, chunk, work,
                     stream));
    splitk_reduce_kernel<float><<<rblocks, 256, 0, stream>>>(m * n, (int)splits, (float)alpha, (const float*)work,
                                                            (float*)out, accumulate);
  } else {
    gemm_kernel<double><<<grid, 256, 0, stream>>>(m, n, k, 1.0, (const double*)A, (const double*)B, nullptr, 0.0,
                                                   nullptr, nullptr, 0, chunk, (double*)work);
    HMC_TRY(check_launch("gemm_kernel (split k)"));
    splitk_reduce_kernel<double><<<rblocks, 256, 0, stream>>>(m * n, (int)splits, alpha, (const double*)work,
                                                             (double*)out, accumulate);
  }
  return check_launch("splitk_reduce_kernel");
}

int gemm_dispatch(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B,
                  const void* bias, void* out, int accumulate, cudaStream_t stream) {
  return gemm_ex(dtype, m, n, k, alpha, A, B, bias, 1.0, nullptr, out, accumulate, stream);
}

}  // namespace hmc

extern "C" int hmc_gemm(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A, const void* B,
                        const void* bias, void* out, int accumulate, void* stream) {
  return hmc::gemm_dispatch(dtype, m, n, k, alpha, A, B, bias, out, accumulate, hmc::as_stream(stream));
}

extern "C" int hmc_gemm_splitk(int dtype, int64_t m, int64_t n, int64_t k, double alpha, const void* A,
                               const void* B, void* out, int accumulate, void* work, int64_t work_elems,
                               void* stream) {
  return hmc::gemm_splitk(dtype, m, n, k, alpha, A, B, out, accumulate, work, work_elems, hmc::as_stream(stream));
}
