// Strided SIMT GEMM with fp32 accumulation.  It is the matrix multiply of the fp32 build
// (the reference's Float32 path, src/gpt.jl:23-31) and of shapes the tcgen05 kernel does not
// take (row pitches that are not multiples of 16 bytes, e.g. the 12 -> n_kv_head gate).
//
// Every result is one chain of multiply-adds over k = 0, 1, ... in order, whatever the tile: a training step's results then are
// the same bits at every tile size.  (K shared by the blocks of a cluster, partial sums added at the end, was nearer to 64 bits, 5e-7 against 1.1e-6
// over a step, but over a dozen updates of the same weights two orders of summation drift 1e-4 apart.)
//
// 64 threads have a W x W tile, 8 x 8 (W = 64) or 4 x 4 (32) results each as pairs (two multiply-adds an instruction): at 64 a step of k
// takes 32 of those for four 16-byte loads from shared memory, which bound it.  The next steps of k are in registers while these run.
// A training step of 600 tokens, 512 wide, four layers (126 products, most of them Newton-Schulz): 15.6 ms with 4 x 4 results a thread,
// scalar loads and nothing in flight, 9.0 ms so; the introductory model (2 x 4 tokens, 32 wide) 1.45 -> 0.78 ms.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace {

constexpr int THREADS = 64;

// Four elements that follow each other in memory; those from `left` on are zero.
template <typename T> __device__ __forceinline__ float4 load4(const T* p, bool vec, int left) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec && left >= 4) {
    if constexpr (sizeof(T) == 4) {
      v = *reinterpret_cast<const float4*>(p);
    } else {
      const uint2 q = *reinterpret_cast<const uint2*>(p);
      v = make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u), __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xffff0000u));
    }
  } else {
    if (left > 0) v.x = to_f<T>(p[0]);
    if (left > 1) v.y = to_f<T>(p[1]);
    if (left > 2) v.z = to_f<T>(p[2]);
    if (left > 3) v.w = to_f<T>(p[3]);
  }
  return v;
}

// A W x TK piece of an operand in registers, and from there in shared memory as [k][W].  Of a k-contiguous operand, TK / 4 neighbouring
// lanes read the TK elements of a row (one row a lane would be 32 lines an instruction), and the transposing stores of a warp
// fall into 32 different banks because the columns of row k are permuted: m is at m ^ at(k).
template <typename T, int W, int TK> struct Piece {
  static constexpr int V = W * TK / (4 * THREADS), PER_M = TK / 4, PER_K = W / 4;      // lanes a row, a step of k
  float4 r[V];
  static __device__ __forceinline__ int at(int k) { return 32 / PER_M * (k >> 2); }
  static __device__ __forceinline__ int row(int i, bool kmajor) { return kmajor ? threadIdx.x / PER_M + THREADS / PER_M * i : threadIdx.x % PER_K * 4; }
  static __device__ __forceinline__ int step(int i, bool kmajor) { return kmajor ? threadIdx.x % PER_M * 4 : threadIdx.x / PER_K + THREADS / PER_K * i; }
  // rows r0.. of n, steps k0.. of K
  __device__ __forceinline__ void load(const T* p, long long ld, bool kmajor, bool vec, int r0, int n, int k0, int K) {
#pragma unroll
    for (int i = 0; i < V; i++) {
      const int m = r0 + row(i, kmajor), k = k0 + step(i, kmajor);
      const int left = kmajor ? (m < n ? K - k : 0) : (k < K ? n - m : 0);
      r[i] = load4<T>(p + (kmajor ? (long long)m * ld + k : (long long)k * ld + m), vec, left);
    }
  }
  __device__ __forceinline__ void store(float (*s)[W], bool kmajor) const {
#pragma unroll
    for (int i = 0; i < V; i++) {
      const int k = step(i, kmajor), m = row(i, kmajor) ^ at(k);
      if (kmajor) {
        s[k][m] = r[i].x; s[k + 1][m] = r[i].y; s[k + 2][m] = r[i].z; s[k + 3][m] = r[i].w;
      } else {
        *reinterpret_cast<float4*>(&s[k][m]) = r[i];
      }
    }
  }
};

template <typename T, int W, int TK>
__global__ void __launch_bounds__(THREADS) gemm_simt_kernel(const GemmArgs g, bool vec_a, bool vec_b) {
  pdl_trigger();
  __shared__ __align__(16) float tiles[2][2][TK][W];       // A and B, two pieces each; afterwards the tile's results
  constexpr int H = W / 32;                                // a thread's rows and columns: four of every 32
  const int bz = blockIdx.z;
  const int m0 = blockIdx.y * W, n0 = blockIdx.x * W;
  pdl_wait();
  if (g.upper_only && m0 > n0) return;
  int bb = bz;
  if (g.groups) {      // runs of rows are multiples of W
    const int run = m0 / g.group_rows;
    if (run >= g.groups[0]) return;
    bb = g.groups[1 + run];
  }
  const T* A = reinterpret_cast<const T*>(g.A) + (long long)bz * g.strideA;
  const T* B = reinterpret_cast<const T*>(g.B) + (long long)bb * g.strideB;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  uint64_t acc[4 * H][2 * H] = {};       // rows 4 ty.. of every 32, columns 4 tx.. of every 32 in pairs
  Piece<T, W, TK> pa, pb;
  auto load = [&](int k) {
    pa.load(A, g.lda, g.a_kmajor, vec_a, m0, g.M, k, g.K);
    pb.load(B, g.ldb, g.b_kmajor, vec_b, n0, g.N, k, g.K);
  };
  load(0);
  int at = 0;
  for (int k = 0; k < g.K; k += TK, at ^= 1) {
    pa.store(tiles[at][0], g.a_kmajor);
    pb.store(tiles[at][1], g.b_kmajor);
    __syncthreads();           // the other two pieces are free: everybody has stored these after reading those
    if (k + TK < g.K) load(k + TK);
#pragma unroll
    for (int q = 0; q < TK; q += 16) {
      if (q > 0 && k + q >= g.K) break;
#pragma unroll
      for (int kk = q; kk < q + 16; kk++) {
        float a[4 * H];
        uint64_t b[2 * H];
#pragma unroll
        for (int h = 0; h < H; h++) {
          const float4 v = *reinterpret_cast<const float4*>(&tiles[at][0][kk][32 * h + (4 * ty ^ Piece<T, W, TK>::at(kk))]);
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&tiles[at][1][kk][32 * h + (4 * tx ^ Piece<T, W, TK>::at(kk))]);
          a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
          b[2 * h] = w.x; b[2 * h + 1] = w.y;
        }
#pragma unroll
        for (int i = 0; i < 4 * H; i++) {
          const uint64_t aa = sm100::pack2(a[i], a[i]);
#pragma unroll
          for (int j = 0; j < 2 * H; j++) acc[i][j] = sm100::fma2(aa, b[j], acc[i][j]);
        }
      }
    }
  }
  __syncthreads();
  float* sum = &tiles[0][0][0][0];       // [W][W]
#pragma unroll
  for (int i = 0; i < 4 * H; i++)
#pragma unroll
    for (int h = 0; h < H; h++)
      *reinterpret_cast<ulonglong2*>(sum + ((i >> 2) * 32 + 4 * ty + (i & 3)) * W + 32 * h + 4 * tx) = make_ulonglong2(acc[i][2 * h], acc[i][2 * h + 1]);
  __syncthreads();

  T* C = reinterpret_cast<T*>(g.C) + (long long)bz * g.strideC;
  float* Cf = reinterpret_cast<float*>(g.C) + (long long)bz * g.strideC;
  const T* aux = reinterpret_cast<const T*>(g.aux) + (long long)bz * g.strideAux;
  const bool both = g.upper_only && m0 < n0;       // the tile below the diagonal is this one transposed
  auto put = [&](int m, int n, T v) {
    C[(long long)m * g.ldc + n] = v;
    if (both) C[(long long)n * g.ldc + m] = v;
  };
  for (int o = tid; o < W * W / 4; o += THREADS) {
    const int r = o / (W / 4), m = m0 + r, c = o % (W / 4) * 4;
    const float4 v4 = *reinterpret_cast<const float4*>(sum + r * W + c);
    if (m >= g.M) continue;
    const float e[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + c + j;
      if (n >= g.N) continue;
      const float v = e[j];
      switch (g.epi) {
        case EPI_STORE: put(m, n, from_f<T>(g.bias ? v + g.bias[n] : v)); break;
        case EPI_RESID:
          C[(long long)m * g.ldc + n] = from_f<T>(to_f<T>(aux[(long long)m * g.ldaux + n]) + v);
          break;
        case EPI_RELU2: { float r = fmaxf(v, 0.f); C[(long long)m * g.ldc + n] = from_f<T>(r * r); } break;
        case EPI_DRELU2:
          C[(long long)m * g.ldc + n] =
              from_f<T>(v * 2.f * sqrtf(fmaxf(to_f<T>(aux[(long long)m * g.ldaux + n]), 0.f)));
          break;
        case EPI_AXPBY: put(m, n, from_f<T>(g.alpha * to_f<T>(aux[(long long)m * g.ldaux + n]) + g.beta * v)); break;
        case EPI_F32: {
          float* dst;
          if (g.nseg == 0) {
            dst = Cf + (long long)m * g.ldc + n;
          } else {
            dst = nullptr;
            for (int s = 0; s < g.nseg; s++)
              if (n >= g.seg_col0[s] && n < g.seg_col0[s] + g.seg_ncol[s])
                dst = g.seg_ptr[s] + (long long)m * g.seg_ld[s] + (n - g.seg_col0[s]);
            if (!dst) break;
          }
          *dst = (g.beta != 0.f ? *dst : 0.f) + g.alpha * v;
        } break;
        default: break;
      }
    }
  }
}

}  // namespace

template <typename T> int gemm_simt(const GemmArgs& g, cudaStream_t s) {
  if (g.epi > EPI_F32) return femto_fail(FEMTO_ERR_UNSUPPORTED, "gemm_simt: epilogue %d needs the tensor-core path", g.epi);
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return femto_fail(FEMTO_ERR_SHAPE, "gemm_simt: empty problem");
  // 16-byte (bf16: 8-byte) loads where every group of four elements starts on such a boundary
  const uintptr_t mask = 4 * sizeof(T) - 1;
  const bool vec_a = ((uintptr_t)g.A & mask) == 0 && ((g.lda | g.strideA) & 3) == 0;
  const bool vec_b = ((uintptr_t)g.B & mask) == 0 && ((g.ldb | g.strideB) & 3) == 0;
  // Fewer than four blocks of two warps a multiprocessor leave it waiting: 32 x 32 tiles then.  The steps above take 12.5 and 1.19 ms with
  // 64 x 64 alone, 9.04 and 0.78 with 32 x 32 alone, 8.97 and 0.78 by this rule (10.1 and 0.78 with the line at one block).
  const long long tiles = (long long)cdiv(g.N, 64) * cdiv(g.M, 64) * g.batch / (g.upper_only ? 2 : 1);
  auto launch = [&](auto kernel, int W) { return launch_dependent(kernel, dim3(cdiv(g.N, W), cdiv(g.M, W), g.batch), dim3(THREADS), 0, s, g, vec_a, vec_b); };
  CUDA_TRY(tiles < 4ll * device_sm_count() ? launch(gemm_simt_kernel<T, 32, 32>, 32) : launch(gemm_simt_kernel<T, 64, 16>, 64));
  KERNEL_CHECK();
  return 0;
}
template int gemm_simt<float>(const GemmArgs&, cudaStream_t);
template int gemm_simt<bf16>(const GemmArgs&, cudaStream_t);

template <> int gemm<float>(const GemmArgs& g, cudaStream_t s) { return gemm_simt<float>(g, s); }
template <> int gemm<bf16>(const GemmArgs& g, cudaStream_t s) {
  if (gemm_tc_supported(g)) return gemm_tc_bf16(g, s);
  return gemm_simt<bf16>(g, s);
}
