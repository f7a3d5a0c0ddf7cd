// Strided SIMT GEMM with fp32 accumulation.  It is the matrix multiply of the fp32 build
// (the reference's Float32 path, src/gpt.jl:23-31) and of shapes the tcgen05 kernel does not
// take (row pitches that are not multiples of 16 bytes, e.g. the 12 -> n_kv_head gate).
//
// 64 threads have a 64 x 64 tile, 8 x 8 results each as pairs (two multiply-adds an instruction): a step of k takes 32 of those
// for four 16-byte loads from shared memory, which bound it (L1 68 % busy, fp32 pipe 34 %).  With so small a block even
// 600 x 512 results are enough blocks once K is shared out: up to eight blocks of a cluster take ranges of K, and each adds
// its share of the rows over the cluster's partial tiles, in order.  The next 16 steps of k are in registers while these run.
// Newton-Schulz of four 512 x 2048 fp32 matrices: 22 TFLOP/s; a training step of 600 tokens, 512 wide (126 products): 14.4 ms
// in them with 4 x 4 results a thread, scalar loads, one block a tile and nothing in flight (12 TFLOP/s), 7.9 ms so.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace {

constexpr int TM = 64, TN = 64, TK = 16, THREADS = 64;

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

// A 64 x 16 piece of an operand: 16 elements a thread, into registers and from there to shared memory as [k][64].
template <typename T> struct Piece {
  float4 r[4];
  // rows r0.. of n, steps k0.. up to k1
  __device__ __forceinline__ void load(const T* p, long long ld, bool kmajor, bool vec, int r0, int n, int k0, int k1) {
    const int t = threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int row = kmajor ? r0 + t : r0 + (t & 15) * 4, k = kmajor ? k0 + 4 * i : k0 + (t >> 4) + 4 * i;
      const int left = kmajor ? (row < n ? k1 - k : 0) : (k < k1 ? n - row : 0);
      r[i] = load4<T>(p + (kmajor ? (long long)row * ld + k : (long long)k * ld + row), vec, left);
    }
  }
  __device__ __forceinline__ void store(float (*s)[TM], bool kmajor) const {
    const int t = threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (kmajor) {
        s[4 * i][t] = r[i].x; s[4 * i + 1][t] = r[i].y; s[4 * i + 2][t] = r[i].z; s[4 * i + 3][t] = r[i].w;
      } else {
        *reinterpret_cast<float4*>(&s[(t >> 4) + 4 * i][(t & 15) * 4]) = r[i];
      }
    }
  }
};

__device__ __forceinline__ float4 cluster_load4(const float* p, int rank) {
  uint32_t at;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(sm100::smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}

// The rows of blockIdx.y's tile, the columns of blockIdx.x / S's; block blockIdx.x % S of the cluster has a range of K.
template <typename T>
__global__ void __launch_bounds__(THREADS) gemm_simt_kernel(const GemmArgs g, int S, bool vec_a, bool vec_b) {
  pdl_trigger();
  __shared__ __align__(16) float tiles[2][2][TK][TM];       // A and B, two pieces each; afterwards the tile's partial sums
  const int bz = blockIdx.z, rank = blockIdx.x % S;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x / S * TN;
  pdl_wait();
  if (g.upper_only && m0 >= n0 + TN) return;                // the whole cluster
  int bb = bz;
  if (g.groups) {      // runs of rows are multiples of TM
    const int run = m0 / g.group_rows;
    if (run >= g.groups[0]) return;
    bb = g.groups[1 + run];
  }
  const T* A = reinterpret_cast<const T*>(g.A) + (long long)bz * g.strideA;
  const T* B = reinterpret_cast<const T*>(g.B) + (long long)bb * g.strideB;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int per = ((g.K + TK - 1) / TK + S - 1) / S * TK, k_begin = rank * per, k_end = min(g.K, k_begin + per);
  uint64_t acc[8][4] = {};       // rows 4 ty.. and 32 + 4 ty.., columns 4 tx.. and 32 + 4 tx.. in pairs
  Piece<T> pa, pb;
  auto load = [&](int k) {
    pa.load(A, g.lda, g.a_kmajor, vec_a, m0, g.M, k, k_end);
    pb.load(B, g.ldb, g.b_kmajor, vec_b, n0, g.N, k, k_end);
  };
  if (k_begin < k_end) load(k_begin);
  int at = 0;
  for (int k = k_begin; k < k_end; k += TK, at ^= 1) {
    pa.store(tiles[at][0], g.a_kmajor);
    pb.store(tiles[at][1], g.b_kmajor);
    __syncthreads();           // the other two pieces are free: everybody has stored these after reading those
    if (k + TK < k_end) load(k + TK);
#pragma unroll
    for (int kk = 0; kk < TK; kk++) {
      const float4 a0 = *reinterpret_cast<const float4*>(&tiles[at][0][kk][4 * ty]), a1 = *reinterpret_cast<const float4*>(&tiles[at][0][kk][32 + 4 * ty]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&tiles[at][1][kk][4 * tx]), b1 = *reinterpret_cast<const ulonglong2*>(&tiles[at][1][kk][32 + 4 * tx]);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint64_t aa = sm100::pack2(a[i], a[i]);
        acc[i][0] = sm100::fma2(aa, b0.x, acc[i][0]); acc[i][1] = sm100::fma2(aa, b0.y, acc[i][1]);
        acc[i][2] = sm100::fma2(aa, b1.x, acc[i][2]); acc[i][3] = sm100::fma2(aa, b1.y, acc[i][3]);
      }
    }
  }
  __syncthreads();
  float* sum = &tiles[0][0][0][0];       // [64][64]
#pragma unroll
  for (int i = 0; i < 8; i++) {
    float* row = sum + ((i >> 2) * 32 + 4 * ty + (i & 3)) * TN;
    *reinterpret_cast<ulonglong2*>(row + 4 * tx) = make_ulonglong2(acc[i][0], acc[i][1]);
    *reinterpret_cast<ulonglong2*>(row + 32 + 4 * tx) = make_ulonglong2(acc[i][2], acc[i][3]);
  }
  if (S > 1) { sm100::cluster_arrive(); sm100::cluster_wait(); }
  else __syncthreads();

  T* C = reinterpret_cast<T*>(g.C) + (long long)bz * g.strideC;
  float* Cf = reinterpret_cast<float*>(g.C) + (long long)bz * g.strideC;
  const T* aux = reinterpret_cast<const T*>(g.aux) + (long long)bz * g.strideAux;
  const bool both = g.upper_only && m0 < n0;       // the tile below the diagonal is this one transposed
  auto put = [&](int m, int n, T v) {
    C[(long long)m * g.ldc + n] = v;
    if (both) C[(long long)n * g.ldc + m] = v;
  };
  const int rows = TM / S;
  for (int o = tid; o < rows * (TN / 4); o += THREADS) {
    const int r = rank * rows + o / (TN / 4), m = m0 + r, c = o % (TN / 4) * 4;
    float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < S; q++) {
      const float4 p = S > 1 ? cluster_load4(sum + r * TN + c, q) : *reinterpret_cast<const float4*>(sum + r * TN + c);
      v4.x += p.x; v4.y += p.y; v4.z += p.z; v4.w += p.w;
    }
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
  if (S > 1) { sm100::cluster_arrive(); sm100::cluster_wait(); }      // nobody leaves while its sums are read
}

}  // namespace

template <typename T> int gemm_simt(const GemmArgs& g, cudaStream_t s) {
  if (g.epi > EPI_F32) return femto_fail(FEMTO_ERR_UNSUPPORTED, "gemm_simt: epilogue %d needs the tensor-core path", g.epi);
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return femto_fail(FEMTO_ERR_SHAPE, "gemm_simt: empty problem");
  // 16-byte (bf16: 8-byte) loads where every group of four elements starts on such a boundary
  const uintptr_t mask = 4 * sizeof(T) - 1;
  const bool vec_a = ((uintptr_t)g.A & mask) == 0 && ((g.lda | g.strideA) & 3) == 0;
  const bool vec_b = ((uintptr_t)g.B & mask) == 0 && ((g.ldb | g.strideB) & 3) == 0;
  // K goes to as many blocks as bring about four to every multiprocessor, with at least 128 steps for each
  const long long tiles = (long long)cdiv(g.N, TN) * cdiv(g.M, TM) * g.batch;
  int S = 1;
  while (S < 8 && tiles * S < 4ll * device_sm_count() && g.K >= 2 * S * 128) S *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cdiv(g.N, TN) * S, cdiv(g.M, TM), g.batch); cfg.blockDim = THREADS; cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = S; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = S > 1 ? 2 : 1;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_simt_kernel<T>, g, S, vec_a, vec_b));
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
