// bf16 GEMM of few rows on the sm_100a tensor cores: narrow tiles, and K cut over the CTAs of a cluster.
//
// The persistent kernel (gemm_sm100.cu) makes tiles of 128 or 256 rows and 256 columns, each with all of K on one CTA or pair.  A
// prompt of some tens to some hundreds of rows has so few of them that most multiprocessors idle: 100 rows by 1280 columns are
// 5 tiles for 148 multiprocessors, and each of them streams 256 columns of the weight alone.  Here a tile is 128 rows by 64 or 128
// columns and a cluster of S CTAs shares it, each with a range of K.  The accumulators meet in shared memory: every
// CTA leaves its 128 x BN sums (fp32) in the ring it has emptied, and after a cluster barrier each adds up 1 / S of the rows over the
// S CTAs, in their order, and runs the epilogue on them.  Nothing goes through global memory, and the order of the sums depends on the
// shape alone.  One tile a cluster: no persistence, the next tile is the next cluster.
#include <algorithm>

#include "sm100_ptx.cuh"

using namespace sm100;

namespace {

constexpr int BM = 128, BK = 64, NTHREADS = 320, MAX_RING = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int RING_BYTES = 192 * 1024;

struct SplitParams {
  GemmArgs g;
  int bn, stages, kblocks, kb_per_cta;      // k-blocks of KS x 64
  uint32_t idesc;
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 cluster_load4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void prefetch_3d(const CUtensorMap* map, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void prefetch_4d(const CUtensorMap* map, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// Eight neighbouring results of a row.
// `aux`: the eight of the residual epilogue where they could be read as 16 bytes.
__device__ __forceinline__ const bf16* aux_of(const GemmArgs& g, long long bz, int m, int n) {
  return reinterpret_cast<const bf16*>(g.aux) + bz * g.strideAux + (long long)m * g.ldaux + n;
}
__device__ __forceinline__ void finish8(const GemmArgs& g, float (&v)[8], long long bz, int m, int n, const uint4& aux8) {
  const bool full = n + 8 <= g.N;
  if (g.epi == EPI_F32) {
    float* C = reinterpret_cast<float*>(g.C) + bz * g.strideC + (long long)m * g.ldc + n;
    const bool vec = full && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    if (vec) {
#pragma unroll
      for (int j = 0; j < 8; j += 4)
        *reinterpret_cast<float4*>(C + j) = make_float4(g.alpha * v[j], g.alpha * v[j + 1], g.alpha * v[j + 2], g.alpha * v[j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) if (n + j < g.N) C[j] = g.alpha * v[j];
    }
    return;
  }
  bf16* C = reinterpret_cast<bf16*>(g.C) + bz * g.strideC + (long long)m * g.ldc + n;
  if (g.epi == EPI_RESID) {
    const bf16* aux = aux_of(g, bz, m, n);
    if (full && (reinterpret_cast<uintptr_t>(aux) & 15) == 0) {
      const bf16* a = reinterpret_cast<const bf16*>(&aux8);
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = __bfloat162float(a[j]) + v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) if (n + j < g.N) v[j] = __bfloat162float(aux[j]) + v[j];
    }
  }
  if (g.epi == EPI_STORE && g.bias) {
#pragma unroll
    for (int j = 0; j < 8; j++) if (n + j < g.N) v[j] += __ldg(g.bias + n + j);
  }
  if (g.epi == EPI_RELU2) {
#pragma unroll
    for (int j = 0; j < 8; j++) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
  }
  if (full && (reinterpret_cast<uintptr_t>(C) & 15) == 0) store_vec<bf16, 8>(C, v);
  else {
#pragma unroll
    for (int j = 0; j < 8; j++) if (n + j < g.N) C[j] = __float2bfloat16_rn(v[j]);
  }
}

// S: CTAs of a cluster, which share K.  ACT: EPI_SWIGLU.
// KS: 64-wide slabs of K a stage; two arrive with one copy of either operand, which halves the handshakes of a stage.
template <bool B_K, int S, bool ACT, int KS>
__global__ void __launch_bounds__(NTHREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);      // the same offset in every CTA
  __shared__ uint64_t full[MAX_RING], empty[MAX_RING], tfull;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const GemmArgs& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int bn = p.bn, nt = blockIdx.x / S, mt = blockIdx.y, bz = blockIdx.z;
  const int m0 = mt * BM, n0 = nt * bn;
  const int kb0 = rank * p.kb_per_cta, kb1 = min(p.kblocks, kb0 + p.kb_per_cta);
  const uint32_t stage_bytes = KS * (A_BYTES + bn * BK * 2);

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(&tfull, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, bn); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  grid_launch_dependents();
  // The weights come from memory: ask L2 for them while the predecessor still runs (it is coherent, so what a predecessor has yet
  // to write is no harm).  Once: every row of tiles reads the same weights.
  if (!g.groups && mt == 0 && warp == 0 && lane == 0) {
    for (int kb = kb0; kb < min(kb1, kb0 + 16); kb++) {
      if (B_K && KS == 1) prefetch_3d(&tmB, kb * BK, n0, g.strideB ? bz : 0);
      else if (B_K) prefetch_4d(&tmB, 0, n0, kb * KS, g.strideB ? bz : 0);
      else prefetch_4d(&tmB, 0, kb * KS * BK, n0 / 64, g.strideB ? bz : 0);
    }
  }
  grid_dependency_wait();

  const bool live = !g.groups || mt < g.groups[0] * (g.group_rows / BM);      // the same in all CTAs of a cluster
  const int bb = g.groups ? (live ? g.groups[1 + m0 / g.group_rows] : 0) : g.strideB ? bz : 0;
  float* sums = reinterpret_cast<float*>(smem);
  const int pitch = bn + 4;      // 4: the rows that eight lanes store fall into different banks
  // a thread's groups of eight results of this CTA's rows: t, t + 256, ...
  const int rows = min(BM, g.M - m0), per = (rows + S - 1) / S, lo = rank * per, hi = min(rows, lo + per);
  const int groups = ACT ? bn / 16 : bn / 8, t = (int)threadIdx.x - 64, n_groups = (hi - lo) * groups;
  constexpr int AUX = 8 / S;      // most of them: 128 / S rows of 128 columns for 256 threads
  uint4 aux[AUX];
  if (live && t >= 0 && !ACT && g.epi == EPI_RESID) {      // read while the products run
#pragma unroll
    for (int q = 0; q < AUX; q++) {
      const int i = t + q * (NTHREADS - 64), n = n0 + i % groups * 8;
      if (i >= n_groups || n + 8 > g.N) continue;
      const bf16* from = aux_of(g, bz, m0 + lo + i / groups, n);
      if ((reinterpret_cast<uintptr_t>(from) & 15) == 0) aux[q] = *reinterpret_cast<const uint4*>(from);
    }
  }

  if (live) {
    // (the issuing warps run converged, as in the persistent kernel)
    if (warp == 0) {
      int stage = 0, n_issued = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, g.status)) break;
        uint8_t* sa = smem + stage * stage_bytes;
        if (elect_one()) {
          mbar_expect_tx(&full[stage], stage_bytes);
          uint8_t* sb = sa + KS * A_BYTES;
          if (KS == 1) tma_load_3d(sa, &tmA, &full[stage], kb * BK, m0, bz);
          else tma_load_4d(sa, &tmA, &full[stage], 0, m0, kb * KS, bz);
          if (B_K && KS == 1) tma_load_3d(sb, &tmB, &full[stage], kb * BK, n0, bb);
          else if (B_K) tma_load_4d(sb, &tmB, &full[stage], 0, n0, kb * KS, bb);
          else tma_load_4d(sb, &tmB, &full[stage], 0, kb * KS * BK, n0 / 64, bb);
        }
        __syncwarp();
        n_issued++;
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (*abort_flag)      // let loads in flight land before the CTA exits
        for (int i = max(0, n_issued - p.stages); i < n_issued; i++)
          for (uint32_t it = 0; it < WAIT_LIMIT && !mbar_try_wait(&full[i % p.stages], (i / p.stages) & 1); ++it) {}
    } else if (warp == 1) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait_warp(&full[stage], phase, abort_flag, g.status)) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * stage_bytes), sb = sa + KS * A_BYTES;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < KS * BK / 16; k++) {
            // K-contiguous: slabs of 64 k, [slab][row][64]; B's columns contiguous: slabs of 64 columns, [slab][k][64]
            const uint64_t ad = smem_desc_sw128(sa + (k >> 2) * A_BYTES + (k & 3) * 32, 16, 1024);
            const uint64_t bd = B_K ? smem_desc_sw128(sb + (k >> 2) * bn * 128 + (k & 3) * 32, 16, 1024) : smem_desc_sw128(sb + k * 2048, KS * 8192, 1024);
            mma_ss(tmem, ad, bd, p.idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          }
          tc_commit(&empty[stage]);
          if (kb + 1 == kb1) tc_commit(&tfull);
        }
        __syncwarp();
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    } else if (mbar_wait_warp(&tfull, 0, abort_flag, g.status)) {
      // every product of this CTA is done, so the ring is free for its sums
      tc_fence_after();
      const int quad = warp & 3, half = (warp - 2) >> 2, row = quad * 32 + lane;
      for (int c = half * (bn / 2); c < (half + 1) * (bn / 2); c += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + c + ((uint32_t)(quad * 32) << 16), r);
        tmem_ld_wait();
        if (m0 + row < g.M) {
          float4* dst = reinterpret_cast<float4*>(sums + row * pitch + c);
#pragma unroll
          for (int j = 0; j < 8; j++)
            dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
        }
      }
      tc_fence_before();
    }
    __syncwarp();
  }
  if (S > 1) { cluster_arrive(); cluster_wait(); } else __syncthreads();
  if (live && warp >= 2) {
    const uint32_t base = smem_u32(sums);
#pragma unroll
    for (int q = 0; q < AUX; q++) {
      const int i = t + q * (NTHREADS - 64);
      if (i >= n_groups) break;
      const int row = lo + i / groups, cg = i % groups;
      const int col = ACT ? (cg >> 2) * 64 + (cg & 3) * 8 : cg * 8;
      if (n0 + col >= g.N) continue;
      float v[8], u[8];
#pragma unroll
      for (int s = 0; s < S; s++) {
        const uint32_t at = (S > 1 ? map_to_rank(base, s) : base) + (row * pitch + col) * 4;
        const float4 a = cluster_load4(at), b = cluster_load4(at + 16);
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = s ? v[j] + f[j] : f[j];
        if constexpr (ACT) {
          const float4 c = cluster_load4(at + 128), e = cluster_load4(at + 144);
          const float h[8] = {c.x, c.y, c.z, c.w, e.x, e.y, e.z, e.w};
#pragma unroll
          for (int j = 0; j < 8; j++) u[j] = s ? u[j] + h[j] : h[j];
        }
      }
      if constexpr (ACT) {
        bf16* C = reinterpret_cast<bf16*>(g.C) + (long long)bz * g.strideC + (long long)(m0 + row) * g.ldc + (n0 + (cg >> 2) * 64) / 2 + (cg & 3) * 8;
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = v[j] * __fdividef(1.f, 1.f + __expf(-v[j])) * u[j];
        store_vec<bf16, 8>(C, v);
      } else {
        finish8(g, v, bz, m0 + row, n0 + col, aux[q]);
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  if (S > 1) { cluster_arrive(); cluster_wait(); } else __syncthreads();      // nobody leaves while a peer reads its sums
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, bn);
  }
}

template <bool B_K, int S, bool ACT, int KS>
int launch_split(const CUtensorMap& tmA, const CUtensorMap& tmB, const SplitParams& p, dim3 grid, size_t smem, cudaStream_t s) {
  static PerDevice attr;
  const int dev = PerDevice::current();
  if (dev < 0 || !attr.done[dev]) {
    CUDA_TRY(cudaFuncSetAttribute(gemm_split_kernel<B_K, S, ACT, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024));
    if (dev >= 0) attr.done[dev] = true;
  }
  CUDA_TRY(launch_dependent_clusters(gemm_split_kernel<B_K, S, ACT, KS>, S, grid, NTHREADS, smem, s, tmA, tmB, p));
  return 0;
}

}  // namespace

// CTAs of clusters of `splits` that run at once: clusters lie within a group of multiprocessors, so the larger leave some of them idle.
static int cluster_ctas(int splits) {
  if (splits == 1) return device_sm_count();
  static PerDevice pd[9];
  const int dev = PerDevice::current();
  if (dev >= 0 && pd[splits].done[dev]) return pd[splits].value[dev];
  auto kernel = splits == 2 ? gemm_split_kernel<false, 2, false, 2> : splits == 4 ? gemm_split_kernel<false, 4, false, 2> : gemm_split_kernel<false, 8, false, 2>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits); cfg.blockDim = dim3(NTHREADS); cfg.dynamicSmemBytes = RING_BYTES + 1024;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  if (dev >= 0) { pd[splits].value[dev] = n * splits; pd[splits].done[dev] = true; }
  return n * splits;
}

// What the kernel takes, beside what gemm_tc_supported() asks.
static bool split_supported(const GemmArgs& g) {
  if (!g.any_size || !g.a_kmajor || g.upper_only || g.nseg) return false;
  if (g.epi != EPI_STORE && g.epi != EPI_RESID && g.epi != EPI_RELU2 && g.epi != EPI_F32 && g.epi != EPI_SWIGLU) return false;
  if (g.epi == EPI_F32 && g.beta != 0.f) return false;      // sums of several products are a training step's
  return g.b_kmajor || !(g.N & 63);
}

// Tile width and cluster size, or false where the persistent kernel is the faster one.  Microseconds of either kernel back to back with
// weights from memory, fitted to 108 shapes (24 to 5000 rows, 768 to 6912 columns, K 768 to 5120; B200): a tile costs this
// kernel 4.2 + 0.225 a k-block of 64 (64 columns) or 5.4 + 0.29 (128), and 0.45 for every doubling of the cluster; the persistent one
// 5.6 + 0.33 a k-block of a wave, and 2 more for the residual of a CTA's only tile.  More tiles than run at once are the persistent
// kernel's.  Measured, before -> now: 24 x 2304 x 768 9.1 -> 5.3, 24 x 768 x 3072 24 -> 5.7, 100 x 1280 x 3456 25.5 -> 8.6,
// 600 x 1280 x 5120 31 -> 18.5, 1500 x 1280 x 1280 14.4 -> 12.5, 1500 x 1280 x 5120 31.8 -> 28.9.
bool gemm_split_plan(const GemmArgs& g, int* bn, int* splits) {
  if (!split_supported(g)) return false;
  const int kb = cdiv(g.K, BK), sms = device_sm_count();
  const bool pair = g.M >= 2 * BM;
  const long long tiles = (long long)cdiv(g.M, pair ? 2 * BM : BM) * cdiv(g.N, 256) * g.batch;
  const int waves = cdiv(tiles, pair ? sms / 2 : sms);
  double best = 0.95 * (5.6 + 0.33 * waves * kb + (g.epi == EPI_RESID && waves == 1 ? 2.0 : 0.0));
  bool found = false;
  for (int w = 64; w <= 128; w *= 2)
    for (int s = 1, doublings = 0; s <= (g.whole_k ? 1 : 8); s *= 2, doublings++) {
      const int stages = cdiv(g.K, 2 * BK), per = cdiv(stages, s);      // of two k-blocks
      if ((s - 1) * per >= stages || (long long)cdiv(g.M, BM) * cdiv(g.N, w) * g.batch * s > cluster_ctas(s)) continue;
      const double cost = (w == 64 ? 4.2 + 0.45 * per : 5.4 + 0.58 * per) + 0.45 * doublings;
      if (cost < best) { best = cost; *bn = w; *splits = s; found = true; }
    }
  return found;
}

// bn columns a tile (64, 128), K over a cluster of `splits` CTAs (1, 2, 4, 8).
int gemm_split_bf16(const GemmArgs& g, int bn, int splits, cudaStream_t s) {
  if (!gemm_tc_supported(g) || !split_supported(g)) return femto_fail(FEMTO_ERR_UNSUPPORTED, "gemm_split: shape/alignment not supported");
  SplitParams p;
  p.g = g;
  p.bn = bn;
  const int ks = g.K & 63 ? 1 : 2;      // a slab of 64 k must not reach into the next row
  p.kblocks = cdiv(g.K, ks * BK);
  p.kb_per_cta = cdiv(p.kblocks, splits);
  const int stage = ks * (A_BYTES + bn * BK * 2);
  p.stages = std::min({RING_BYTES / stage, MAX_RING, std::max(2, p.kb_per_cta)});
  p.idesc = idesc_bf16(BM, bn, false, !g.b_kmajor);
  const int nbB = g.groups ? g.n_groups : g.strideB ? g.batch : 1;
  CUtensorMap tmA, tmB;
  auto slabs = [&](CUtensorMap* m, const void* base, int rows, long long ld, int n, long long stride, int box) {      // [slab of 64 k][row][64]
    const uint64_t dims[4] = {64, (uint64_t)rows, (uint64_t)g.K / 64, (uint64_t)n}, st[3] = {(uint64_t)ld, 64, n > 1 ? (uint64_t)stride : (uint64_t)ld * rows};
    const uint32_t b[4] = {64, (uint32_t)box, (uint32_t)ks, 1};
    return make_tmap_nd_bf16(m, base, 4, dims, st, b);
  };
  if (ks == 1) FEMTO_TRY(make_tmap_3d_bf16(&tmA, g.A, g.K, g.M, g.batch, g.lda, g.strideA, BK, BM));
  else FEMTO_TRY(slabs(&tmA, g.A, g.M, g.lda, g.batch, g.strideA, BM));
  if (!g.b_kmajor) {
    if (make_tmap_4d_slabs_bf16(&tmB, g.B, g.N, g.K, nbB, g.ldb, g.strideB, ks * BK, bn / 64)) return femto_fail(FEMTO_ERR_ALIGN, "gemm_split: operand B");
  } else if (ks == 1) {
    FEMTO_TRY(make_tmap_3d_bf16(&tmB, g.B, g.K, g.N, nbB, g.ldb, g.strideB, BK, bn));
  } else {
    FEMTO_TRY(slabs(&tmB, g.B, g.N, g.ldb, nbB, g.strideB, bn));
  }
  const dim3 grid(cdiv(g.N, bn) * splits, cdiv(g.M, BM), g.batch);
  const size_t ring = (size_t)p.stages * stage, sums = (size_t)BM * (bn + 4) * 4, smem = std::max(ring, sums) + 1024;
  int r = 0;
#define LAUNCH2(S, KS) (g.epi == EPI_SWIGLU ? launch_split<true, S, true, KS>(tmA, tmB, p, grid, smem, s) \
                        : g.b_kmajor        ? launch_split<true, S, false, KS>(tmA, tmB, p, grid, smem, s) \
                                            : launch_split<false, S, false, KS>(tmA, tmB, p, grid, smem, s))
#define LAUNCH(S) (ks == 2 ? LAUNCH2(S, 2) : LAUNCH2(S, 1))
  {
    GemmSpan span(g, s);
    if (splits == 1) r = LAUNCH(1);
    else if (splits == 2) r = LAUNCH(2);
    else if (splits == 4) r = LAUNCH(4);
    else r = LAUNCH(8);
  }
#undef LAUNCH
#undef LAUNCH2
  FEMTO_TRY(r);
  KERNEL_CHECK();
  return 0;
}
