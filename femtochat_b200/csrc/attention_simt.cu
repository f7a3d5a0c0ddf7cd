// Plain SIMT attention (forward and reverse) for any head_dim <= 256 and any dtype.  It serves
// the fp32 build (the reference's Float32 path, src/kernels.jl:131-219,287-379) and head sizes
// the tcgen05 kernels do not take.  One warp owns one output row, keys are visited in order, so
// results are deterministic.  Mask: key k is visible to query t iff t-left <= k <= t
// (src/kernels.jl:38) and, with doc_start, k >= doc_start[t].
#include "common.cuh"

namespace {

// elements per lane (EPL): head_dim <= 32 EPL, 1, 2, 4 or 8
// A row visits its keys (a key its queries) U at a time: the dot products, their sums over the warp and the exponentials of U
// keys do not wait for one another.  What a row sums it sums key by key all the same, rescaled at every key as if these came one at a
// time, each operation written out so that no compiler contracts it otherwise: the results of a training step do not depend on U.
// Time: 3 x 200 tokens, 4 heads of 128 in fp32, one key at a time 175 us (forward), 99 (dQ), 162 (dK, dV); so 56, 91, 109 us.
constexpr int U = 4;

template <typename T, int EPL>
__global__ void __launch_bounds__(128) attn_fwd_simt_kernel(AttnArgs a) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t = blockIdx.x * 4 + warp, h = blockIdx.y, b = blockIdx.z;
  if (t >= a.T) return;
  const int kvh = h / (a.H / a.Hkv);
  const int hd = a.hd;
  const float scale = rsqrtf((float)hd);
  const T* q = reinterpret_cast<const T*>(a.Q) + ((long long)b * a.T + t) * a.q_stride + (long long)h * hd;
  float qv[EPL], acc[EPL];
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    qv[e] = d < hd ? to_f<T>(q[d]) : 0.f;
    acc[e] = 0.f;
  }
  int k0 = max(0, t - a.window_left);
  if (a.doc_start) k0 = max(k0, a.doc_start[(long long)b * a.T + t]);
  float m = -INFINITY, l = 0.f;
  const T* kb = reinterpret_cast<const T*>(a.K) + (long long)b * a.T * a.kv_stride + (long long)kvh * hd;
  const T* vb = reinterpret_cast<const T*>(a.V) + (long long)b * a.T * a.kv_stride + (long long)kvh * hd;
  for (int k = k0; k <= t; k += U) {
    float s[U], v[U][EPL];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long long at = min(k + u, t) * a.kv_stride;      // past the end: the last key again, with no weight
      s[u] = 0.f;
#pragma unroll
      for (int e = 0; e < EPL; e++) {
        const int d = lane + 32 * e;
        if (d < hd) s[u] = fmaf(qv[e], to_f<T>(kb[at + d]), s[u]);
        v[u][e] = d < hd ? to_f<T>(vb[at + d]) : 0.f;
      }
    }
    // the running maximum before each key; what follows from it is then independent but for the sums
    float mu[U + 1];
    mu[0] = m;
#pragma unroll
    for (int u = 0; u < U; u++) {
      s[u] = __fmul_rn(warp_sum(s[u]), scale);
      mu[u + 1] = k + u <= t ? fmaxf(mu[u], s[u]) : mu[u];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (k + u > t) break;
      const float alpha = expf(mu[u] - mu[u + 1]), p = expf(__fsub_rn(s[u], mu[u + 1]));
      l = fmaf(l, alpha, p);
#pragma unroll
      for (int e = 0; e < EPL; e++) acc[e] = fmaf(acc[e], alpha, __fmul_rn(p, v[u][e]));
    }
    m = mu[U];
  }
  T* o = reinterpret_cast<T*>(a.O) + ((long long)b * a.T + t) * a.o_stride + (long long)h * hd;
  float inv = 1.f / l;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    if (d < hd) o[d] = from_f<T>(acc[e] * inv);
  }
  if (lane == 0) {
    long long si = ((long long)b * a.H + h) * a.T + t;
    if (a.lse) a.lse[si] = m + logf(l);
    if (a.l) a.l[si] = l;
    if (a.m) a.m[si] = m;
  }
}

// dQ and the row term D = sum(dO*O): one warp per (b, h, query).
template <typename T, int EPL>
__global__ void __launch_bounds__(128) attn_bwd_dq_simt_kernel(AttnArgs a, float* Dbuf) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t = blockIdx.x * 4 + warp, h = blockIdx.y, b = blockIdx.z;
  if (t >= a.T) return;
  const int kvh = h / (a.H / a.Hkv);
  const int hd = a.hd;
  const float scale = rsqrtf((float)hd);
  const long long row = (long long)b * a.T + t;
  const T* q = reinterpret_cast<const T*>(a.Q) + row * a.q_stride + (long long)h * hd;
  const T* o = reinterpret_cast<const T*>(a.O) + row * a.o_stride + (long long)h * hd;
  const T* dO = reinterpret_cast<const T*>(a.dO) + row * a.do_stride + (long long)h * hd;
  float qv[EPL], dov[EPL], acc[EPL];
  float D = 0.f;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    qv[e] = d < hd ? to_f<T>(q[d]) : 0.f;
    dov[e] = d < hd ? to_f<T>(dO[d]) : 0.f;
    D = __fadd_rn(D, d < hd ? __fmul_rn(dov[e], to_f<T>(o[d])) : 0.f);
    acc[e] = 0.f;
  }
  D = warp_sum(D);
  const long long si = ((long long)b * a.H + h) * a.T + t;
  if (lane == 0) Dbuf[si] = D;
  const float lse = a.lse[si];
  int k0 = max(0, t - a.window_left);
  if (a.doc_start) k0 = max(k0, a.doc_start[row]);
  const T* kb = reinterpret_cast<const T*>(a.K) + (long long)b * a.T * a.kv_stride + (long long)kvh * hd;
  const T* vb = reinterpret_cast<const T*>(a.V) + (long long)b * a.T * a.kv_stride + (long long)kvh * hd;
  for (int k = k0; k <= t; k += U) {
    float s[U], dp[U], kv[U][EPL];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long long at = min(k + u, t) * a.kv_stride;
      s[u] = dp[u] = 0.f;
#pragma unroll
      for (int e = 0; e < EPL; e++) {
        const int d = lane + 32 * e;
        kv[u][e] = d < hd ? to_f<T>(kb[at + d]) : 0.f;
        s[u] = fmaf(qv[e], kv[u][e], s[u]);
        if (d < hd) dp[u] = fmaf(dov[e], to_f<T>(vb[at + d]), dp[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      s[u] = warp_sum(s[u]);
      dp[u] = warp_sum(dp[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (k + u > t) break;
      const float ds = expf(fmaf(s[u], scale, -lse)) * (dp[u] - D) * scale;
#pragma unroll
      for (int e = 0; e < EPL; e++) acc[e] = fmaf(ds, kv[u][e], acc[e]);
    }
  }
  T* dq = reinterpret_cast<T*>(a.dQ) + row * a.dq_stride + (long long)h * hd;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    if (d < hd) dq[d] = from_f<T>(a.accumulate ? to_f<T>(dq[d]) + acc[e] : acc[e]);
  }
}

// dK, dV: one warp per (b, kv head, key); loops over the heads of the GQA group and the queries
// that see this key, in order.
template <typename T, int EPL>
__global__ void __launch_bounds__(128) attn_bwd_dkv_simt_kernel(AttnArgs a, const float* Dbuf) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int k = blockIdx.x * 4 + warp, kvh = blockIdx.y, b = blockIdx.z;
  if (k >= a.T) return;
  const int g = a.H / a.Hkv;
  const int hd = a.hd;
  const float scale = rsqrtf((float)hd);
  const long long krow = (long long)b * a.T + k;
  const T* kp = reinterpret_cast<const T*>(a.K) + krow * a.kv_stride + (long long)kvh * hd;
  const T* vp = reinterpret_cast<const T*>(a.V) + krow * a.kv_stride + (long long)kvh * hd;
  float kv[EPL], vv[EPL], dk[EPL], dv[EPL];
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    kv[e] = d < hd ? to_f<T>(kp[d]) : 0.f;
    vv[e] = d < hd ? to_f<T>(vp[d]) : 0.f;
    dk[e] = 0.f;
    dv[e] = 0.f;
  }
  const long long t1 = min((long long)a.T - 1, (long long)k + a.window_left);
  for (int hh = 0; hh < g; hh++) {
    const int h = kvh * g + hh;
    for (long long t = k; t <= t1; t += U) {
      float qv[U][EPL], dov[U][EPL], s[U], dp[U], lse[U], Dt[U];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long long tu = min(t + u, t1), row = (long long)b * a.T + tu, si = ((long long)b * a.H + h) * a.T + tu;
        ok[u] = t + u <= t1 && !(a.doc_start && a.doc_start[row] > k);
        const T* q = reinterpret_cast<const T*>(a.Q) + row * a.q_stride + (long long)h * hd;
        const T* dO = reinterpret_cast<const T*>(a.dO) + row * a.do_stride + (long long)h * hd;
        lse[u] = a.lse[si];
        Dt[u] = Dbuf[si];
        s[u] = dp[u] = 0.f;
#pragma unroll
        for (int e = 0; e < EPL; e++) {
          const int d = lane + 32 * e;
          qv[u][e] = d < hd ? to_f<T>(q[d]) : 0.f;
          dov[u][e] = d < hd ? to_f<T>(dO[d]) : 0.f;
          s[u] = fmaf(qv[u][e], kv[e], s[u]);
          dp[u] = fmaf(dov[u][e], vv[e], dp[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        s[u] = warp_sum(s[u]);
        dp[u] = warp_sum(dp[u]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (!ok[u]) continue;
        const float p = expf(fmaf(s[u], scale, -lse[u])), ds = p * (dp[u] - Dt[u]) * scale;
#pragma unroll
        for (int e = 0; e < EPL; e++) {
          dk[e] = fmaf(ds, qv[u][e], dk[e]);
          dv[e] = fmaf(p, dov[u][e], dv[e]);
        }
      }
    }
  }
  T* dkp = reinterpret_cast<T*>(a.dK) + krow * a.dkv_stride + (long long)kvh * hd;
  T* dvp = reinterpret_cast<T*>(a.dV) + krow * a.dkv_stride + (long long)kvh * hd;
#pragma unroll
  for (int e = 0; e < EPL; e++) {
    int d = lane + 32 * e;
    if (d < hd) {
      dkp[d] = from_f<T>(a.accumulate ? to_f<T>(dkp[d]) + dk[e] : dk[e]);
      dvp[d] = from_f<T>(a.accumulate ? to_f<T>(dvp[d]) + dv[e] : dv[e]);
    }
  }
}

}  // namespace

#define FOR_WIDTH(hd, ...)                                        \
  do {                                                            \
    if ((hd) <= 32) { constexpr int EPL = 1; __VA_ARGS__; }       \
    else if ((hd) <= 64) { constexpr int EPL = 2; __VA_ARGS__; }  \
    else if ((hd) <= 128) { constexpr int EPL = 4; __VA_ARGS__; } \
    else { constexpr int EPL = 8; __VA_ARGS__; }                  \
  } while (0)
template <typename T> int attention_fwd_simt(const AttnArgs& a, cudaStream_t s) {
  if (a.hd > 256) return femto_fail(FEMTO_ERR_UNSUPPORTED, "attention: head_dim %d > %d", a.hd, 256);
  dim3 grid(cdiv(a.T, 4), a.H, a.B);
  FOR_WIDTH(a.hd, (attn_fwd_simt_kernel<T, EPL><<<grid, 128, 0, s>>>(a)));
  KERNEL_CHECK();
  return 0;
}
template <typename T> int attention_bwd_simt(const AttnArgs& a, cudaStream_t s) {
  if (a.hd > 256) return femto_fail(FEMTO_ERR_UNSUPPORTED, "attention: head_dim %d > %d", a.hd, 256);
  size_t need = sizeof(float) * (size_t)a.B * a.H * a.T;
  if (!a.ws || a.ws_bytes < need) return femto_fail(FEMTO_ERR_ARG, "attention_bwd: workspace too small");
  float* D = reinterpret_cast<float*>(a.ws);
  dim3 grid(cdiv(a.T, 4), a.H, a.B);
  FOR_WIDTH(a.hd, (attn_bwd_dq_simt_kernel<T, EPL><<<grid, 128, 0, s>>>(a, D)));
  KERNEL_CHECK();
  dim3 grid2(cdiv(a.T, 4), a.Hkv, a.B);
  FOR_WIDTH(a.hd, (attn_bwd_dkv_simt_kernel<T, EPL><<<grid2, 128, 0, s>>>(a, D)));
  KERNEL_CHECK();
  return 0;
}
template int attention_fwd_simt<float>(const AttnArgs&, cudaStream_t);
template int attention_fwd_simt<bf16>(const AttnArgs&, cudaStream_t);
template int attention_bwd_simt<float>(const AttnArgs&, cudaStream_t);
template int attention_bwd_simt<bf16>(const AttnArgs&, cudaStream_t);

template <> int attention_fwd<float>(const AttnArgs& a, cudaStream_t s) { return attention_fwd_simt<float>(a, s); }
template <> int attention_bwd<float>(const AttnArgs& a, cudaStream_t s) { return attention_bwd_simt<float>(a, s); }
// A training step whose length does not fill the 128-row tiles stays with these kernels, forward and reverse: they keep P and dS in
// fp32, where the tensor cores multiply bf16 parts of them.  The difference is below a bf16 rounding of O, but a training step
// magnifies it: single elements of a table's gradient by more than the rms of the table after a few updates.  (5 x 1000 tokens, 6 heads:
// 1.7 ms forward, 2.0 and 2.3 reverse here; 0.03, 0.03 and 0.05 on the tensor cores.)
template <> int attention_fwd<bf16>(const AttnArgs& a, cudaStream_t s) {
  if (attention_tc_supported(a) && (attention_whole_tiles(a) || !a.reverse_follows)) return attention_fwd_tc(a, s);
  return attention_fwd_simt<bf16>(a, s);
}
template <> int attention_bwd<bf16>(const AttnArgs& a, cudaStream_t s) {
  if (attention_tc_supported(a) && attention_whole_tiles(a)) return attention_bwd_tc(a, s);
  return attention_bwd_simt<bf16>(a, s);
}
