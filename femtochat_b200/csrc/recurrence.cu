// Recurrent token mixers with an fp32 matrix state per head: a decayed sum of outer products (lightning attention) and
// the gated delta rule with one decay per key channel.  The state is kept as [vdim][dim]: its vdim columns are independent
// recurrences that share q, k and the decays, so a block owns 32 of them, eight lanes each, for any number of tokens.
#include "decoder.cuh"
#include "sm100_ptx.cuh"

namespace {

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
// log(1 + e^z) without overflow or cancellation
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

template <int NI> struct Tile { static constexpr int TOK = NI >= 8 ? 8 : 16; };   // tokens staged at a time

// q / k / g of one head, v of this block's 32 columns and beta for `n` tokens from row `r0` into shared memory.
template <typename T, bool DELTA, int NI>
__global__ void __launch_bounds__(256) k_recurrence(const RecurrenceArgs a) {
  pdl_trigger();
  prefetch_l2(a.S + (((long long)blockIdx.z * a.heads + blockIdx.y) * a.vdim + blockIdx.x * 32) * a.dim, 4ll * a.dim * min(32, a.vdim - (int)blockIdx.x * 32),
              threadIdx.x, 256);
  pdl_wait();
  constexpr int DP = 32 * NI, TT = Tile<NI>::TOK;
  __shared__ __align__(16) float sq[TT][DP], sk[TT][DP], sg[DELTA ? TT : 1][DELTA ? DP : 4], sv[TT][32], sb[TT];
  const int h = blockIdx.y, b = blockIdx.z;
  const int lane = threadIdx.x & 31, sub = lane & 7, colb = (threadIdx.x >> 5) * 4 + (lane >> 3);
  const int e = blockIdx.x * 32 + colb;
  const int qh = h / (a.heads / a.qk_heads);
  const int D = a.dim, E = a.vdim;
  float* Sp = a.S + (((long long)b * a.heads + h) * E + min(e, E - 1)) * D;
  float s[NI * 4];
  const bool vec = (D & 3) == 0;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int d = 4 * (sub + 8 * i);
    if (vec) {
      const float4 v = e < E && d < D ? *reinterpret_cast<const float4*>(Sp + d) : make_float4(0.f, 0.f, 0.f, 0.f);
      s[i * 4] = v.x; s[i * 4 + 1] = v.y; s[i * 4 + 2] = v.z; s[i * 4 + 3] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) s[i * 4 + j] = (e < E && d + j < D) ? Sp[d + j] : 0.f;
    }
  }
  const float decay = DELTA ? 1.f : a.decay[h];
  for (int t0 = 0; t0 < a.T; t0 += TT) {
    const int n = min(TT, a.T - t0);
    const long long r0 = (long long)b * a.T + t0;
    __syncthreads();
    for (int i = threadIdx.x; i < n * DP; i += 256) {
      const int t = i / DP, d = i % DP;
      float q = 0.f, k = 0.f;
      if (d < D) {
        const long long iq = (r0 + t) * a.ldq + (long long)qh * D + d, ik = (r0 + t) * a.ldk + (long long)qh * D + d;
        if (DELTA) {
          q = reinterpret_cast<const float*>(a.q)[iq]; k = reinterpret_cast<const float*>(a.k)[ik];
        } else {
          q = silu_f(to_f<T>(reinterpret_cast<const T*>(a.q)[iq])); k = silu_f(to_f<T>(reinterpret_cast<const T*>(a.k)[ik]));
        }
      }
      sq[t][d] = q; sk[t][d] = k;
      if (DELTA) sg[t][d] = d < D ? a.g[(r0 + t) * ((long long)a.heads * D) + (long long)h * D + d] : 0.f;
    }
    for (int i = threadIdx.x; i < n * 32; i += 256) {
      const int t = i / 32, c = blockIdx.x * 32 + i % 32;
      float v = c < E ? to_f<T>(reinterpret_cast<const T*>(a.v)[(r0 + t) * a.ldv + (long long)h * E + c]) : 0.f;
      if (!DELTA) v = silu_f(v);
      sv[t][i % 32] = v;
    }
    if (DELTA && threadIdx.x < n) sb[threadIdx.x] = a.beta[(r0 + threadIdx.x) * a.heads + h];
    __syncthreads();
    for (int t = 0; t < n; t++) {
      float o = 0.f;
      if constexpr (DELTA) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const float4 g = *reinterpret_cast<const float4*>(&sg[t][4 * (sub + 8 * i)]), k = *reinterpret_cast<const float4*>(&sk[t][4 * (sub + 8 * i)]);
          s[i * 4] *= g.x; s[i * 4 + 1] *= g.y; s[i * 4 + 2] *= g.z; s[i * 4 + 3] *= g.w;
          dot += s[i * 4] * k.x; dot += s[i * 4 + 1] * k.y; dot += s[i * 4 + 2] * k.z; dot += s[i * 4 + 3] * k.w;
        }
        dot += __shfl_xor_sync(0xffffffffu, dot, 1); dot += __shfl_xor_sync(0xffffffffu, dot, 2); dot += __shfl_xor_sync(0xffffffffu, dot, 4);
        const float u = sb[t] * (sv[t][colb] - dot);
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const float4 k = *reinterpret_cast<const float4*>(&sk[t][4 * (sub + 8 * i)]), q = *reinterpret_cast<const float4*>(&sq[t][4 * (sub + 8 * i)]);
          s[i * 4] += k.x * u; s[i * 4 + 1] += k.y * u; s[i * 4 + 2] += k.z * u; s[i * 4 + 3] += k.w * u;
          o += s[i * 4] * q.x; o += s[i * 4 + 1] * q.y; o += s[i * 4 + 2] * q.z; o += s[i * 4 + 3] * q.w;
        }
      } else {
        const float u = sv[t][colb];
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const float4 k = *reinterpret_cast<const float4*>(&sk[t][4 * (sub + 8 * i)]), q = *reinterpret_cast<const float4*>(&sq[t][4 * (sub + 8 * i)]);
          s[i * 4] = decay * s[i * 4] + k.x * u; s[i * 4 + 1] = decay * s[i * 4 + 1] + k.y * u;
          s[i * 4 + 2] = decay * s[i * 4 + 2] + k.z * u; s[i * 4 + 3] = decay * s[i * 4 + 3] + k.w * u;
          o += s[i * 4] * q.x; o += s[i * 4 + 1] * q.y; o += s[i * 4 + 2] * q.z; o += s[i * 4 + 3] * q.w;
        }
      }
      o += __shfl_xor_sync(0xffffffffu, o, 1); o += __shfl_xor_sync(0xffffffffu, o, 2); o += __shfl_xor_sync(0xffffffffu, o, 4);
      if (sub == 0 && e < E) reinterpret_cast<T*>(a.o)[(r0 + t) * ((long long)a.heads * E) + (long long)h * E + e] = from_f<T>(o);
    }
  }
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int d = 4 * (sub + 8 * i);
    if (e >= E) continue;
    if (vec) {
      if (d < D) *reinterpret_cast<float4*>(Sp + d) = make_float4(s[i * 4], s[i * 4 + 1], s[i * 4 + 2], s[i * 4 + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) if (d + j < D) Sp[d + j] = s[i * 4 + j];
    }
  }
}

// Input x[t - back] of channel c: from this call's rows, or from the inputs kept of earlier calls (zeros before the start).
template <typename T>
__device__ __forceinline__ float conv_input(const DeltaPrepArgs& a, int b, int t, int back, int seg, int c, int chan, int channels) {
  const int r = t - back;
  if (r >= 0) return to_f<T>(reinterpret_cast<const T*>(a.proj)[((long long)b * a.T + r) * a.ldp + seg + c]);
  return to_f<T>(reinterpret_cast<const T*>(a.tail_in)[((long long)b * (a.taps - 1) + (a.taps - 1 + r)) * channels + chan]);
}

// One warp per unit: q head, k head (convolution, silu, unit vector), v head (convolution, silu), or the decays of a head.
template <typename T>
__global__ void __launch_bounds__(256) k_delta_prep(const DeltaPrepArgs a) {
  pdl_trigger();
  pdl_wait();
  const int units = 2 * a.kv_heads + 2 * a.heads;
  const long long it = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (it >= (long long)a.B * a.T * units) return;
  const int lane = threadIdx.x & 31;
  const long long row = it / units;
  int u = (int)(it % units);
  const int b = (int)(row / a.T), t = (int)(row % a.T);
  const int G = a.kv_heads, H = a.heads, D = a.dim, E = a.vdim, n = a.taps;
  const int channels = 2 * G * D + H * E;
  if (u < 2 * G + H) {
    const bool is_q = u < G, is_v = u >= 2 * G;
    const int head = is_q ? u : is_v ? u - 2 * G : u - G, size = is_v ? E : D;
    const int seg = is_q ? a.s_q : is_v ? a.s_v : a.s_k;
    const int chan0 = is_q ? 0 : is_v ? 2 * G * D : G * D;
    const float* taps = is_q ? a.conv_q : is_v ? a.conv_v : a.conv_k;
    float ss = 0.f;
    float y[8];                      // sizes up to 256
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = head * size + i * 32 + lane;
      y[i] = 0.f;
      if (i * 32 + lane < size) {
        float acc = 0.f;
        for (int j = 0; j < n; j++) acc += taps[(long long)c * n + j] * conv_input<T>(a, b, t, n - 1 - j, seg, c, chan0 + c, channels);
        y[i] = silu_f(acc);
        ss += y[i] * y[i];
      }
    }
    float f = 1.f;
    if (!is_v) {
      f = 1.f / sqrtf(warp_sum(ss) + 1e-6f);
      if (is_q) f *= 1.f / sqrtf((float)D);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = i * 32 + lane;
      if (c < size) {
        if (is_v) reinterpret_cast<T*>(a.vv)[row * H * E + (long long)head * E + c] = from_f<T>(y[i]);
        else (is_q ? a.qn : a.kn)[row * G * D + (long long)head * D + c] = y[i] * f;
      }
    }
  } else {
    const int head = u - 2 * G - H;
    const float rate = expf(a.a_log[head]);
    for (int c = lane; c < D; c += 32) {
      const long long i = row * H * D + (long long)head * D + c;
      a.gd[i] = expf(-rate * softplus_f(a.gd[i] + a.dt_bias[head * D + c]));
    }
    if (lane == 0) {
      const float z = to_f<T>(reinterpret_cast<const T*>(a.proj)[row * a.ldp + a.s_b + head]);
      a.beta[row * H + head] = 1.f / (1.f + expf(-z));
    }
  }
}

// The last taps - 1 inputs of every convolution after this call's rows.
template <typename T>
__global__ void __launch_bounds__(256) k_conv_tail(const DeltaPrepArgs a) {
  pdl_trigger();
  pdl_wait();
  const int G = a.kv_heads, D = a.dim, channels = 2 * G * D + a.heads * a.vdim, keep = a.taps - 1;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)a.B * keep * channels) return;
  const int chan = (int)(i % channels), k = (int)(i / channels % keep), b = (int)(i / channels / keep);
  const int seg = chan < G * D ? a.s_q + chan : chan < 2 * G * D ? a.s_k + chan - G * D : a.s_v + chan - 2 * G * D;
  const int r = a.T - keep + k;
  reinterpret_cast<T*>(a.tail_out)[i] = r >= 0 ? reinterpret_cast<const T*>(a.proj)[((long long)b * a.T + r) * a.ldp + seg]
                                               : reinterpret_cast<const T*>(a.tail_in)[((long long)b * keep + keep + r) * channels + chan];
}

// ---- one token -----------------------------------------------------------------------------------------------------------
// The whole mixer between the packed projection and the output projection for one new token: convolutions, unit vectors,
// both low-rank projections, state update, read-out, norm and gate.  grid (heads x cluster, columns).  Bound by the chain of
// dependent loads and sums, so a head's E rows of state and its D + E low-rank rows are shared by the CTAs of a cluster: each makes
// q, k and its own v, decays and gates; the decays reach the others through distributed shared memory, the state's rows are
// on their way to registers meanwhile, and the squares for the norm meet the same way.  A warp has whole rows of the state.  Clocks of
// one block's thread (10 heads, 128 x 128) found what to mend: four rows a warp where it has one, and 4-way bank conflicts, were 5.5 us of 14.
// From the projections' end, one column: 14.4 us with those, 8.3 without (10.2 in the chain as it is now).
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }

__device__ __forceinline__ void store_peer(const float* p, uint32_t rank, float v) {
  uint32_t at;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(sm100::smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}

// SI: 128 channels of a row of the state each; ROWS: rows of the state a warp has in flight
template <typename T, int SI, int ROWS>
__global__ void __launch_bounds__(1024) k_delta_decode(const DeltaDecodeArgs a, int cl, int staged) {
  pdl_trigger();
  constexpr int V = VecN<T>::n, HELD = 2;      // low-rank rows of a warp loaded before the wait
  const DeltaPrepArgs& p = a.p;
  const int h = blockIdx.x / cl, rank = blockIdx.x % cl, b = blockIdx.y, tid = threadIdx.x, threads = blockDim.x, warp = tid >> 5, warps = threads >> 5, lane = tid & 31;
  const int H = p.heads, G = p.kv_heads, D = p.dim, E = p.vdim, n = p.taps, keep = n - 1;
  const int qh = h / (H / G), channels = 2 * G * D + H * E;
  // this CTA's decays, and its rows of state, values and gates
  const int dn = (D + cl - 1) / cl, d0 = min(D, rank * dn), d1 = min(D, d0 + dn), en = (E + cl - 1) / cl, e0 = min(E, rank * en), e1 = min(E, e0 + en);
  const int low = d1 - d0 + e1 - e0;
  extern __shared__ __align__(16) float sm[];
  float *sa = sm, *sb = sa + a.ra, *sq = sb + a.rg, *sk = sq + D, *sg = sk + D, *sv = sg + D, *so = sv + en, *sz = so + en, *st = sz + en;      // ranks are padded to 8
  __shared__ float f_q, f_k, squares[8];
  const T* tin = reinterpret_cast<const T*>(p.tail_in) + (long long)b * keep * channels;
  T* tout = reinterpret_cast<T*>(p.tail_out) + (long long)b * keep * channels;
  float* S = a.S + (((long long)b * H + h) * E + e0) * D;
  // low-rank row i of this CTA
  auto low_row = [&](int i) {
    const bool decay = i < d1 - d0;
    const int c = decay ? d0 + i : e0 + i - (d1 - d0);
    return decay ? reinterpret_cast<const T*>(a.w_a2) + (long long)(h * D + c) * a.ra : reinterpret_cast<const T*>(a.w_g2) + (long long)(h * E + c) * a.rg;
  };
  auto low_rank = [&](int i) { return i < d1 - d0 ? a.ra : a.rg; };
  prefetch_l2(S, 4ll * (e1 - e0) * D, tid, threads);
  prefetch_l2(p.dt_bias + (long long)h * D + d0, 4ll * (d1 - d0), tid, threads);
  prefetch_l2(a.norm + e0, 4ll * (e1 - e0), tid, threads);
  if (tid == 0) prefetch_l2(p.a_log + h);
  for (int j = 0; j < keep; j++) {
    prefetch_l2(tin + (long long)j * channels + qh * D, (long long)sizeof(T) * D, tid, threads);
    prefetch_l2(tin + (long long)j * channels + (G + qh) * D, (long long)sizeof(T) * D, tid, threads);
    prefetch_l2(tin + (long long)j * channels + 2 * G * D + h * E + e0, (long long)sizeof(T) * (e1 - e0), tid, threads);
  }
  prefetch_l2(reinterpret_cast<const T*>(a.w_a2) + (long long)(h * D + d0) * a.ra, (long long)sizeof(T) * (d1 - d0) * a.ra, tid, threads);
  prefetch_l2(reinterpret_cast<const T*>(a.w_g2) + (long long)(h * E + e0) * a.rg, (long long)sizeof(T) * (e1 - e0) * a.rg, tid, threads);
  // weights, which no kernel of the chain writes: taps, and the first low-rank rows of each warp
  for (int i = tid; staged && i < (2 * D + e1 - e0) * n; i += threads)
    st[i] = i < D * n ? p.conv_q[(long long)qh * D * n + i] : i < 2 * D * n ? p.conv_k[(long long)qh * D * n + i - D * n] : p.conv_v[(long long)(h * E + e0) * n + i - 2 * D * n];
  uint4 held[HELD];
#pragma unroll
  for (int u = 0; u < HELD; u++) {
    const int i = warp + u * warps;
    if (i < low && lane * V < low_rank(i)) held[u] = *reinterpret_cast<const uint4*>(low_row(i) + lane * V);
  }
  const float rate = expf(p.a_log[h]);
  auto bias_of = [&](int i) { return i < d1 - d0 ? p.dt_bias[h * D + d0 + i] : 0.f; };
  float bias[HELD];
#pragma unroll
  for (int u = 0; u < HELD; u++) bias[u] = bias_of(warp + u * warps);
  const float norm = tid < e1 - e0 ? a.norm[e0 + tid] : 0.f;
  if (cl > 1) sm100::cluster_arrive();        // the others have started
  pdl_wait();
  __syncthreads();      // the taps
  const bool vec = (D & 3) == 0;
  // rows r0 + r warps + warp of this CTA's part of the state
  float s[ROWS][SI][4];
  auto load_state = [&](int r0) {
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
      for (int i = 0; i < SI; i++) {
        const int e = r0 + r * warps + warp, d = 4 * lane + 128 * i;
        const bool there = e < e1 - e0;
        const float* Sp = S + (long long)e * D + d;
        if (vec) {
          const float4 v = d < D && there ? *reinterpret_cast<const float4*>(Sp) : make_float4(0.f, 0.f, 0.f, 0.f);
          s[r][i][0] = v.x; s[r][i][1] = v.y; s[r][i][2] = v.z; s[r][i][3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) s[r][i][j] = d + j < D && there ? Sp[j] : 0.f;
        }
      }
  };
  if (ROWS == 1) load_state(0);       // on its way from here on
  const T* proj = reinterpret_cast<const T*>(p.proj) + (long long)b * p.ldp;
  for (int i = tid; i < a.ra + a.rg; i += threads) sa[i] = to_f<T>(i < a.ra ? proj[a.s_a1 + i] : proj[a.s_g1 + i - a.ra]);
  for (int i = tid; i < 2 * D + e1 - e0; i += threads) {
    const int which = i < D ? 0 : i < 2 * D ? 1 : 2, c = which == 2 ? i - 2 * D : i - which * D;
    const int at = which == 2 ? h * E + e0 + c : qh * D + c, chan = (which == 0 ? 0 : which == 1 ? G * D : 2 * G * D) + at;
    const float* taps = staged ? st + i * n : (which == 0 ? p.conv_q : which == 1 ? p.conv_k : p.conv_v) + (long long)at * n;
    const T now = proj[(which == 0 ? p.s_q : which == 1 ? p.s_k : p.s_v) + at];
    const bool writes = which == 2 || (rank == 0 && h % (H / G) == 0);      // the heads of a group share q and k
    float acc = 0.f;
    for (int j0 = 0; j0 < keep; j0 += 4) {          // four loads in flight before the first store
      T x[4];
#pragma unroll
      for (int j = 0; j < 4; j++) if (j0 + j < keep) x[j] = tin[(long long)(j0 + j) * channels + chan];
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (j0 + j < keep) {
          acc = fmaf(taps[j0 + j], to_f<T>(x[j]), acc);
          if (writes && j0 + j > 0) tout[(long long)(j0 + j - 1) * channels + chan] = x[j];
        }
    }
    if (writes && keep > 0) tout[(long long)(keep - 1) * channels + chan] = now;
    const float y = silu_f(fmaf(taps[keep], to_f<T>(now), acc));
    if (which == 2) sv[c] = round_to<T>(y);
    else (which ? sk : sq)[c] = y;
  }
  if (cl > 1) sm100::cluster_wait();
  __syncthreads();
  if (warp >= warps - 2) {
    const float* x = warp & 1 ? sk : sq;
    float ss = 0.f;
    for (int c = lane; c < D; c += 32) ss += x[c] * x[c];
    ss = 1.f / sqrtf(warp_sum(ss) + 1e-6f);
    if (lane == 0) { if (warp & 1) f_k = ss; else f_q = ss * (1.f / sqrtf((float)D)); }
  }
  for (int i0 = warp, u = 0; i0 < low; i0 += warps, u++) {
    const bool decay = i0 < d1 - d0;
    const float* x = decay ? sa : sb;
    const int r = low_rank(i0);
    const T* w = low_row(i0);
    float z = 0.f;
    for (int c = lane * V; c < r; c += 32 * V) {       // rows are padded to multiples of 8 with zeros
      const uint4 q = c < 32 * V && u < HELD ? (u ? held[1] : held[0]) : *reinterpret_cast<const uint4*>(w + c);
      const T* f = reinterpret_cast<const T*>(&q);
#pragma unroll
      for (int e = 0; e < V; e += 4) {
        const float4 v = *reinterpret_cast<const float4*>(x + c + e);
        z = fmaf(to_f<T>(f[e]), v.x, z); z = fmaf(to_f<T>(f[e + 1]), v.y, z); z = fmaf(to_f<T>(f[e + 2]), v.z, z); z = fmaf(to_f<T>(f[e + 3]), v.w, z);
      }
    }
    z = warp_sum(z);
    if (decay) {
      const int c = d0 + i0;
      z = expf(-rate * softplus_f(z + (u < HELD ? (u ? bias[1] : bias[0]) : bias_of(i0))));
      if (cl == 1) { if (lane == 0) sg[c] = z; }
      else if (lane < cl) store_peer(sg + c, lane, z);
    } else if (lane == 0) {
      sz[i0 - (d1 - d0)] = sigmoid_f(round_to<T>(z));
    }
  }
  if (cl > 1) sm100::cluster_arrive(); else __syncthreads();
  const float beta = sigmoid_f(to_f<T>(proj[p.s_b + h]));
  bool waited = cl == 1;
  for (int r0 = 0; r0 < en; r0 += ROWS * warps) {
    if (ROWS > 1 || r0 > 0) load_state(r0);
    if (!waited) { sm100::cluster_wait(); waited = true; }       // all decays are here, and with them f_q and f_k
    float dot[ROWS] = {}, o[ROWS] = {}, cg[SI][4], ck[SI][4], cq[SI][4];      // decay, key and query of this lane's channels
#pragma unroll
    for (int i = 0; i < SI; i++) {
      const int d = 4 * lane + 128 * i;
      if (vec && d < D) {
        const float4 vg = *reinterpret_cast<const float4*>(sg + d), vk = *reinterpret_cast<const float4*>(sk + d), vq = *reinterpret_cast<const float4*>(sq + d);
        cg[i][0] = vg.x; cg[i][1] = vg.y; cg[i][2] = vg.z; cg[i][3] = vg.w;
        ck[i][0] = vk.x; ck[i][1] = vk.y; ck[i][2] = vk.z; ck[i][3] = vk.w;
        cq[i][0] = vq.x; cq[i][1] = vq.y; cq[i][2] = vq.z; cq[i][3] = vq.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) { const bool in = d + j < D; cg[i][j] = in ? sg[d + j] : 0.f; ck[i][j] = in ? sk[d + j] : 0.f; cq[i][j] = in ? sq[d + j] : 0.f; }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) { ck[i][j] *= f_k; cq[i][j] *= f_q; }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
      for (int i = 0; i < SI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          s[r][i][j] *= cg[i][j];
          dot[r] = fmaf(s[r][i][j], ck[i][j], dot[r]);
        }
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      const int e = r0 + r * warps + warp;
      const float u = beta * ((e < e1 - e0 ? sv[e] : 0.f) - warp_sum(dot[r]));
#pragma unroll
      for (int i = 0; i < SI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          s[r][i][j] = fmaf(ck[i][j], u, s[r][i][j]);
          o[r] = fmaf(s[r][i][j], cq[i][j], o[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      const int e = r0 + r * warps + warp;
      o[r] = warp_sum(o[r]);
      if (e >= e1 - e0) continue;
      if (lane == 0) so[e] = round_to<T>(o[r]);
#pragma unroll
      for (int i = 0; i < SI; i++) {
        const int d = 4 * lane + 128 * i;
        float* Sp = S + (long long)e * D + d;
        if (vec) {
          if (d < D) *reinterpret_cast<float4*>(Sp) = make_float4(s[r][i][0], s[r][i][1], s[r][i][2], s[r][i][3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) if (d + j < D) Sp[j] = s[r][i][j];
        }
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    float ss = 0.f;
    for (int c = lane; c < e1 - e0; c += 32) ss += so[c] * so[c];
    ss = warp_sum(ss);
    if (cl == 1) { if (lane == 0) squares[0] = ss; }
    else if (lane < cl) store_peer(squares + rank, lane, ss);
  }
  if (cl > 1) { sm100::cluster_arrive(); sm100::cluster_wait(); } else __syncthreads();
  float ss = 0.f;
  for (int r = 0; r < cl; r++) ss += squares[r];
  const float inv = 1.f / sqrtf(ss / E + a.eps);
  T* out = reinterpret_cast<T*>(a.out) + ((long long)b * H + h) * E + e0;
  for (int c = tid; c < e1 - e0; c += threads) out[c] = from_f<T>(so[c] * inv * (c == tid ? norm : a.norm[e0 + c]) * sz[c]);
}

}  // namespace

template <typename T> int recurrence(const RecurrenceArgs& a, cudaStream_t s) {
  const dim3 grid(cdiv(a.vdim, 32), a.heads, a.B);
  const bool delta = a.beta != nullptr;
#define LAUNCH(NI) if (delta) CUDA_TRY(launch_dependent(k_recurrence<T, true, NI>, grid, 256, 0, s, a)); else CUDA_TRY(launch_dependent(k_recurrence<T, false, NI>, grid, 256, 0, s, a))
  if (a.dim <= 32) { LAUNCH(1); }
  else if (a.dim <= 64) { LAUNCH(2); }
  else if (a.dim <= 128) { LAUNCH(4); }
  else if (a.dim <= 256) { LAUNCH(8); }
  else return femto_fail(FEMTO_ERR_UNSUPPORTED, "recurrence: dim %d > 256", a.dim);
#undef LAUNCH
  KERNEL_CHECK();
  return 0;
}
template int recurrence<float>(const RecurrenceArgs&, cudaStream_t);
template int recurrence<bf16>(const RecurrenceArgs&, cudaStream_t);

template <typename T> int conv_tail(const DeltaPrepArgs& a, cudaStream_t s) {
  if (a.taps <= 1) return 0;
  const long long m = (long long)a.B * (a.taps - 1) * (2 * a.kv_heads * a.dim + a.heads * a.vdim);
  CUDA_TRY(launch_dependent(k_conv_tail<T>, cdiv(m, 256), 256, 0, s, a));
  KERNEL_CHECK();
  return 0;
}
template int conv_tail<float>(const DeltaPrepArgs&, cudaStream_t);
template int conv_tail<bf16>(const DeltaPrepArgs&, cudaStream_t);

template <typename T> int delta_prep(const DeltaPrepArgs& a, cudaStream_t s) {
  if (a.dim > 256 || a.vdim > 256) return femto_fail(FEMTO_ERR_UNSUPPORTED, "delta rule: dim %d / vdim %d > 256", a.dim, a.vdim);
  const long long n = (long long)a.B * a.T * (2 * a.kv_heads + 2 * a.heads);
  CUDA_TRY(launch_dependent(k_delta_prep<T>, cdiv(n, 8), 256, 0, s, a));
  KERNEL_CHECK();
  return conv_tail<T>(a, s);
}
template int delta_prep<float>(const DeltaPrepArgs&, cudaStream_t);
template int delta_prep<bf16>(const DeltaPrepArgs&, cudaStream_t);

// Heads and columns that leave multiprocessors idle share a head among up to eight of them.
template <typename T> int delta_decode(const DeltaDecodeArgs& a, cudaStream_t s) {
  if (a.p.dim > 256 || a.p.vdim > 256) return femto_fail(FEMTO_ERR_UNSUPPORTED, "delta rule: dim %d / vdim %d > 256", a.p.dim, a.p.vdim);
  int cl = 1;
  while (cl < 8 && 2ll * cl * a.p.heads * a.p.B <= device_sm_count()) cl *= 2;
  const int en = cdiv(a.p.vdim, cl), threads = cl >= 4 ? 512 : 1024;
  size_t smem = 4 * ((size_t)3 * a.p.dim + 3 * en + a.ra + a.rg);
  const size_t taps = 4 * (2 * (size_t)a.p.dim + en) * a.p.taps;
  const int staged = smem + taps <= 47 * 1024;      // many taps are read where they lie
  if (staged) smem += taps;
  if (smem > 48 * 1024 - 64) return femto_fail(FEMTO_ERR_UNSUPPORTED, "delta rule: ranks %d and %d are too large", a.ra, a.rg);
  auto launch = [&](auto kernel) { return launch_dependent_clusters(kernel, cl, dim3(a.p.heads * cl, a.p.B), threads, smem, s, a, cl, staged); };
  const bool once = en <= threads / 32;      // a warp has one row of the state
  if (a.p.dim <= 128) CUDA_TRY(once ? launch(k_delta_decode<T, 1, 1>) : launch(k_delta_decode<T, 1, 4>));
  else CUDA_TRY(once ? launch(k_delta_decode<T, 2, 1>) : launch(k_delta_decode<T, 2, 2>));
  KERNEL_CHECK();
  return 0;
}
template int delta_decode<float>(const DeltaDecodeArgs&, cudaStream_t);
template int delta_decode<bf16>(const DeltaDecodeArgs&, cudaStream_t);
