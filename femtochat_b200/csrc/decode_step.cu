// One new token of every column of a bf16 GPT as one resident kernel (src/gpt.jl:129-170 for one row a column).
//
// A decode step is bound by HBM: its weights are read once (d12 with its head 270 MB, 41 us at 6.65 TB/s; d20 888 MB, 134 us).
// As a chain of launches it took 28 times that, 1.15 ms (d12, one column): 14 launches a block, each of which started its
// weight stream only when its predecessor had finished.  Here one block per multiprocessor stays for the whole step.  One warp of
// it copies the weights of the block's share of ALL products of the step by TMA into a ring in shared memory and knows nothing of
// the rest, so the stream runs on while the chain of dependent phases - norm + QKV, attention, output projection, norm + MLP up,
// MLP down - passes from block to block through counters in global memory.  A token: d12, one column 1150 -> 328 us; d20, eight columns of 540 tokens 2600 -> 1136 us.
// (Copies issued by the eight computing warps
// themselves, cp.async, held up their loads of activations: 400 us a token, d12.)
//
// Shares: an item is 64 output columns times d rows of a matrix, so that QKV, wo and fc have N / 64 items and proj four times
// d / 64 (its four partial sums are added by whoever reads them, in order).  Items go round the blocks without a restart
// from product to product, which balances the stream.  The rows of X are the 8-column operand of mma.m16n8k16, the
// weights its 16-row operand: a lane takes 8 columns of the four rows of W that are its own in the fragment, and byte
// permutations make the (k, k+1) pairs.  RMS norms have no weights here, so the reciprocal root multiplies the product.
#include <algorithm>

#include "decode_step.cuh"
#include "sm100_ptx.cuh"
#include "warp_mma.cuh"

namespace {

constexpr int THREADS = 256, WARPS = 8, SLOT = 128 * 64 * 2,      // computing threads; a slot of the ring: 128 rows of 64 columns
              HD = 128, MAX_SPLITS = 32, COUNTER_STRIDE = 16;   // counters 64 bytes apart
constexpr int RED_PITCH = 66;      // floats per fragment register pair of a warp's sums; 66: a column's eight land in eight banks
constexpr long long SPIN_LIMIT = 1 << 20;

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(s));
  return r;
}
// What other blocks wrote is read past L1
__device__ __forceinline__ float4 ld4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// The computing warps only
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// Rows of X are permuted within every 16 columns so that the four a lane needs (2 c, 2 c + 1, 2 c + 8, 2 c + 9) lie together
__device__ __forceinline__ void put4(bf16* row, int col, uint32_t lo, uint32_t hi) {      // col: a multiple of 4
  uint32_t* w = reinterpret_cast<uint32_t*>(row + (col & ~15)) + (col & 4) + ((col >> 3) & 1);
  w[0] = lo; w[2] = hi;
}

// ---- the new token of every column: its id and position, normalised embedding and smear; counters to zero -------------
__global__ void __launch_bounds__(THREADS) k_step_begin(const DecodeStepArgs a, const int* tokens, const int* positions, int base, int vocab,
                                                        int maxdoc) {
  const int b = blockIdx.x, tid = threadIdx.x;
  if (b == 0)
    for (int i = tid; i < a.n_counters; i += THREADS) a.counters[i * COUNTER_STRIDE] = 0;
  int tk = tokens[b] - base;
  bool bad = tk < 0 || tk >= vocab;
  tk = min(max(tk, 0), vocab - 1);
  __shared__ float red[WARPS];
  __shared__ int pos_s;
  if (tid == 0) {
    int p = positions ? positions[b] : a.lastpos[b] + 1;
    if (p < 0 || p >= maxdoc) { bad = true; p = min(max(p, 0), maxdoc - 1); }
    if (bad) atomicOr(a.status, ST_BAD_TOKEN);
    pos_s = p;
  }
  const bf16* src = a.wte + (long long)tk * a.d;
  float ss = 0.f;
  for (int c = tid; c < a.d; c += THREADS) { const float f = __bfloat162float(src[c]); ss += f * f; }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < WARPS; i++) ss += red[i];
  const float inv = rsqrtf(ss / a.d + a.eps);
  if (tid == 0) {
    const int p = pos_s;
    a.tok0[b] = tk; a.pos[b] = p; a.lastpos[b] = p;
    a.doc_start[b] = max(0, a.t - p);   // index (within the column) of the first token of this token's document
  }
  // every warp sums the smear gate's 24 inputs by itself
  const int lane = tid & 31;
  float pre = lane < 24 ? __bfloat162float(__float2bfloat16_rn(__bfloat162float(src[lane]) * inv)) * a.theta[a.off_smear + lane] : 0.f;
  pre = warp_sum(pre);
  const float gate = a.theta[a.off_lam_s] * (1.f / (1.f + expf(-pre)));
  bf16* prev = a.xe_prev + (long long)b * a.d;
  for (int c = tid; c < a.d; c += THREADS) {
    const bf16 e = __float2bfloat16_rn(__bfloat162float(src[c]) * inv);
    a.x0[(long long)b * a.d + c] = __bfloat162float(e) + gate * __bfloat162float(prev[c]);
    prev[c] = e;
  }
}

// ---- the step ----------------------------------------------------------------------------------------------------------
template <int NT, int GMAX, int RING>
__global__ void __launch_bounds__(THREADS + 32, 1) k_decode_step(const DecodeStepArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3, cta = blockIdx.x, grid = gridDim.x;
  const int d = a.d, B = a.B, xp = d + 16;        // 16: the eight rows of an 8-byte fragment load fall into different banks
  unsigned char* ring = smem;
  bf16* X = reinterpret_cast<bf16*>(smem + RING * SLOT);
  float* red = reinterpret_cast<float*>(X + 8 * NT * xp);
  const DecodeBlock* blocks = reinterpret_cast<const DecodeBlock*>(reinterpret_cast<unsigned char*>(red) + a.red_bytes);
  __shared__ float ssp[8 * NT][33], inv_s[8 * NT], qs[GMAX][HD], kvs[2][HD];
  __shared__ int given_up;
  __shared__ uint64_t full[RING], empty[RING];
  const int steps = d >> 7, np = 4 * a.L + 1;
  const int4 items = make_int4(a.dq >> 6, d >> 6, d >> 4, d >> 4);      // QKV, wo, fc, proj (a quarter of its rows each)
  const int per_block = items.x + items.y + items.z + items.w;
  // the matrix p of the step and the first of its items that is this block's
  auto items_of = [&](int p) { const int k = p & 3; return p == np - 1 ? a.Vp >> 6 : k == 0 ? items.x : k == 1 ? items.y : k == 2 ? items.z : items.w; };
  auto first_item = [&](int p) {
    const int k = p & 3, before = (p >> 2) * per_block + (k > 0 ? items.x : 0) + (k > 1 ? items.y : 0) + (k > 2 ? items.z : 0);
    const int j = cta - before % grid;
    return j < 0 ? j + grid : j;
  };
  auto blocks_of = [&](int p) { return min(items_of(p), grid); };
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(a.blocks);
    uint32_t* dst = const_cast<uint32_t*>(reinterpret_cast<const uint32_t*>(blocks));
    for (int i = tid; i < a.L * (int)sizeof(DecodeBlock) / 4; i += THREADS + 32) dst[i] = src[i];
  }
  for (int i = tid; i < 8 * NT * xp / 2; i += THREADS + 32) reinterpret_cast<uint32_t*>(X)[i] = 0;   // rows from B on stay zero
  if (tid == 0) {
    given_up = 0;
    for (int i = 0; i < RING; i++) { sm100::mbar_init(&full[i], 1); sm100::mbar_init(&empty[i], WARPS); }
    sm100::fence_barrier_init();
  }
  __syncthreads();

  // ---- the stream of weights ----
  if (warp == WARPS) {
    if (lane) return;
    int n = 0, slot = 0, turn = 0;
    for (int p = 0; p < np; p++) {
      const int tiles = (p & 3) == 3 ? d >> 6 : 1 << 30;
      for (int j = first_item(p); j < items_of(p); j += grid) {
        const int ks = j / tiles, tile = j - ks * tiles;
        for (int s = 0; s < steps; s++) {
          if (turn && !sm100::mbar_wait(&empty[slot], (turn & 1) ^ 1, &given_up, a.status)) goto done;
          sm100::mbar_expect_tx(&full[slot], SLOT);
          sm100::tma_load_2d(ring + slot * SLOT, a.maps + p, &full[slot], tile * 64, ks * d + s * 128);
          n++;
          if (++slot == RING) { slot = 0; turn++; }
        }
      }
    }
  done:      // the last copies have landed before the block's shared memory is given back
    for (int i = max(0, n - RING); i < n; i++)
      for (uint32_t k = 0; k < sm100::WAIT_LIMIT && !sm100::mbar_try_wait(&full[i % RING], (i / RING) & 1); k++) {}
    return;
  }
  int slot = 0;
  uint32_t parity = 0;

  // A wait ends when `n` blocks have arrived, or, with an error in the status word, after about a second.
  auto wait = [&](int counter, int n) {
    if (tid == 0 && !*(volatile int*)&given_up) {
      const unsigned int* p = a.counters + counter * COUNTER_STRIDE;
      for (long long spin = 0;; spin++) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= (unsigned int)n) break;
        if (spin >= SPIN_LIMIT) { atomicOr(a.status, ST_WAIT_TIMEOUT); given_up = 1; break; }
      }
    }
    compute_sync();
  };
  auto arrive = [&](int counter) {
    compute_sync();
    if (tid == 0) {
      __threadfence();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counters + counter * COUNTER_STRIDE) : "memory");
    }
  };
  // One item: sums of this warp's steps over the ring, then over the warps in order; out(b, column, sum).
  auto product = [&](int tile, bool normed, auto&& out) {
    float acc[4][NT][4] = {};
    const bf16* xr = X + g * xp + warp * 16 + 4 * c;
    // this lane's rows 2 c, 2 c + 1, 2 c + 8, 2 c + 9 of the warp's 16, 16-byte unit g of each where the 128-byte swizzle put it
    const unsigned char* wl = ring + (warp * 16 + 2 * c) * 128;
    const int u0 = (g ^ (2 * c)) * 16, u1 = (g ^ (2 * c + 1)) * 16;
    auto step = [&](const uint4 (&w)[4], const uint2 (&x)[NT]) {
      const uint32_t* w0 = &w[0].x; const uint32_t* w1 = &w[1].x; const uint32_t* w2 = &w[2].x; const uint32_t* w3 = &w[3].x;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t f[4] = {prmt(w0[j], w1[j], 0x5410), prmt(w0[j], w1[j], 0x7632), prmt(w2[j], w3[j], 0x5410), prmt(w2[j], w3[j], 0x7632)};
#pragma unroll
        for (int t = 0; t < NT; t++) mma16816(acc[j][t], f, x[t].x, x[t].y);
      }
    };
    auto fetch = [&](int s, uint4 (&w)[4], uint2 (&x)[NT]) {
      sm100::mbar_wait(&full[slot], parity, &given_up, a.status);
      const unsigned char* q = wl + slot * SLOT;
      w[0] = *reinterpret_cast<const uint4*>(q + u0);        w[1] = *reinterpret_cast<const uint4*>(q + 128 + u1);
      w[2] = *reinterpret_cast<const uint4*>(q + 1024 + u0); w[3] = *reinterpret_cast<const uint4*>(q + 1152 + u1);
#pragma unroll
      for (int t = 0; t < NT; t++) x[t] = *reinterpret_cast<const uint2*>(xr + 8 * t * xp + s * 128);
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&empty[slot]);
      if (++slot == RING) { slot = 0; parity ^= 1; }
    };
    int s = 0;
    for (; s + 2 <= steps; s += 2) {
      uint4 w[2][4];
      uint2 x[2][NT];
      fetch(s, w[0], x[0]);
      fetch(s + 1, w[1], x[1]);
      step(w[0], x[0]);
      step(w[1], x[1]);
    }
    if (s < steps) {
      uint4 w[4];
      uint2 x[NT];
      fetch(s, w, x);
      step(w, x);
    }
    // register pair (j, i, t): column 8 g + 2 j + i of rows 8 t + 2 c and 8 t + 2 c + 1
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int t = 0; t < NT; t++)
          *reinterpret_cast<float2*>(red + ((warp * 8 + 2 * j + i) * NT + t) * RED_PITCH + 2 * lane) = make_float2(acc[j][t][2 * i], acc[j][t][2 * i + 1]);
    if (normed && tid < B) {
      float ss = 0.f;
      for (int i = 0; i < steps; i++) ss += ssp[tid][i];
      inv_s[tid] = 1.f / sqrtf(ss / d + a.eps);
    }
    compute_sync();
    for (int o = tid; o < 64 * B; o += THREADS) {
      const int b = o >> 6, n = o & 63;
      const float* p = red + ((n & 7) * NT + (b >> 3)) * RED_PITCH + (n >> 3) * 8 + (b & 7);
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; w++) v += p[w * 8 * NT * RED_PITCH];
      out(b, tile * 64 + n, normed ? v * inv_s[b] : v);
    }
    compute_sync();
  };
  // Rows of X from value(b, column) (four at a time), with the sums of squares of every 128 columns.  The loads of several
  // pieces are in flight together: they are latency, 0.8 us a piece if each waits for the one before.
  auto rows_of = [&](auto&& value, auto&& done) {
    constexpr int U = 4;
    for (int q0 = warp; q0 < B * steps; q0 += WARPS * U) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int q = q0 + u * WARPS;
        if (q < B * steps) v[u] = value(q / steps, q % steps * 128 + lane * 4);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int q = q0 + u * WARPS;
        if (q >= B * steps) break;
        const int b = q / steps, k = q % steps, col = k * 128 + lane * 4;
        const float4 x = done(b, col, v[u]);
        put4(X + b * xp, col, pack2(x.x, x.y), pack2(x.z, x.w));
        const float ss = warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w);
        if (lane == 0) ssp[b][k] = ss;
      }
    }
    compute_sync();
  };
  // the residual stream after a block: what the attention left, plus the four partial sums of its MLP
  const long long Bd = (long long)B * d;
  auto stream = [&](int b, int col) {
    const long long at = (long long)b * d + col;
    float4 v = ld4(a.xa + at);
#pragma unroll
    for (int s = 0; s < 4; s++) { const float4 p = ld4(a.part + s * Bd + at); v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w; }
    return v;
  };
  const int G = a.H / a.Hkv, n_attn = B * a.Hkv * a.splits;

  for (int l = 0; l < a.L; l++) {
    const DecodeBlock& blk = blocks[l];
    // ---- mix, norm, QKV ----
    if (int j = first_item(4 * l); j < items.x) {
      const float lb = a.theta[blk.lam_b], l0 = a.theta[blk.lam_x0];
      if (l > 0) wait(5 * l - 1, blocks_of(4 * l - 1));
      const bool writer = j == 0;
      if (l == 0)      // the stream is the embedding
        rows_of([&](int b, int col) { return ld4(a.x0 + (long long)b * d + col); },
                [&](int b, int col, float4 x) {
                  const float4 m = make_float4(lb * x.x + l0 * x.x, lb * x.y + l0 * x.y, lb * x.z + l0 * x.z, lb * x.w + l0 * x.w);
                  if (writer) *reinterpret_cast<float4*>(a.xm + (long long)b * d + col) = m;
                  return m;
                });
      else
        rows_of([&](int b, int col) {
                  const float4 e = ld4(a.x0 + (long long)b * d + col), x = stream(b, col);
                  return make_float4(lb * x.x + l0 * e.x, lb * x.y + l0 * e.y, lb * x.z + l0 * e.z, lb * x.w + l0 * e.w);
                },
                [&](int b, int col, float4 m) {
                  const long long at = (long long)b * d + col;
                  if (writer) {
                    *reinterpret_cast<float4*>(a.xm + at) = m;
                    if (l == a.backout + 1) *reinterpret_cast<float4*>(a.xb + at) = stream(b, col);
                  }
                  return m;
                });
      for (; j < items.x; j += grid)
        product(j, true, [&](int b, int col, float v) { a.qkv[(long long)b * a.dq + col] = v; });
      if (writer && tid < B) a.inv[tid] = inv_s[tid];
      arrive(5 * l);
    }
    // ---- attention: one item is a column's key head and a range of its keys ----
    int j = first_item(4 * l) - items.x % grid;
    if (j < 0) j += grid;
    bool any = false;
    for (; j < n_attn; j += grid) {
      const int sp = j % a.splits, kvh = j / a.splits % a.Hkv, b = j / a.splits / a.Hkv;
      int lo = max(0, a.t - blk.window);
      if (a.docs) lo = max(lo, a.doc_start[b]);
      const int nk = a.t - lo, per = (nk + a.splits - 1) / a.splits;       // cached keys; the new one goes with the last range
      const int k0 = min(a.t, lo + sp * per), k1 = min(a.t, k0 + per);
      const bool last = sp == a.splits - 1;
      bf16* Kb = blk.K + (long long)b * a.maxT * a.kv + (long long)kvh * HD;
      bf16* Vb = blk.V + (long long)b * a.maxT * a.kv + (long long)kvh * HD;
      const long long rot = (long long)a.pos[b] * (HD / 2) + 2 * lane;
      const float2 cs = *reinterpret_cast<const float2*>(a.cos_t + rot), sn = *reinterpret_cast<const float2*>(a.sin_t + rot);
      uint2 ve = make_uint2(0, 0);
      float wg = 0.f;
      if (last && blk.ve) {
        ve = *reinterpret_cast<const uint2*>(blk.ve + (long long)a.tok0[b] * a.kv + (long long)kvh * HD + 4 * lane);
        if (lane < 12) wg = a.theta[blk.ve_gate + lane * a.Hkv + kvh];
      }
      if (!any) {
        for (int i = tid; i < (k1 - k0) * 4; i += THREADS) {      // the cached rows are on their way while the projections finish
          const bf16* r = (i & 2 ? Vb : Kb) + (long long)(k0 + (i >> 2)) * a.kv + (i & 1) * 64;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(r));
        }
        wait(5 * l, blocks_of(4 * l));
      }
      any = true;
      // queries, and with the last range the new key and value: one warp a vector
      for (int v = warp; v < G + (last ? 2 : 0); v += WARPS) {
        const int col = v < G ? (kvh * G + v) * HD : d + (v - G) * a.kv + kvh * HD;
        const float* src = a.qkv + (long long)b * a.dq + col;
        if (v < G + 1) {        // channels 2 lane, 2 lane + 1 and their partners 64 further
          const float2 x1 = __ldcg(reinterpret_cast<const float2*>(src + 2 * lane)), x2 = __ldcg(reinterpret_cast<const float2*>(src + 64 + 2 * lane));
          const float c0 = round_to<bf16>(cs.x), c1 = round_to<bf16>(cs.y), s0 = round_to<bf16>(sn.x), s1 = round_to<bf16>(sn.y);
          const float y0 = x1.x * c0 + x2.x * s0, y1 = x1.y * c1 + x2.y * s1, z0 = -x1.x * s0 + x2.x * c0, z1 = -x1.y * s1 + x2.y * c1;
          const float r = 1.2f / sqrtf(warp_sum(y0 * y0 + y1 * y1 + z0 * z0 + z1 * z1) / HD + a.eps);
          if (v < G) {
            const float f = r * rsqrtf((float)HD);
            *reinterpret_cast<float2*>(&qs[v][2 * lane]) = make_float2(y0 * f, y1 * f);
            *reinterpret_cast<float2*>(&qs[v][64 + 2 * lane]) = make_float2(z0 * f, z1 * f);
          } else {
            const uint32_t p = pack2(y0 * r, y1 * r), q = pack2(z0 * r, z1 * r);
            bf16* dst = Kb + (long long)a.t * a.kv;
            *reinterpret_cast<uint32_t*>(dst + 2 * lane) = p;
            *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = q;
            kvs[0][2 * lane] = __uint_as_float(p << 16); kvs[0][2 * lane + 1] = __uint_as_float(p & 0xffff0000u);
            kvs[0][64 + 2 * lane] = __uint_as_float(q << 16); kvs[0][65 + 2 * lane] = __uint_as_float(q & 0xffff0000u);
          }
        } else {
          float4 x = ld4(src + 4 * lane);
          if (blk.ve) {
            const float pre = warp_sum(lane < 12 ? __ldcg(a.xm + (long long)b * d + lane) * __ldcg(a.inv + b) * wg : 0.f);
            const float gate = 3.f / (1.f + expf(-pre));
            x.x += gate * __uint_as_float(ve.x << 16); x.y += gate * __uint_as_float(ve.x & 0xffff0000u);
            x.z += gate * __uint_as_float(ve.y << 16); x.w += gate * __uint_as_float(ve.y & 0xffff0000u);
          }
          const uint32_t p = pack2(x.x, x.y), q = pack2(x.z, x.w);
          *reinterpret_cast<uint2*>(Vb + (long long)a.t * a.kv + 4 * lane) = make_uint2(p, q);
          kvs[1][4 * lane] = __uint_as_float(p << 16); kvs[1][4 * lane + 1] = __uint_as_float(p & 0xffff0000u);
          kvs[1][4 * lane + 2] = __uint_as_float(q << 16); kvs[1][4 * lane + 3] = __uint_as_float(q & 0xffff0000u);
        }
      }
      compute_sync();
      // half a warp takes every sixteenth key, four at a time; a lane has eight channels
      const int hl = lane & 15, str = warp * 2 + (lane >> 4);
      constexpr int U = GMAX > 2 ? 2 : 4;
      constexpr int QR = GMAX > 2 ? 1 : GMAX;      // many heads: their queries stay in shared memory
      float q[QR][8], o[GMAX][8] = {}, m[GMAX], lsum[GMAX] = {};
#pragma unroll
      for (int h = 0; h < GMAX; h++) {
        m[h] = -INFINITY;
        if (h >= QR) continue;
#pragma unroll
        for (int e = 0; e < 8; e++) q[h][e] = h < G ? qs[h][hl * 8 + e] : 0.f;
      }
      const int rounds = k1 - k0 + (last ? 1 : 0);
      for (int base = 0; base < rounds; base += 16 * U) {
        float kf[U][8], vf[U][8];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int k = base + 16 * u + str;
          ok[u] = k < rounds;
          if (k < k1 - k0) {
            load_vec<bf16, 8>(Kb + (long long)(k0 + k) * a.kv + hl * 8, kf[u]);
            load_vec<bf16, 8>(Vb + (long long)(k0 + k) * a.kv + hl * 8, vf[u]);
          } else {
#pragma unroll
            for (int e = 0; e < 8; e++) { kf[u][e] = ok[u] ? kvs[0][hl * 8 + e] : 0.f; vf[u][e] = ok[u] ? kvs[1][hl * 8 + e] : 0.f; }
          }
        }
#pragma unroll
        for (int h = 0; h < GMAX; h++) {
          if (h >= G) break;
          float s[U], mn = m[h];
#pragma unroll
          for (int u = 0; u < U; u++) {
            s[u] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e++) s[u] = fmaf(GMAX > 2 ? qs[h][hl * 8 + e] : q[h < QR ? h : 0][e], kf[u][e], s[u]);
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], x);
            if (ok[u]) mn = fmaxf(mn, s[u]);
          }
          if (mn == -INFINITY) continue;      // no key yet (the shuffles above were for both halves)
          const float corr = __expf(m[h] - mn);          // 0 for the first keys
          lsum[h] *= corr;
#pragma unroll
          for (int e = 0; e < 8; e++) o[h][e] *= corr;
#pragma unroll
          for (int u = 0; u < U; u++) {
            const float p = ok[u] ? __expf(s[u] - mn) : 0.f;
            lsum[h] += p;
#pragma unroll
            for (int e = 0; e < 8; e++) o[h][e] = fmaf(p, vf[u][e], o[h][e]);
          }
          m[h] = mn;
        }
      }
      // the two halves of a warp, then the warps in order
#pragma unroll
      for (int h = 0; h < GMAX; h++) {
        if (h >= G) break;
        const float mo = __shfl_xor_sync(0xffffffffu, m[h], 16), mn = fmaxf(m[h], mo);
        const float f = m[h] == -INFINITY ? 0.f : __expf(m[h] - mn);
        float L = lsum[h] * f;
        L += __shfl_xor_sync(0xffffffffu, L, 16);
        float* r = red + (warp * GMAX + h) * (HD + 4);
#pragma unroll
        for (int e = 0; e < 8; e++) {
          float v = o[h][e] * f;
          v += __shfl_xor_sync(0xffffffffu, v, 16);
          if (lane < 16) r[hl * 8 + e] = v;
        }
        if (lane == 0) { r[HD] = mn; r[HD + 1] = L; }
      }
      compute_sync();
      for (int i = tid; i < G * HD; i += THREADS) {
        const int h = i / HD, ch = i % HD;
        float M = -INFINITY, L = 0.f, v = 0.f;
        for (int w = 0; w < WARPS; w++) M = fmaxf(M, red[(w * GMAX + h) * (HD + 4) + HD]);
        for (int w = 0; w < WARPS; w++) {
          const float* r = red + (w * GMAX + h) * (HD + 4);
          const float f = r[HD] == -INFINITY ? 0.f : __expf(r[HD] - M);
          L += r[HD + 1] * f; v += r[ch] * f;
        }
        const long long at = ((long long)b * a.H + kvh * G + h) * a.splits + sp;
        a.att[at * HD + ch] = v;
        if (ch == 0) a.att_ml[at] = make_float2(M, L);
      }
      compute_sync();
    }
    if (any) arrive(5 * l + 1);
    // ---- output projection ----
    if (int j2 = first_item(4 * l + 1); j2 < items.y) {
      wait(5 * l + 1, min(n_attn, grid));
      constexpr int U = 4;
      for (int q0 = warp; q0 < B * a.H; q0 += WARPS * U) {       // a warp joins the ranges of a head, U heads at a time
        float2 ml[U];
        float4 v[U] = {};
#pragma unroll
        for (int u = 0; u < U; u++) {
          ml[u] = make_float2(-INFINITY, 0.f);
          if (lane < a.splits && q0 + u * WARPS < B * a.H) ml[u] = __ldcg(a.att_ml + (long long)(q0 + u * WARPS) * a.splits + lane);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          ml[u].x = __expf(ml[u].x - warp_max(ml[u].x));      // 0 in the lanes without a range
        }
#pragma unroll 4
        for (int s = 0; s < a.splits; s++) {
          float4 p[U];
#pragma unroll
          for (int u = 0; u < U; u++)
            p[u] = ld4(a.att + ((long long)min(q0 + u * WARPS, B * a.H - 1) * a.splits + s) * HD + lane * 4);
#pragma unroll
          for (int u = 0; u < U; u++) {
            const float w = __shfl_sync(0xffffffffu, ml[u].x, s);
            v[u].x += w * p[u].x; v[u].y += w * p[u].y; v[u].z += w * p[u].z; v[u].w += w * p[u].w;
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int q = q0 + u * WARPS;
          if (q >= B * a.H) break;
          const float r = 1.f / warp_sum(ml[u].y * ml[u].x);
          put4(X + q / a.H * xp, q % a.H * HD + lane * 4, pack2(v[u].x * r, v[u].y * r), pack2(v[u].z * r, v[u].w * r));
        }
      }
      compute_sync();
      for (; j2 < items.y; j2 += grid)
        product(j2, false, [&](int b, int col, float v) { const long long at = (long long)b * d + col; a.xa[at] = __ldcg(a.xm + at) + v; });
      arrive(5 * l + 2);
    }
    // ---- norm, MLP up ----
    if (int j2 = first_item(4 * l + 2); j2 < items.z) {
      wait(5 * l + 2, blocks_of(4 * l + 1));
      rows_of([&](int b, int col) { return ld4(a.xa + (long long)b * d + col); }, [](int, int, float4 v) { return v; });
      for (; j2 < items.z; j2 += grid)
        product(j2, true, [&](int b, int col, float v) { v = fmaxf(v, 0.f); a.up[(long long)b * 4 * d + col] = __float2bfloat16_rn(v * v); });
      arrive(5 * l + 3);
    }
    // ---- MLP down: a quarter of the inner rows an item ----
    if (int j2 = first_item(4 * l + 3); j2 < items.w) {
      wait(5 * l + 3, blocks_of(4 * l + 2));
      for (; j2 < items.w; j2 += grid) {
        const int tiles = d >> 6, ks = j2 / tiles, n8 = d >> 3;
        constexpr int U = 4;
        for (int i0 = tid; i0 < B * n8; i0 += THREADS * U) {
          uint4 v[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int i = min(i0 + u * THREADS, B * n8 - 1);
            v[u] = __ldcg(reinterpret_cast<const uint4*>(a.up + (long long)(i / n8) * 4 * d + ks * d + i % n8 * 8));
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int i = i0 + u * THREADS;
            if (i >= B * n8) break;
            bf16* row = X + i / n8 * xp;
            put4(row, i % n8 * 8, v[u].x, v[u].y);
            put4(row, i % n8 * 8 + 4, v[u].z, v[u].w);
          }
        }
        compute_sync();
        product(j2 - ks * tiles, false, [&](int b, int col, float v) { a.part[ks * Bd + (long long)b * d + col] = v; });
      }
      arrive(5 * l + 4);
    }
  }
  // ---- backout, norm, head ----
  if (int j = first_item(4 * a.L); j < a.Vp >> 6) {
    const float ly = a.theta[a.off_lam_y];
    wait(5 * a.L - 1, blocks_of(4 * a.L - 1));
    const bool same = a.backout == a.L - 1;
    rows_of([&](int b, int col) {
              const float4 x = stream(b, col), y = same ? x : ld4(a.xb + (long long)b * d + col);
              return make_float4(x.x - ly * y.x, x.y - ly * y.y, x.z - ly * y.z, x.w - ly * y.w);
            },
            [](int, int, float4 v) { return v; });
    for (; j < a.Vp >> 6; j += grid)
      product(j, true, [&](int b, int col, float v) { if (col < a.V) a.logits[(long long)b * a.V + col] = 15.f * tanhf(v / 15.f); });
  }
}

template <int NT> constexpr int ring_of() { return NT == 1 ? 10 : 8; }
size_t red_bytes(int nt, int gmax) { return std::max((size_t)4 * WARPS * 8 * nt * RED_PITCH, (size_t)4 * WARPS * gmax * (HD + 4)); }
size_t smem_bytes(int d, int L, int nt, int gmax) {
  return (size_t)(nt == 1 ? ring_of<1>() : ring_of<2>()) * SLOT + (size_t)8 * nt * (d + 16) * 2 + red_bytes(nt, gmax) + sizeof(DecodeBlock) * L;
}

// blocks that stay on the device together, or 0
template <int NT, int GMAX> int resident_blocks(size_t smem) {
  auto kernel = k_decode_step<NT, GMAX, ring_of<NT>()>;
  int per = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, THREADS + 32, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per > 0 ? device_sm_count() : 0;
}
int resident(int nt, int gmax, size_t smem) {
  if (nt == 1) return gmax == 2 ? resident_blocks<1, 2>(smem) : resident_blocks<1, 8>(smem);
  return gmax == 2 ? resident_blocks<2, 2>(smem) : resident_blocks<2, 8>(smem);
}

}  // namespace

// bf16, heads of 128 channels (so every width is a multiple of 128), at most 8 query heads a key head, and as many columns as
// leave room for the ring (16 up to d = 2000 or so, 8 up to 3000); anything else takes the chain of kernels of decode.cu.
void decode_step_plan(const femto_handle* h, int max_batch, DecodeStepState& st) {
  st.blocks_n = st.columns = 0;
  if (!h->bf || h->hd != HD || (h->d & 127) || (h->Vp & 63) || h->H % h->Hkv || h->H / h->Hkv > 8 || h->d > 128 * 32) return;
  const int gmax = h->H / h->Hkv <= 2 ? 2 : 8;
  for (int nt = 1; nt <= (max_batch > 8 ? 2 : 1); nt++) {
    const int n = resident(nt, gmax, smem_bytes(h->d, h->L, nt, gmax));
    if (!n) return;
    st.blocks_n = n; st.columns = std::min(max_batch, 8 * nt);
  }
}

size_t decode_step_bytes(const femto_handle* h, DecodeStepState st) {
  char* p = nullptr;
  decode_step_carve(h, p, st);
  return (size_t)(p - (char*)nullptr);
}

void decode_step_carve(const femto_handle* h, char*& p, DecodeStepState& st) {
  auto take = [&](auto*& q, size_t bytes) { q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(p); p += (bytes + 255) & ~(size_t)255; };
  const size_t d = h->d, n = st.columns;
  take(st.maps, sizeof(CUtensorMap) * (4 * h->L + 1));
  take(st.blocks, sizeof(DecodeBlock) * h->L);
  take(st.counters, 4 * COUNTER_STRIDE * (size_t)(5 * h->L));
  take(st.x0, 4 * n * d); take(st.xm, 4 * n * d); take(st.xa, 4 * n * d); take(st.xb, 4 * n * d);
  take(st.part, 16 * n * d); take(st.qkv, 4 * n * h->dq); take(st.inv, 4 * n);
  take(st.up, 2 * n * 4 * d);
  take(st.att, 4 * n * h->H * MAX_SPLITS * HD); take(st.att_ml, 8 * n * h->H * MAX_SPLITS);
}

int decode_step_setup(const femto_handle* h, DecodeStepState& st, const std::vector<void*>& K, const std::vector<void*>& V) {
  std::vector<CUtensorMap> maps;
  std::vector<DecodeBlock> bl;
  auto put = [&](const void* W, int rows, int cols) {      // boxes of 128 rows and 64 columns: one slot of the ring
    const uint64_t dims[2] = {(uint64_t)cols, (uint64_t)rows}, stride[1] = {(uint64_t)cols};
    const uint32_t box[2] = {64, 128};
    maps.emplace_back();
    return make_tmap_nd_bf16(&maps.back(), W, 2, dims, stride, box);
  };
  for (int i = 0; i < h->L; i++) {
    const LayerBuf& l = h->lb[i];
    const LayerP& p = h->lp[i];
    FEMTO_TRY(put(l.sh_wqkv, h->d, h->dq)); FEMTO_TRY(put(l.sh_wo, h->d, h->d));
    FEMTO_TRY(put(l.sh_fc, h->d, 4 * h->d)); FEMTO_TRY(put(l.sh_proj, 4 * h->d, h->d));
    DecodeBlock b = {};
    b.K = (bf16*)K[i]; b.V = (bf16*)V[i]; b.ve = p.ve ? (const bf16*)l.sh_ve : nullptr;
    b.lam_b = p.lam_b; b.lam_x0 = p.lam_x0; b.ve_gate = p.ve_gate; b.window = p.window;
    bl.push_back(b);
  }
  FEMTO_TRY(put(h->sh_lm, h->d, h->Vp));
  CUDA_TRY(cudaMemcpy(st.blocks, bl.data(), sizeof(DecodeBlock) * bl.size(), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(st.maps, maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice));
  return 0;
}

int decode_step_run(const femto_handle* h, const DecodeStepState& st, DecodeStepArgs a, const int* tokens, const int* positions, cudaStream_t s) {
  a.blocks = st.blocks; a.maps = st.maps; a.counters = st.counters; a.n_counters = 5 * h->L;
  a.x0 = st.x0; a.xm = st.xm; a.xa = st.xa; a.xb = st.xb; a.part = st.part; a.qkv = st.qkv; a.inv = st.inv; a.up = st.up; a.att = st.att;
  a.att_ml = st.att_ml;
  a.wte = (const bf16*)h->sh_wte; a.sin_t = h->sin_t; a.cos_t = h->cos_t; a.status = h->status;
  a.off_smear = h->off_smear; a.off_lam_s = h->off_lam_s; a.off_lam_y = h->off_lam_y;
  a.d = h->d; a.dq = h->dq; a.kv = h->kv; a.H = h->H; a.Hkv = h->Hkv; a.V = h->V; a.Vp = h->Vp; a.L = h->L; a.backout = h->backout; a.eps = h->eps;
  a.docs = h->cfg.doc_mask ? 1 : 0;
  // ranges of about 64 keys, as many as there are blocks for
  int keys = 0;
  for (const LayerP& p : h->lp) keys = std::max(keys, std::min(a.t + 1, p.window + 1));
  a.splits = std::max(1, std::min({MAX_SPLITS, cdiv(keys, 64), st.blocks_n / (a.B * a.Hkv)}));
  k_step_begin<<<a.B, THREADS, 0, s>>>(a, tokens, positions, h->cfg.index_base, h->V, h->cfg.max_document_tokens);
  KERNEL_CHECK();
  const int nt = a.B <= 8 ? 1 : 2, gmax = a.H / a.Hkv <= 2 ? 2 : 8;
  const size_t smem = smem_bytes(a.d, a.L, nt, gmax);
  a.red_bytes = (int)red_bytes(nt, gmax);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = st.blocks_n; cfg.blockDim = THREADS + 32; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;      // the blocks wait for one another: all of them are resident or none is
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
#define LAUNCH(NT, GM) CUDA_TRY(cudaLaunchKernelEx(&cfg, k_decode_step<NT, GM, ring_of<NT>()>, a))
  if (nt == 1) { if (gmax == 2) LAUNCH(1, 2); else LAUNCH(1, 8); }
  else { if (gmax == 2) LAUNCH(2, 2); else LAUNCH(2, 8); }
#undef LAUNCH
  KERNEL_CHECK();
  return 0;
}
