// One new token of every column of a bf16 GPT as one resident kernel (src/gpt.jl:129-170 for one row a column).
//
// A decode step is bound by HBM: its weights are read once (d12 with its head 270 MB, 41 us at 6.65 TB/s; d20 888 MB, 134 us).
// As a chain of launches it took 28 times that, 1.15 ms (d12, one column): 14 launches a block, each of which started its
// weight stream only when its predecessor had finished.  Here one block per multiprocessor stays for the whole step.  One warp of
// it copies the weights of the block's share of ALL products of the step by TMA into a ring in shared memory and knows nothing of
// the rest, so the stream runs on while the chain of dependent phases - norm + QKV, attention, output projection, norm + MLP up,
// MLP down - passes from block to block.  (Copies issued by the eight computing warps themselves, cp.async, held up their loads of
// activations: 400 us a token, d12.)
//
// What a phase leaves goes to global memory as words that carry a name, the launch and the layer, beside their data: 4 bytes of data in 8
// (fp32 values that few read), 12 in 16 (the bf16 rows that every block reads; 16 bytes an access asked L2 half as often as 8 did).  Who
// needs a word reads until its name is right.  A store and a load carry a value across, where data, a fence, a counter and a poll (the
// first form of this kernel) took 2 us a phase and 328 us a token of d12, 1136 us of eight columns of d20.  No buffer is
// written again before its readers of the layer before are done, since every phase needs all of the one before it.
// With many words a phase is waited for by ONE thread of a block, on a count of finished items that has no order of its own, and the
// words are read once it says that they should be there: 148 blocks that polled 30 KB each kept the words from arriving, 5 to 11 us a
// phase (d20, eight columns).  With few, a warp polls its first word and then reads the rest.
// Measured a token: d12, one column, chain of launches 1150 us, named words of 8 bytes and 64-column items 204, now 179; d20, eight columns
// of 540 tokens 2600, 873, 650.  Of a layer's 30 us there (6 would stream its weights), 1.9 are the read of the rows in each of four
// phases, 1.4 to 2 each product, 5 the attention; 12 blocks have two items of the MLP's 160, which costs 4.
//
// Shares: an item is 32 output columns times d rows of a matrix, so that QKV, wo and fc have N / 32 items and proj four times
// d / 32 (its four partial sums are added, in order, by the block that has the first).  (64 columns left 108 of 148 blocks without a part
// of QKV, 128 of wo.)  Items go round the blocks without a restart
// from product to product, which balances the stream.  The rows of X are the 8-column operand of mma.m16n8k16, the
// weights its 16-row operand, turned by ldmatrix on its way from the ring.  RMS norms have no weights here, so the reciprocal root
// multiplies the product.
#include <algorithm>

#include "decode_step.cuh"
#include "named_words.cuh"
#include "sm100_ptx.cuh"
#include "warp_mma.cuh"

namespace {

constexpr int THREADS = 256, WARPS = 8, HD = 128, MAX_SPLITS = 32;      // computing threads
constexpr int TILE = 32;           // columns of an item
constexpr int RED_PITCH = 36;      // floats of a warp's sums of one row; 36: the four rows that eight lanes each store land in 32 banks
constexpr int SPIN_LIMIT = 1 << 20;
// How many items of a kind the step has finished, counted without order beside the words themselves: see rows_of
// (what QKV and head read, QKV, attention, what the MLP reads, four quarters of its inside, its partial sums)
enum { HINT_ROWS, HINT_QKV, HINT_ATT, HINT_MID, HINT_UP, HINT_PART = HINT_UP + 4, HINTS };

// Words that carry their name, straight from and to L2.  Each is ONE 64-bit scalar, which the memory model never tears: a vector of
// 32-bit elements is several accesses without order, and a reader could see the new name beside the old data.  (Two words a load: a
// vector of two such scalars, each with a name of its own.)
__device__ __forceinline__ uint4 named_load2(const uint2* p) {
  uint4 v;
  asm volatile("{\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 named_load(const uint2* p) {
  uint2 v;
  asm volatile("{\n\t.reg .b64 a;\n\tld.relaxed.gpu.global.b64 a, [%2];\n\tmov.b64 {%0, %1}, a;\n\t}" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void named_store(uint2* p, uint32_t data, uint32_t name) {
  asm volatile("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], a;\n\t}" ::"l"(p), "r"(data), "r"(name) : "memory");
}
// 16 columns of a row are three words: columns 0 to 5, 6 to 11, and 12 to 15 (its third pair is not used).  A row has a word more than it
// needs, in memory and in shared memory, where the words are copied as they are: the rows then start in different banks.
__host__ __device__ constexpr int words_of(int columns) { return columns / 16 * 3; }
__host__ __device__ constexpr int pitch_of(int d) { return words_of(d) + 1; }
// where pair i of 16 columns is, in 32-bit units
__device__ __forceinline__ int place(int i) { return i / 3 * 4 + i % 3; }
__device__ __forceinline__ void named_store(uint2* p, float data, uint32_t name) { named_store(p, __float_as_uint(data), name); }
__device__ __forceinline__ float lo_f(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float hi_f(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// The computing warps only
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// ---- the new token of every column: its id and position, normalised embedding and smear, and the first block's mixed stream ----
// launches[0] counts the launches so far, launches[1] is this one's number for the blocks of the step.  What the cache keeps from
// token to token (xe_prev, lastpos) is read only, and the caller swaps the buffers once the step is launched: where that is refused, the
// chain of kernels starts from the same state.
__global__ void __launch_bounds__(THREADS) k_step_begin(const DecodeStepArgs a, const int* tokens, const int* positions, int base, int vocab,
                                                        int maxdoc) {
  const int b = blockIdx.x, tid = threadIdx.x;
  const uint32_t launch = a.launches[0] + 1, name = launch * (a.L + 1) + 1;
  if (b == 0 && tid == 0) a.launches[1] = launch;
  if (b == 0 && tid < HINTS) a.hints[tid * 32] = 0;
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
  const bf16* row = a.wte + (long long)tk * a.d;
  auto src = [&](int c) { return __bfloat162float(row[c]); };
  float ss = 0.f;
  for (int c = tid; c < a.d; c += THREADS) { const float f = src(c); ss += f * f; }
  ss = warp_sum(ss);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int i = 0; i < WARPS; i++) ss += red[i];
  const float inv = rsqrtf(ss / a.d + a.eps);
  if (tid == 0) {
    const int p = pos_s;
    a.tok0[b] = tk; a.pos[b] = p;
    a.doc_start[b] = max(0, a.t - p);   // index (within the column) of the first token of this token's document
  }
  // every warp sums the smear gate's 24 inputs by itself
  const int lane = tid & 31;
  float pre = lane < 24 ? __bfloat162float(__float2bfloat16_rn(src(lane) * inv)) * a.theta[a.off_smear + lane] : 0.f;
  pre = warp_sum(pre);
  const float gate = a.theta[a.off_lam_s] * (1.f / (1.f + expf(-pre)));
  const bf16* prev = a.xe_prev + (long long)b * a.d;
  bf16* next = a.xe_new + (long long)b * a.d;
  const float mix = a.theta[a.blocks[0].lam_b] + a.theta[a.blocks[0].lam_x0];
  for (int c = 2 * tid; c < a.d; c += 2 * THREADS) {
    float x[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const bf16 e = __float2bfloat16_rn(src(c + i) * inv);
      x[i] = __bfloat162float(e) + gate * __bfloat162float(prev[c + i]);
      next[c + i] = e;
      const long long at = (long long)b * a.d + c + i;
      a.x0[at] = x[i];
      x[i] *= mix;
      named_store(a.xm + at, x[i], name);
    }
    const uint32_t w0 = pack2(x[0], x[1]), w1 = __shfl_down_sync(0xffffffffu, w0, 1), w2 = __shfl_down_sync(0xffffffffu, w0, 2);   // whole warps: d / 2 is a multiple of 64
    if ((tid & 7) % 3 == 0) named_store(a.xn + (long long)b * pitch_of(a.d) + words_of(c) + (tid & 7) / 3, w0, w1, w2, name);
  }
}

constexpr int slot_bytes(int ks) { return 128 * ks * TILE * 2; }
constexpr int MAX_RING = 20, MIN_RING = 4;

// ---- the step ----------------------------------------------------------------------------------------------------------
// KS: steps of 16 rows that a warp has of a slot of the ring, which is 8 KS x 16 rows of a tile
template <int NT, int GMAX, int KS>
__global__ void __launch_bounds__(THREADS + 128, 1) k_decode_step(const DecodeStepArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int SLOT = slot_bytes(KS);
  const int RING = a.ring;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3, cta = blockIdx.x, grid = gridDim.x;
  const int d = a.d, B = a.B, pitch = pitch_of(d);
  unsigned char* ring = smem;
  uint4* X = reinterpret_cast<uint4*>(smem + RING * SLOT);
  float* red = reinterpret_cast<float*>(X + 8 * NT * pitch);
  const DecodeBlock* blocks = reinterpret_cast<const DecodeBlock*>(reinterpret_cast<unsigned char*>(red) + a.red_bytes);
  __shared__ float ssp[8 * NT][WARPS + 1], inv_s[8 * NT], qs[GMAX][HD], kvs[2][HD];
  const uint32_t launch = a.launches[1];
  __shared__ int given_up;
  __shared__ uint64_t full[MAX_RING], empty[MAX_RING];
  const int slots = d / (128 * KS), np = 4 * a.L + 1;
  const int4 items = make_int4(a.dq / TILE, d / TILE, 4 * d / TILE, 4 * d / TILE);      // QKV, wo, fc, proj (a quarter of its rows each)
  const int per_block = items.x + items.y + items.z + items.w;
  // the matrix p of the step and the first of its items that is this block's
  auto items_of = [&](int p) { const int k = p & 3; return p == np - 1 ? a.Vp / TILE : k == 0 ? items.x : k == 1 ? items.y : k == 2 ? items.z : items.w; };
  auto first_item = [&](int p) {
    const int k = p & 3, before = (p >> 2) * per_block + (k > 0 ? items.x : 0) + (k > 1 ? items.y : 0) + (k > 2 ? items.z : 0);
    const int j = cta - before % grid;
    return j < 0 ? j + grid : j;
  };
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(a.blocks);
    uint32_t* dst = const_cast<uint32_t*>(reinterpret_cast<const uint32_t*>(blocks));
    for (int i = tid; i < a.L * (int)sizeof(DecodeBlock) / 4; i += THREADS + 128) dst[i] = src[i];
  }
  for (int i = tid; i < 8 * NT * pitch; i += THREADS + 128) X[i] = make_uint4(0, 0, 0, 0);   // rows from B on stay zero
  if (tid == 0) {
    if (cta == 0) a.launches[0] = launch;
    given_up = 0;
    for (int i = 0; i < RING; i++) { sm100::mbar_init(&full[i], 1); sm100::mbar_init(&empty[i], WARPS); }
    sm100::fence_barrier_init();
  }
  __syncthreads();

  // ---- the stream of weights ----
  // (a warpgroup for it, which gives its registers to the computing ones: 4 x 24 + 8 x 240 = 12 x 168 a lane)
  if (warp >= WARPS) {
    sm100::reg_dealloc<24>();
    if (warp > WARPS || lane) return;
    int n = 0, slot = 0, turn = 0;
    for (int p = 0; p < np; p++) {
      const int tiles = (p & 3) == 3 ? d / TILE : 1 << 30;
      for (int j = first_item(p); j < items_of(p); j += grid) {
        const int ks = j / tiles, tile = j - ks * tiles;
        for (int s = 0; s < slots; s++) {
          if (turn && !sm100::mbar_wait(&empty[slot], (turn & 1) ^ 1, &given_up, a.status)) goto done;
          sm100::mbar_expect_tx(&full[slot], SLOT);
          sm100::tma_load_3d(ring + slot * SLOT, a.maps + p, &full[slot], tile * TILE, ks * d + s * 128 * KS, 0);
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
  sm100::reg_alloc<240>();
  int slot = 0;
  uint32_t parity = 0;

  // Reads until done() says that every word has its name, or, with an error in the status word, for about a second.
  auto until = [&](auto&& done) {
    for (int spin = 0; !done(); spin++) {
      if (spin < SPIN_LIMIT && ((spin & 63) != 63 || !*(volatile int*)&given_up)) continue;
      if (spin >= SPIN_LIMIT) { atomicOr(a.status, ST_WAIT_TIMEOUT); *(volatile int*)&given_up = 1; }
      break;
    }
  };
  auto word = [&](const uint2* p, uint32_t name) {
    uint2 v;
    until([&] { v = named_load(p); return v.y == name; });
    return __uint_as_float(v.x);
  };
  // One item: sums of this warp's steps over the ring, then over the warps in order; out(k, b, column, sum).
  // A warp has the 32 columns of one row b = warp + 8 k at a time.  `normed`: times the reciprocal root of the row's mean square, which the warps
  // sum from the pieces of X that they multiply.
  auto product = [&](int tile, bool normed, auto&& out) {
    float acc[2][NT][4] = {}, ss[NT] = {};
    const uint32_t* xr = reinterpret_cast<const uint32_t*>(X + g * pitch + warp * KS * 3);      // pairs c and c + 4 of every 16 columns
    const int p0 = place(c), p1 = place(c + 4);
    // this lane's row of a 16 x 16 piece, and its 16-byte unit of either piece where the 64-byte swizzle put it
    const int row = warp * 16 * KS + (lane & 7) + ((lane >> 4) << 3), unit = (lane >> 3) & 1, turned = (row >> 1) & 3;      // 16 rows further: the same turn
    const unsigned char* wl = ring + row * 64;
    const int u0 = (unit ^ turned) * 16, u1 = ((2 + unit) ^ turned) * 16;
    auto fetch = [&](int s, uint32_t (&f)[KS][2][4], uint2 (&x)[KS][NT]) {
      sm100::mbar_wait(&full[slot], parity, &given_up, a.status);
      const unsigned char* q = wl + slot * SLOT;
#pragma unroll
      for (int k = 0; k < KS; k++) {
        ldsm4t(f[k][0], q + k * 1024 + u0);
        ldsm4t(f[k][1], q + k * 1024 + u1);
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const uint32_t* w = xr + (8 * t * pitch + (s * 8 * KS + k) * 3) * 4;
          x[k][t] = make_uint2(w[p0], w[p1]);
        }
      }
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&empty[slot]);
      if (++slot == RING) { slot = 0; parity ^= 1; }
    };
    auto multiply = [&](const uint32_t (&f)[KS][2][4], const uint2 (&x)[KS][NT]) {
#pragma unroll
      for (int k = 0; k < KS; k++)
#pragma unroll
        for (int t = 0; t < NT; t++) {
#pragma unroll
          for (int i = 0; i < 2; i++) mma16816(acc[i][t], f[k][i], x[k][t].x, x[k][t].y);
          if (!normed) continue;
          const float e = lo_f(x[k][t].x), h = hi_f(x[k][t].x), u = lo_f(x[k][t].y), v = hi_f(x[k][t].y);
          ss[t] += (e * e + h * h) + (u * u + v * v);
        }
    };
    int s = 0;
    for (; s + 2 <= slots; s += 2) {
      uint32_t f[2][KS][2][4];
      uint2 x[2][KS][NT];
      fetch(s, f[0], x[0]);
      fetch(s + 1, f[1], x[1]);
      multiply(f[0], x[0]);
      multiply(f[1], x[1]);
    }
    if (s < slots) {
      uint32_t f[KS][2][4];
      uint2 x[KS][NT];
      fetch(s, f, x);
      multiply(f, x);
    }
    // registers (i, t): columns 16 i + g and 16 i + g + 8 of rows 8 t + 2 c and 8 t + 2 c + 1
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int e = 0; e < 4; e++) red[((warp * NT + t) * 8 + 2 * c + (e & 1)) * RED_PITCH + 16 * i + g + 8 * (e >> 1)] = acc[i][t][e];
    if (normed) {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 1);
        ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 2);
        if (c == 0) ssp[8 * t + g][warp] = ss[t];
      }
    }
    compute_sync();
#pragma unroll
    for (int k = 0; k < NT; k++) {
      const int b = warp + 8 * k;
      if (b >= B) break;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; w++) v += red[(w * NT * 8 + b) * RED_PITCH + lane];
      if (normed) {
        float q = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) q += ssp[b][w];
        const float inv = 1.f / sqrtf(q / d + a.eps);      // correctly rounded, as every other norm of the model
        if (lane == 0) inv_s[b] = inv;
        v *= inv;
      }
      out(k, b, tile * TILE + lane, v);
    }
    compute_sync();
  };
  auto finished = [&](int kind) {      // after the stores of all threads have been issued
    if (tid == 0) count_one(a.hints + kind * 32);
  };
  // 32 neighbouring columns of a row, one a lane
  auto store_row = [&](uint4* row, int col, float v, uint32_t name) {
    const uint32_t w0 = pack2(v, __shfl_down_sync(0xffffffffu, v, 1)), w1 = __shfl_down_sync(0xffffffffu, w0, 2), w2 = __shfl_down_sync(0xffffffffu, w0, 4);
    if ((lane & 15) % 6 == 0) named_store(row + words_of(col) + (lane & 15) / 6, w0, w1, w2, name);
  };
  // One thread waits until `count` items of a kind are done, so that the other 255, and all other blocks, do not keep asking L2 for
  // words that nobody has written: that made a hand-over of eight rows of 1280 5 to 11 us long where 2 do (the more blocks waited, the
  // longer).  The count carries no order: the words' names say what has arrived.
  const bool counted = B * pitch > 2 * THREADS;
  auto wait_for = [&](int kind, uint32_t count) {
    if (!counted) return;
    if (tid == 0) {
      const unsigned int* p = a.hints + kind * 32;
      for (int spin = 0; spin < SPIN_LIMIT >> 4; spin++) {
        if (counted_so_far(p) >= count || ((spin & 63) == 63 && *(volatile int*)&given_up)) break;
      }
    }
    compute_sync();
  };
  // Rows of X, all of `src`.  All loads of a thread are in flight together (8: eight rows of 1280 and a few; one in most steps of few columns).
  // Every round of polls writes every v: what it left as it was would stay in registers beside the new (700 bytes of spills, 16 us more a
  // token of d12).
  auto rows_of = [&](const uint4* src, uint32_t name) {
    constexpr int U = 8;
    const int n = B * pitch, last = pitch - 1;      // (the word that a row has too much is nobody's)
    for (int i0 = tid; i0 < n; i0 += THREADS * U) {
      uint4 v[U];
      bool need[U];
#pragma unroll
      for (int u = 0; u < U; u++) need[u] = i0 + u * THREADS < n && (i0 + u * THREADS) % pitch != last;
      if (!counted && need[0]) {
        const int at = i0 & ~31;
        const uint4* one = src + at + (at % pitch == last ? 1 : 0);
        until([&] { return named_load(one).w == name; });
      }
      until([&] {
        bool ok = true;
        auto ask = [&](int u) {
          v[u] = make_uint4(0, 0, 0, name);
          if (need[u]) v[u] = named_load(src + i0 + u * THREADS);
          ok &= v[u].w == name;
        };
        ask(0); ask(1);
        if (i0 - tid + 2 * THREADS < n) {
#pragma unroll
          for (int u = 2; u < U; u++) ask(u);
        } else {
#pragma unroll
          for (int u = 2; u < U; u++) v[u] = make_uint4(0, 0, 0, 0);
        }
        return ok;
      });
#pragma unroll
      for (int u = 0; u < U; u++)
        if (need[u]) X[i0 + u * THREADS] = v[u];
    }
    compute_sync();
  };
  const long long Bd = (long long)B * d;
  const int G = a.H / a.Hkv, n_attn = B * a.Hkv * a.splits;

  for (int l = 0; l < a.L; l++) {
    const DecodeBlock& blk = blocks[l];
    const uint32_t name = launch * (a.L + 1) + l + 1;
    // ---- norm, QKV ----
    if (int j = first_item(4 * l); j < items.x) {
      wait_for(HINT_ROWS, l * (d / TILE));
      rows_of(a.xn, name);
      const bool first = j == 0;
      for (; j < items.x; j += grid) {
        product(j, true, [&](int, int b, int col, float v) { named_store(a.qkv + (long long)b * a.dq + col, v, name); });
        finished(HINT_QKV);
      }
      if (first)       // the first sixteen of the normalised row, for the gate of the value embeddings
        for (int i = tid; i < 16 * B; i += THREADS) {
          const int b = i >> 4, k = i & 15;
          const uint32_t pair = reinterpret_cast<const uint32_t*>(X + b * pitch)[place(k >> 1)];
          named_store(a.h16 + i, (k & 1 ? hi_f(pair) : lo_f(pair)) * inv_s[b], name);
        }
      compute_sync();
    }
    // ---- attention: one item is a column's key head and a range of its keys ----
    int j = first_item(4 * l) - items.x % grid;
    if (j < 0) j += grid;
    for (; j < n_attn; j += grid) {
      const int sp = j % a.splits, kvh = j / a.splits % a.Hkv, b = j / a.splits / a.Hkv;
      int lo = max(0, a.t - blk.window);
      if (a.docs) lo = max(lo, a.doc_start[b]);
      const int nk = a.t - lo, per = (nk + a.splits - 1) / a.splits;       // cached keys; the new one goes with the last range
      const int k0 = min(a.t, lo + sp * per), n_old = min(a.t, k0 + per) - k0;
      const bool last = sp == a.splits - 1;
      bf16* Kb = blk.K + (long long)b * a.maxT * a.kv + (long long)kvh * HD;
      bf16* Vb = blk.V + (long long)b * a.maxT * a.kv + (long long)kvh * HD;
      // half a warp takes every sixteenth key, U at a time; a lane has eight channels.  What does not depend on the projections -
      // rotation, value embedding, cached keys and values - is on its way before they are waited for.
      const int hl = lane & 15, str = warp * 2 + (lane >> 4);
      constexpr int U = GMAX > 2 ? 2 : 4;
      uint4 kr[U], vr[U];
      auto cached = [&](int at) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
          const long long k = at + 16 * u + str;
          if (k < n_old) {
            kr[u] = *reinterpret_cast<const uint4*>(Kb + (k0 + k) * a.kv + hl * 8);
            vr[u] = *reinterpret_cast<const uint4*>(Vb + (k0 + k) * a.kv + hl * 8);
          }
        }
      };
      for (int i = tid + 64 * U; i < n_old * 4; i += THREADS) {
        const bf16* r = (i & 2 ? Vb : Kb) + (long long)(k0 + (i >> 2)) * a.kv + (i & 1) * 64;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(r));
      }
      const long long rot = (long long)a.pos[b] * (HD / 2) + 2 * lane;
      const float2 cs = *reinterpret_cast<const float2*>(a.cos_t + rot), sn = *reinterpret_cast<const float2*>(a.sin_t + rot);
      uint2 ve = make_uint2(0, 0);
      float wg = 0.f;
      if (last && blk.ve) {
        ve = *reinterpret_cast<const uint2*>(blk.ve + (long long)a.tok0[b] * a.kv + (long long)kvh * HD + 4 * lane);
        if (lane < 12) wg = a.theta[blk.ve_gate + lane * a.Hkv + kvh];
      }
      cached(0);
      wait_for(HINT_QKV, (l + 1) * items.x);
      // queries, and with the last range the new key and value: one warp a vector
      for (int v = warp; v < G + (last ? 2 : 0); v += WARPS) {
        const int col = v < G ? (kvh * G + v) * HD : d + (v - G) * a.kv + kvh * HD;
        const uint2* src = a.qkv + (long long)b * a.dq + col;
        uint4 p, q;
        const int at = v <= G ? 2 * lane : 4 * lane;
        until([&] {
          p = named_load2(src + at); q = named_load2(src + at + (v <= G ? 64 : 2));
          return p.y == name && p.w == name && q.y == name && q.w == name;
        });
        float4 x = make_float4(__uint_as_float(p.x), __uint_as_float(p.z), __uint_as_float(q.x), __uint_as_float(q.z));
        if (v <= G) {        // channels 2 lane, 2 lane + 1 and their partners 64 further
          const float c0 = round_to<bf16>(cs.x), c1 = round_to<bf16>(cs.y), s0 = round_to<bf16>(sn.x), s1 = round_to<bf16>(sn.y);
          const float y0 = x.x * c0 + x.z * s0, y1 = x.y * c1 + x.w * s1, z0 = -x.x * s0 + x.z * c0, z1 = -x.y * s1 + x.w * c1;
          const float r = 1.2f / sqrtf(warp_sum(y0 * y0 + y1 * y1 + z0 * z0 + z1 * z1) / HD + a.eps);
          if (v < G) {
            const float f = r * rsqrtf((float)HD);
            *reinterpret_cast<float2*>(&qs[v][2 * lane]) = make_float2(y0 * f, y1 * f);
            *reinterpret_cast<float2*>(&qs[v][64 + 2 * lane]) = make_float2(z0 * f, z1 * f);
          } else {
            const uint32_t lo2 = pack2(y0 * r, y1 * r), hi2 = pack2(z0 * r, z1 * r);
            bf16* dst = Kb + (long long)a.t * a.kv;
            *reinterpret_cast<uint32_t*>(dst + 2 * lane) = lo2;
            *reinterpret_cast<uint32_t*>(dst + 64 + 2 * lane) = hi2;
            kvs[0][2 * lane] = lo_f(lo2); kvs[0][2 * lane + 1] = hi_f(lo2);
            kvs[0][64 + 2 * lane] = lo_f(hi2); kvs[0][65 + 2 * lane] = hi_f(hi2);
          }
        } else {
          if (blk.ve) {
            const float pre = warp_sum(lane < 12 ? word(a.h16 + b * 16 + lane, name) * wg : 0.f);
            const float gate = 3.f / (1.f + expf(-pre));
            x.x += gate * lo_f(ve.x); x.y += gate * hi_f(ve.x); x.z += gate * lo_f(ve.y); x.w += gate * hi_f(ve.y);
          }
          const uint32_t lo2 = pack2(x.x, x.y), hi2 = pack2(x.z, x.w);
          *reinterpret_cast<uint2*>(Vb + (long long)a.t * a.kv + 4 * lane) = make_uint2(lo2, hi2);
          kvs[1][4 * lane] = lo_f(lo2); kvs[1][4 * lane + 1] = hi_f(lo2); kvs[1][4 * lane + 2] = lo_f(hi2); kvs[1][4 * lane + 3] = hi_f(hi2);
        }
      }
      compute_sync();
      constexpr int QR = GMAX > 2 ? 1 : GMAX;      // many heads: their queries stay in shared memory
      float q[QR][8], o[GMAX][8] = {}, m[GMAX], lsum[GMAX] = {};
#pragma unroll
      for (int h = 0; h < GMAX; h++) {
        m[h] = -INFINITY;
        if (h >= QR) continue;
#pragma unroll
        for (int e = 0; e < 8; e++) q[h][e] = h < G ? qs[h][hl * 8 + e] : 0.f;
      }
      const int n_keys = n_old + (last ? 1 : 0);
      for (int base = 0; base < n_keys; base += 16 * U) {
        float kf[U][8], vf[U][8];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int k = base + 16 * u + str;
          ok[u] = k < n_keys;
          const uint32_t pk[4] = {kr[u].x, kr[u].y, kr[u].z, kr[u].w}, pv[4] = {vr[u].x, vr[u].y, vr[u].z, vr[u].w};
#pragma unroll
          for (int e = 0; e < 8; e++) {
            kf[u][e] = e & 1 ? hi_f(pk[e >> 1]) : lo_f(pk[e >> 1]);
            vf[u][e] = e & 1 ? hi_f(pv[e >> 1]) : lo_f(pv[e >> 1]);
          }
          if (k == n_old && last) {
#pragma unroll
            for (int e = 0; e < 8; e++) { kf[u][e] = kvs[0][hl * 8 + e]; vf[u][e] = kvs[1][hl * 8 + e]; }
          }
        }
        if (base + 16 * U < n_old) cached(base + 16 * U);
#pragma unroll
        for (int h = 0; h < GMAX; h++) {
          if (h >= G) break;
          float s[U], mn = m[h];
#pragma unroll
          for (int u = 0; u < U; u++) {
            s[u] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e++) s[u] = fmaf(GMAX > 2 ? qs[h][hl * 8 + e] : q[h < QR ? h : 0][e], kf[u][e], s[u]);
          }
#pragma unroll
          for (int x = 8; x > 0; x >>= 1)
#pragma unroll
            for (int u = 0; u < U; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], x);
#pragma unroll
          for (int u = 0; u < U; u++)
            if (ok[u]) mn = fmaxf(mn, s[u]);
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
      // and the ranges, in order, by the block that has the first (several ranges: an item a block, so nobody it waits for waits for it)
      for (int i = tid; i < G * HD; i += THREADS) {
        const int h = i / HD, ch = i % HD;
        float M = -INFINITY, L = 0.f, v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; w++) M = fmaxf(M, red[(w * GMAX + h) * (HD + 4) + HD]);
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
          const float* r = red + (w * GMAX + h) * (HD + 4);
          const float f = r[HD] == -INFINITY ? 0.f : __expf(r[HD] - M);
          L += r[HD + 1] * f; v += r[ch] * f;
        }
        const long long head = (long long)b * a.H + kvh * G + h;
        uint2* part = a.att_part + head * MAX_SPLITS * (HD + 2);
        if (sp > 0) {
          part += sp * (HD + 2);
          named_store(part + 2 + ch, v, name);
          if (ch < 2) named_store(part + ch, ch ? L : M, name);
          continue;
        }
        for (int s0 = 1; s0 < a.splits; s0 += 4) {
          uint4 ml[4];
          uint2 ov[4];
          until([&] {
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int s = min(s0 + u, a.splits - 1);
              ml[u] = named_load2(part + s * (HD + 2));
              ov[u] = named_load(part + s * (HD + 2) + 2 + ch);
              ok &= ml[u].y == name && ml[u].w == name && ov[u].y == name;
            }
            return ok;
          });
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const float ms = s0 + u < a.splits ? __uint_as_float(ml[u].x) : -INFINITY, mn = fmaxf(M, ms);
            if (mn == -INFINITY) continue;
            const float f = M == -INFINITY ? 0.f : __expf(M - mn), e = ms == -INFINITY ? 0.f : __expf(ms - mn);
            L = L * f + __uint_as_float(ml[u].z) * e; v = v * f + __uint_as_float(ov[u].x) * e; M = mn;
          }
        }
        store_row(a.att + (long long)b * pitch, (kvh * G + h) * HD + ch, v / L, name);
      }
      compute_sync();
      if (sp == 0) finished(HINT_ATT);
    }
    // ---- output projection ----
    if (int j2 = first_item(4 * l + 1); j2 < items.y) {
      float x[NT];      // the stream, on its way before the attention is waited for
      auto stream = [&] {
#pragma unroll
        for (int k = 0; k < NT; k++) {
          const int b = warp + 8 * k;
          x[k] = b < B ? word(a.xm + (long long)b * d + j2 * TILE + lane, name) : 0.f;
        }
      };
      wait_for(HINT_ROWS, l * (d / TILE));
      stream();
      wait_for(HINT_ATT, (l + 1) * B * a.Hkv);
      rows_of(a.att, name);
      for (;;) {
        product(j2, false, [&](int k, int b, int col, float v) {
          v += x[k];
          named_store(a.xa + (long long)b * d + col, v, name);
          store_row(a.xa2 + (long long)b * pitch, col, v, name);
        });
        finished(HINT_MID);
        if ((j2 += grid) >= items.y) break;
        stream();
      }
    }
    // ---- norm, MLP up ----
    if (int j2 = first_item(4 * l + 2); j2 < items.z) {
      wait_for(HINT_MID, (l + 1) * (d / TILE));
      rows_of(a.xa2, name);
      for (; j2 < items.z; j2 += grid) {
        product(j2, true, [&](int, int b, int col, float v) {
          v = fmaxf(v, 0.f);
          const int ks = col / d;      // the same for the 32 columns
          store_row(a.up + ((long long)ks * B + b) * pitch, col - ks * d, v * v, name);
        });
        finished(HINT_UP + j2 / (d / TILE));
      }
    }
    // ---- MLP down: a quarter of the inner rows an item ----
    if (int j2 = first_item(4 * l + 3), tiles = d / TILE; j2 < items.w) {
      const int first = j2;
      for (; j2 < items.w; j2 += grid) {
        const int ks = j2 / tiles;
        wait_for(HINT_UP + ks, (l + 1) * tiles);
        rows_of(a.up + ks * (long long)B * pitch, name);
        product(j2 - ks * tiles, false, [&](int, int b, int col, float v) { named_store(a.part + ks * Bd + (long long)b * d + col, v, name); });
        finished(HINT_PART);
      }
      // the stream after the block, by who had the first quarter of its columns: the next block's mix, or what the head reads
      const bool end = l + 1 == a.L;
      const float lb = end ? 0.f : a.theta[blocks[l + 1].lam_b], l0 = end ? -a.theta[a.off_lam_y] : a.theta[blocks[l + 1].lam_x0];
      if (first < tiles) wait_for(HINT_PART, (l + 1) * items.w);
      for (int t = first; t < tiles; t += grid) {
#pragma unroll
        for (int k = 0; k < NT; k++) {
          const int b = warp + 8 * k, col = t * TILE + lane;
          if (b >= B) break;
          const long long at = (long long)b * d + col;
          const float e = a.x0[at];
          uint2 w[5];
          until([&] {
            w[0] = named_load(a.xa + at);
            bool ok = w[0].y == name;
#pragma unroll
            for (int s = 0; s < 4; s++) { w[1 + s] = named_load(a.part + s * Bd + at); ok &= w[1 + s].y == name; }
            return ok;
          });
          float x = __uint_as_float(w[0].x);
#pragma unroll
          for (int s = 0; s < 4; s++) x += __uint_as_float(w[1 + s].x);
          if (l == a.backout && !end) named_store(a.xb + at, x, name);
          if (end) x += l0 * (l == a.backout ? x : word(a.xb + at, launch * (a.L + 1) + a.backout + 1));
          else { x = lb * x + l0 * e; named_store(a.xm + at, x, name + 1); }
          store_row(a.xn + (long long)b * pitch, col, x, name + 1);
        }
        compute_sync();
        finished(HINT_ROWS);
      }
    }
  }
  // ---- norm, head ----
  if (int j = first_item(4 * a.L); j < a.Vp / TILE) {
    wait_for(HINT_ROWS, a.L * (d / TILE));
    rows_of(a.xn, (launch + 1) * (a.L + 1));
    for (; j < a.Vp / TILE; j += grid)
      product(j, true, [&](int, int b, int col, float v) { if (col < a.V) a.logits[(long long)b * a.V + col] = 15.f * tanhf(v / 15.f); });
  }
}

size_t red_bytes(int nt, int gmax) { return std::max((size_t)4 * WARPS * 8 * nt * RED_PITCH, (size_t)4 * WARPS * gmax * (HD + 4)); }
size_t smem_bytes(int d, int L, int nt, int gmax) { return (size_t)8 * nt * pitch_of(d) * 16 + red_bytes(nt, gmax) + sizeof(DecodeBlock) * L; }      // beside the ring

// blocks that stay on the device together, or 0.  The limit of dynamic shared memory belongs to the function and the device, not to
// a model, so it is always set to all that a block may have: caches of several models decode in turn.
// `ring`: slots that fit beside the rest, 160 KB of them at most (a share of the weights of two or three phases ahead).
template <int NT, int GMAX, int KS> int resident_blocks(size_t smem, int& ring) {
  auto kernel = k_decode_step<NT, GMAX, KS>;
  int per = 0, dev = 0, most = 0;
  cudaFuncAttributes fixed;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fixed, kernel) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fixed.sharedSizeBytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const long long left = most - (long long)fixed.sharedSizeBytes - (long long)smem;
  ring = (int)std::min<long long>(left, 160 * 1024) / slot_bytes(KS);
  if (left < 0 || ring < MIN_RING) return 0;
  smem += (size_t)ring * slot_bytes(KS);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, THREADS + 128, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per > 0 ? device_sm_count() : 0;
}
int steps_of(int d) { return d % 256 ? 1 : 2; }      // slots are 128 or 256 rows
int resident(int nt, int gmax, int ks, size_t smem, int& ring) {
  if (ks == 1) {
    if (nt == 1) return gmax == 2 ? resident_blocks<1, 2, 1>(smem, ring) : resident_blocks<1, 8, 1>(smem, ring);
    return gmax == 2 ? resident_blocks<2, 2, 1>(smem, ring) : resident_blocks<2, 8, 1>(smem, ring);
  }
  if (nt == 1) return gmax == 2 ? resident_blocks<1, 2, 2>(smem, ring) : resident_blocks<1, 8, 2>(smem, ring);
  return gmax == 2 ? resident_blocks<2, 2, 2>(smem, ring) : resident_blocks<2, 8, 2>(smem, ring);
}

}  // namespace

// bf16, heads of 128 channels (so every width is a multiple of 128), at most 8 query heads a key head, d up to 4096, and as many columns as
// leave room for MIN_RING slots of the ring: 8, or 16 up to d = 2816 (2560 with more than two query heads a key head; odd multiples of 128
// have slots of half the size and go up to 3456 and 3200).  Anything else takes the chain of kernels of decode.cu.
void decode_step_plan(const femto_handle* h, int max_batch, DecodeStepState& st) {
  st.blocks_n = st.columns = 0;
  if (!h->bf || h->hd != HD || (h->d & 127) || (h->Vp & (TILE - 1)) || h->H % h->Hkv || h->H / h->Hkv > 8 || h->d > 128 * 32) return;
  const int gmax = h->H / h->Hkv <= 2 ? 2 : 8;
  for (int nt = 1; nt <= (max_batch > 8 ? 2 : 1); nt++) {
    const int n = resident(nt, gmax, steps_of(h->d), smem_bytes(h->d, h->L, nt, gmax), st.ring[nt - 1]);
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
  char* first = p;
  st.hint_bytes = 128 * HINTS;
  take(st.launches, 8); take(st.hints, st.hint_bytes);
  const size_t words = 16 * n * pitch_of(h->d);
  take(st.xn, words); take(st.xm, 8 * n * d); take(st.xa, 8 * n * d); take(st.xa2, words); take(st.xb, 8 * n * d);
  take(st.part, 32 * n * d); take(st.qkv, 8 * n * h->dq); take(st.h16, 8 * 16 * n); take(st.up, 4 * words); take(st.att, words);
  take(st.att_part, 8 * n * h->H * MAX_SPLITS * (HD + 2));
  st.named_bytes = p - first;
  take(st.x0, 4 * n * d);
}

int decode_step_setup(const femto_handle* h, DecodeStepState& st, const std::vector<void*>& K, const std::vector<void*>& V) {
  std::vector<CUtensorMap> maps;
  std::vector<DecodeBlock> bl;
  auto put = [&](const void* W, int rows, int cols) {      // boxes of 128 or 256 rows and 32 columns, 64-byte swizzle: one slot of the ring
    maps.emplace_back();
    return make_tmap_3d_bf16_sw(&maps.back(), W, cols, rows, 1, cols, 0, TILE, 128 * steps_of(h->d), 2);
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
  CUDA_TRY(cudaMemset(st.launches, 0, st.named_bytes));      // no word has a name yet
  CUDA_TRY(cudaMemcpy(st.maps, maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));      // the caller's stream may be one that does not wait for the legacy stream
  return 0;
}

int decode_step_run(const femto_handle* h, const DecodeStepState& st, DecodeStepArgs a, const int* tokens, const int* positions, cudaStream_t s, bool* ran) {
  a.blocks = st.blocks; a.maps = st.maps; a.launches = st.launches; a.hints = st.hints; a.x0 = st.x0;
  a.xn = st.xn; a.xm = st.xm; a.xa = st.xa; a.xa2 = st.xa2; a.xb = st.xb; a.part = st.part; a.qkv = st.qkv; a.h16 = st.h16; a.up = st.up;
  a.att = st.att; a.att_part = st.att_part;
  a.wte = (const bf16*)h->sh_wte; a.sin_t = h->sin_t; a.cos_t = h->cos_t; a.status = h->status;
  a.off_smear = h->off_smear; a.off_lam_s = h->off_lam_s; a.off_lam_y = h->off_lam_y;
  a.d = h->d; a.dq = h->dq; a.kv = h->kv; a.H = h->H; a.Hkv = h->Hkv; a.V = h->V; a.Vp = h->Vp; a.L = h->L; a.backout = h->backout; a.eps = h->eps;
  a.docs = h->cfg.doc_mask ? 1 : 0;
  // ranges of about 64 keys, as many as there are blocks for
  int keys = 0;
  for (const LayerP& p : h->lp) keys = std::max(keys, std::min(a.t + 1, p.window + 1));
  a.splits = std::max(1, std::min({MAX_SPLITS, cdiv(keys, 64), st.blocks_n / (a.B * a.Hkv)}));
  if (tokens) {
    k_step_begin<<<a.B, THREADS, 0, s>>>(a, tokens, positions, h->cfg.index_base, h->V, h->cfg.max_document_tokens);
    KERNEL_CHECK();
  } else {      // the self test: words of a launch that nobody writes
    CUDA_TRY(cudaMemsetAsync(st.launches + 1, 0x5a, 4, s));
  }
  const int nt = a.B <= 8 ? 1 : 2, gmax = a.H / a.Hkv <= 2 ? 2 : 8;
  a.ring = st.ring[nt - 1];
  const size_t smem = smem_bytes(a.d, a.L, nt, gmax) + (size_t)a.ring * slot_bytes(steps_of(a.d));
  a.red_bytes = (int)red_bytes(nt, gmax);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = st.blocks_n; cfg.blockDim = THREADS + 128; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;      // the blocks wait for one another: all of them are resident or none is
  at[0].val.cooperative = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  cudaError_t e;
#define LAUNCH(NT, GM) e = steps_of(a.d) == 2 ? cudaLaunchKernelEx(&cfg, k_decode_step<NT, GM, 2>, a) : cudaLaunchKernelEx(&cfg, k_decode_step<NT, GM, 1>, a)
  if (nt == 1) { if (gmax == 2) LAUNCH(1, 2); else LAUNCH(1, 8); }
  else { if (gmax == 2) LAUNCH(2, 2); else LAUNCH(2, 8); }
#undef LAUNCH
  // a context or stream with fewer multiprocessors than the device has: nothing is lost, the caller takes the chain of kernels
  *ran = e != cudaErrorCooperativeLaunchTooLarge;
  if (!*ran) { cudaGetLastError(); return 0; }
  CUDA_TRY(e);
  KERNEL_CHECK();
  return 0;
}
