// Hyena operator on the tensor cores: the long convolution of a channel by blocks of 16 tokens.
//
// Within a block behind state S (8 complex modes)   c[n] = sum_{k<=n} h[n-k] x[k] + Re sum_s R_s p_s^{n+1} S_s   (n = 0..15)
// and                                               S'  = p^16 S + E,   E_s = sum_k p_s^{15-k} x[k],
// so with the blocks of one channel as the 16 rows of an mma.sync tile the three sums are products with constants of the channel:
// X (16 x 16 tokens) . T (16 x 16 outputs), X . P (16 x 16: re, im of 8 modes) and S (16 x 16) . Q (16 x 16 outputs).
// Precision is fp32's: x is bf16 as it stands; T, P, Q are computed in 64 bits and enter as three bf16 parts (24 bits), S (fp32) as three
// parts too, with all six products down to 2^-16 of the leading one; sums are fp32.  What was 48 fp32 multiply-adds per token and channel on
// the CUDA cores is 24 mma per 256 tokens and channel.
//
// An item is 32 channels x one batch row x one segment of L, walked in tiles of 16 rows x R blocks (256 R tokens); row r owns R consecutive blocks.
//   producer           copies the raw rows of x1, v and x2 (32 channels x 128 tokens and the two in front) into a ring of slots
//   element-wise warps A: thread = (channel quad, 8 tokens): FIR of x1 and v, x1*v, transposed through registers: 8 tokens of a channel per 16 bytes
//                      C: FIR of x2, product with what the tensor-core warps left in the place of x, store.  A of tile q + 1 runs before C of tile q
//   tensor-core warps  B: a channel at a time: E of all blocks; the rows' ends folded over the 8 lanes that hold a fragment column's rows (three shuffle
//                      steps with powers p^{16R}, p^{32R}, p^{64R}); then every block's c, rounded, + D x, back into the place of x
// The fragment layouts of A operands and sums agree (a lane owns 4 consecutive tokens of rows g and g + 8), so B needs no shuffle besides the fold.
// z is read once and y written once.
// Measured (B200, D = 4096, constants included): 8 x 8193 tokens 834 us sustained (modal scan on the CUDA cores 953), 1 x 1999 41.5 us (138), 4 x 1000 76 us (123), 1 x 301 20 us (42).
// A steady tile of 1024 tokens takes 24.5 k cycles, all of them the tensor-core warps' (tensor pipe 6.7 k, fp32 pipe 9 k, issue 10 k per scheduler): bound by the
// latencies of its dependent steps with two such warps per scheduler (5.6 cycles per instruction each, by clock stamps; ncu on 1 x 8193: issue slots 59 % used, tensor pipe 23 %).  Register shares of 128 / 88 or 136 / 80
// are 2 - 3 % slower: the element-wise warps then spill more (the output kernels spill 16 to 112 bytes as it is, -Xptxas -v).
// A channel whose x or state is not finite (or beyond 1e30), or whose poles lie so far outside the unit circle that their powers are not, goes
// token by token in that tile: a product with a structural zero would otherwise carry an infinity to earlier tokens of its block.
#pragma once
#include "waits.cuh"

namespace evo_hytc {

using namespace evo;

constexpr int NS = 8;
constexpr int CH = 32;                       // channels per item
constexpr int ROWS = 16;                     // rows of an mma tile
constexpr int BLK = 16;                      // tokens of a block
constexpr int MMA_WARPS = 8, EW_WARPS = 8;
constexpr int THREADS = (MMA_WARPS + EW_WARPS + 4) * 32;      // the last warpgroup: one producer lane
// registers: 640 threads are launched with 96 each; the warpgroups then share them out
constexpr int MMA_REGS = 120, EW_REGS = 96, PRODUCER_REGS = 40;
static_assert(MMA_WARPS * 32 * MMA_REGS + EW_WARPS * 32 * EW_REGS + 128 * PRODUCER_REGS <= THREADS * 96, "register shares exceed the launch");
constexpr int STAGE = 128;                   // tokens of a ring slot (one signal), with two rows in front
constexpr int SLOTS = 6;
constexpr int SLOT_BYTES = (STAGE + 2) * CH * 2;
constexpr int TAB_WORDS = 36;                // fragment words per lane and channel: P, T, Q (12 each)
constexpr int POW_ROWS = 9;                  // p^16, then p^{16 R k} for k = 1..8
constexpr int CONST_BYTES = TAB_WORDS * 32 * 4 + POW_ROWS * NS * 8;       // of one channel (a multiple of 16)

struct Args {
  const bf16* z; bf16* y;
  const bf16* fir_w; const bf16* fir_b; const bf16* Dskip;
  const float* poles; const float* residues;
  const bf16* halo; const float* state_in; float* state_out;
  float* seg_states;                         // (B, nseg, D, 8, 2) zero-start end states of the segments
  const uint8_t* consts;                     // (D, CONST_BYTES): 9 x 32 x 16 bytes of fragment words, then (9, 8) powers
  const float2* seg_pow;                     // (D, 8) p^seg_len
  int B, D, nseg, items, y_wide;
  long long L, seg_len;
  WaitLimit waits;
};

constexpr size_t table_bytes(int D) { return (size_t)D * (CONST_BYTES + NS * 8); }
constexpr int smem_bytes(int R) { return SLOTS * SLOT_BYTES + 2 * CH * ROWS * BLK * 2 * R + MMA_WARPS * CONST_BYTES + CH * NS * 8 * 2 + CH * 32 + CH * 4 + (2 * SLOTS + 4) * 8; }

__device__ __forceinline__ uint32_t mulbf(uint32_t a, uint32_t b) { uint32_t d; asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t addbf(uint32_t a, uint32_t b) { uint32_t d; asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ float2 up2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {        // sums start from zero
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// ---- the constants of a channel, one warp each, in 64 bits
struct D2 { double r, i; };
__device__ __forceinline__ D2 mul(D2 a, D2 b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
// the fp32 value of a constant as three bf16 parts, cut off: 8 + 8 + 8 bits
__device__ __forceinline__ void parts3(double v, uint32_t (&out)[3]) {
  float f = (float)v;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t t = __float_as_uint(f) & 0xffff0000u;
    out[k] = t >> 16;
    f -= __uint_as_float(t);
  }
}

// the last two inputs of a sequence, for what continues it: element idx = (b, column) of (B, 3D, 2)
__device__ __forceinline__ void fir_state(const bf16* __restrict__ z, const bf16* __restrict__ halo, bf16* __restrict__ out, long long idx, long long L, long long C3) {
  const long long b = idx / C3, c = idx % C3;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long t = L - 2 + k;
    bf16 v = __float2bfloat16_rn(0.f);
    if (t >= 0) v = z[(b * L + t) * C3 + c];
    else if (halo) v = halo[(b * 2 + (t + 2)) * C3 + c];
    out[idx * 2 + k] = v;
  }
}

// The operator's kernel is launched dependent where a call is short: its CTAs start where this one's have ended, and filter their first inputs while the rest of the constants is computed.  The blocks behind
// the channels' copy the inputs that a state keeps, which had a launch of their own (B, L, C3 are theirs; fir_out NULL: none).
constexpr int PREP_WARPS = 4;
__global__ void __launch_bounds__(PREP_WARPS * 32) hyena_tc_constants_kernel(const float* __restrict__ poles, const float* __restrict__ residues, uint8_t* __restrict__ consts,
                                                                             float2* __restrict__ seg_pow, int D, int R, long long seg_len, const bf16* __restrict__ z,
                                                                             const bf16* __restrict__ halo, bf16* __restrict__ fir_out, int B, long long L) {
  pdl_wait();                                               // itself launched dependent: what it writes may still be read, and what the operator reads before its own wait must be there
  pdl_launch_dependents();
  if ((int)blockIdx.x >= D / PREP_WARPS) {
    const long long idx = (long long)(blockIdx.x - D / PREP_WARPS) * (PREP_WARPS * 32) + threadIdx.x;
    if (idx < (long long)B * 3 * D) fir_state(z, halo, fir_out, idx, L, 3ll * D);
    return;
  }
  __shared__ D2 pw[PREP_WARPS][NS][BLK + 1];
  __shared__ D2 rq[PREP_WARPS][NS][BLK + 1];                // R_s p_s^k
  __shared__ double h[PREP_WARPS][BLK];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, ch = blockIdx.x * PREP_WARPS + w;
  if (ch >= D) return;
  const int s = lane & 7, q = lane >> 3;
  const float2 pf = reinterpret_cast<const float2*>(poles)[(long long)ch * NS + s], rf = reinterpret_cast<const float2*>(residues)[(long long)ch * NS + s];
  const D2 p = {pf.x, pf.y}, r = {rf.x, rf.y};
  // lane (s, q) computes p^k for k = 4q .. 4q + 3
  const D2 p2 = mul(p, p), p4 = mul(p2, p2), p8 = mul(p4, p4), p16 = mul(p8, p8);
  D2 v = {1.0, 0.0};
  if (q & 1) v = p4;
  if (q & 2) v = (q & 1) ? mul(p8, p4) : p8;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    pw[w][s][4 * q + k] = v;
    rq[w][s][4 * q + k] = mul(r, v);
    v = mul(v, p);
  }
  if (q == 3) { pw[w][s][BLK] = p16; rq[w][s][BLK] = mul(r, p16); }
  if (q == 0) {
    float2* out = reinterpret_cast<float2*>(consts + (size_t)ch * CONST_BYTES + TAB_WORDS * 128) + s;
    out[0] = make_float2((float)p16.r, (float)p16.i);
    D2 row = p16;
    for (int k = 1; k < R; k <<= 1) row = mul(row, row);      // p^{16 R}, R a power of two
    D2 u = row;
#pragma unroll
    for (int k = 1; k <= 8; ++k) { out[k * NS] = make_float2((float)u.r, (float)u.i); u = mul(u, row); }
  } else if (q == 1 && seg_len > 0) {
    D2 acc = {1.0, 0.0}, b = p;
    for (long long n = seg_len; n > 0; n >>= 1) { if (n & 1) acc = mul(acc, b); b = mul(b, b); }
    seg_pow[(long long)ch * NS + s] = make_float2((float)acc.r, (float)acc.i);
  }
  __syncwarp();
  if (lane < BLK) {
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < NS; ++m) acc += rq[w][m][lane].r;
    h[w][lane] = acc;
  }
  __syncwarp();
  const int g = lane >> 2, tq = lane & 3;
  uint32_t word[TAB_WORDS];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int reg = 0; reg < 2; ++reg) {
      const int k0 = 4 * tq + 2 * reg;                         // the two tokens (P, T) of this register; for Q: the mode
      const int n = 4 * (g >> 1) + 2 * nt + (g & 1);           // the output token of column g
      const int mode = 4 * nt + (g >> 1), m = 4 * reg + tq;
      const D2 pa = pw[w][mode][BLK - 1 - k0], pb = pw[w][mode][BLK - 2 - k0];
      const double vals[3][2] = {{(g & 1) ? pa.i : pa.r, (g & 1) ? pb.i : pb.r},
                                 {n >= k0 ? h[w][n - k0 < 0 ? 0 : n - k0] : 0.0, n >= k0 + 1 ? h[w][n - k0 - 1 < 0 ? 0 : n - k0 - 1] : 0.0},
                                 {rq[w][m][n + 1].r, -rq[w][m][n + 1].i}};
#pragma unroll
      for (int kind = 0; kind < 3; ++kind) {
        uint32_t a3[3], b3[3];
        parts3(vals[kind][0], a3); parts3(vals[kind][1], b3);
#pragma unroll
        for (int k = 0; k < 3; ++k) word[kind * 12 + (nt * 2 + reg) * 3 + k] = a3[k] | (b3[k] << 16);
      }
    }
  uint4* t = reinterpret_cast<uint4*>(consts + (size_t)ch * CONST_BYTES) + lane;
#pragma unroll
  for (int i = 0; i < 9; ++i) t[i * 32] = make_uint4(word[4 * i], word[4 * i + 1], word[4 * i + 2], word[4 * i + 3]);
}

__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {        // a b + c
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}
__device__ __forceinline__ float2 shfl_up2(float2 v, int d) { return make_float2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d)); }
__device__ __forceinline__ float2 shfl2(float2 v, int src) { return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)); }
// byte offset of granule `gran` (8 tokens) of row `row` of channel c in the tile: the low three bits of the granule index are mixed with the channel
// quad (phases A and C: 8 lanes = 8 quads) and with the row (phase B: 4 rows x 2 granules), so that both access patterns touch every bank once
template <int R> __device__ __forceinline__ uint32_t cell(int c, int row, int gran) {
  const int rs = R == 4 ? (row & 3) << 1 : (R == 2 ? (row & 2) : 0);
  return (uint32_t)c * (ROWS * BLK * 2 * R) + (uint32_t)(((row * 2 * R + gran) ^ ((c >> 2) & 7) ^ rs) << 4);
}

__device__ __forceinline__ void lds64(uint32_t& a, uint32_t& b, uint32_t addr) { asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr)); }
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) { asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory"); }
__device__ __forceinline__ uint2 ldg64(const bf16* p) { return __ldg(reinterpret_cast<const uint2*>(p)); }
// three taps of four channels (24 consecutive bytes) as two channel pairs, kept as they are stored: [pair][tap] packed, and the biases
struct Taps { uint32_t w[2][3]; uint2 bias; };
__device__ __forceinline__ Taps load_taps(const bf16* fir_w, const bf16* fir_b, int col) {
  const uint2* f = reinterpret_cast<const uint2*>(fir_w + 3LL * col);
  const uint2 q0 = __ldg(f), q1 = __ldg(f + 1), q2 = __ldg(f + 2);
  const uint32_t e[6] = {q0.x, q0.y, q1.x, q1.y, q2.x, q2.y};           // channel 0 taps 0 1 | tap 2, channel 1 tap 0 | taps 1 2 | ..
  Taps t;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    t.w[u][0] = __byte_perm(e[3 * u], e[3 * u + 1], 0x7610);
    t.w[u][1] = __byte_perm(e[3 * u], e[3 * u + 2], 0x5432);
    t.w[u][2] = __byte_perm(e[3 * u + 1], e[3 * u + 2], 0x7610);
  }
  t.bias = ldg64(fir_b + col);
  return t;
}
// short FIR (fp32 accumulate, rounded) + bias (rounded) of one channel pair: eight tokens from ten raw rows; take(e, f) gets each result
template <typename F> __device__ __forceinline__ void fir8(const uint32_t (&wq)[3], uint32_t bias, const uint32_t (&z)[10], F take) {
  const float2 w0 = up2(wq[0]), w1 = up2(wq[1]), w2 = up2(wq[2]);
  float2 h0 = up2(z[0]), h1 = up2(z[1]);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float2 c = up2(z[e + 2]);
    const float2 acc = __ffma2_rn(w2, c, __ffma2_rn(w1, h1, __fmul2_rn(w0, h0)));
    h0 = h1; h1 = c;
    take(e, addbf(pack_bf16(acc.x, acc.y), bias));
  }
}

// a warp's wait: what one lane lost all have lost
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, const WaitLimit& w) { return __all_sync(0xffffffffu, wait_or_give_up(bar, parity, w)); }

// position in the sequence of tiles that a CTA walks: its items (channel block, batch row, segment), tile by tile
struct Walk {
  int item, k, n_tiles, b, seg, ch0, t0, t1;                            // (tokens of a sequence are counted in 32 bits: copy coordinates are)
  __device__ __forceinline__ void open(const Args& a, int tile) {
    const int ncb = a.D / CH;
    ch0 = (item % ncb) * CH; b = (item / ncb) % a.B; seg = item / (ncb * a.B);
    t0 = seg * (int)a.seg_len; t1 = min((int)a.L, t0 + (int)a.seg_len);
    n_tiles = (t1 - t0 + tile - 1) / tile;
    k = 0;
  }
  __device__ __forceinline__ bool more(const Args& a) const { return item < a.items; }
  __device__ __forceinline__ void next(const Args& a, int tile) {
    if (++k < n_tiles) return;
    item += gridDim.x;
    if (item < a.items) open(a, tile);
  }
  __device__ __forceinline__ int first(int tile) const { return t0 + k * tile; }
  __device__ __forceinline__ int tokens(int tile) const { return min(tile, t1 - first(tile)); }
};
// what the second phase of a tile has to know of it
struct Tile {
  int first, n, b, ch0;
  __device__ __forceinline__ void of(const Walk& w, int tile) { first = w.first(tile); n = w.tokens(tile); b = w.b; ch0 = w.ch0; }
};

template <int R, bool STATE_ONLY>
__global__ void __launch_bounds__(THREADS, 1) hyena_tc_kernel(const __grid_constant__ CUtensorMap tmZ, const Args a) {
  constexpr int TILE = ROWS * BLK * R;                 // tokens per tile
  constexpr int HD = 128;
  extern __shared__ __align__(128) uint8_t sm[];
  uint8_t* ring = sm;                                                   // [SLOTS] raw rows of one signal: 2 + STAGE tokens x 32 channels
  uint8_t* xbuf = ring + SLOTS * SLOT_BYTES;                            // [2][CH][TILE] bf16, see cell()
  uint8_t* cons = xbuf + 2 * CH * TILE * 2;                             // [MMA_WARPS] constants of the channel in work
  float2* carry = reinterpret_cast<float2*>(cons + MMA_WARPS * CONST_BYTES);        // [CH][8] state entering the tile
  float2* fin = carry + CH * NS;                                        // [CH][8] state entering the segment's last, unfinished block
  uint32_t* xlast = reinterpret_cast<uint32_t*>(fin + CH * NS);         // [CH][8] that block's x
  int* finm = reinterpret_cast<int*>(xlast + CH * 8);                   // [CH]    and its number of tokens
  uint64_t* zfull = reinterpret_cast<uint64_t*>(finm + CH);
  uint64_t* zempty = zfull + SLOTS;
  uint64_t* xfull = zempty + SLOTS;                                     // [2] x of a tile is complete
  uint64_t* xdone = xfull + 2;                                          // [2] the convolution has replaced it

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < SLOTS; ++i) { mbar_init(&zfull[i], 1); mbar_init(&zempty[i], EW_WARPS / 2); }
    for (int i = 0; i < 2; ++i) { mbar_init(&xfull[i], EW_WARPS); mbar_init(&xdone[i], MMA_WARPS); }
    fence_barrier_init();
  }
  __syncthreads();
  Walk w;
  w.item = blockIdx.x;
  w.open(a, TILE);                                                      // the grid has at most as many CTAs as items

  if (warp >= MMA_WARPS + EW_WARPS) {
    // ================================================ producer: one lane; the order in which the element-wise warps consume
    regs_down<PRODUCER_REGS>();
    if (warp == MMA_WARPS + EW_WARPS && lane == 0) {
      tma_prefetch_desc(&tmZ);
      uint32_t s = 0;                                                   // running slot number
      bool ok = true;
      auto put = [&](int col, int t, int b) {
        const uint32_t i = s % SLOTS, round = s / SLOTS;
        if (ok && round > 0) ok = wait_or_give_up(&zempty[i], (round - 1) & 1, a.waits);
        if (ok) {
          mbar_arrive_expect_tx(&zfull[i], SLOT_BYTES);
          tma_load_3d(ring + i * SLOT_BYTES, &tmZ, &zfull[i], col, t - 2, b);
          ++s;
        }
      };
      auto column = [&](int ch0, int sig) { return (ch0 / HD) * 3 * HD + ch0 % HD + sig * HD; };
      Tile p;
      p.of(w, TILE);
      bool any = false;
      while (ok && (w.more(a) || any)) {
        if (w.more(a))
          for (int i = 0; i * STAGE < w.tokens(TILE); ++i) { put(column(w.ch0, 1), w.first(TILE) + i * STAGE, w.b); put(column(w.ch0, 2), w.first(TILE) + i * STAGE, w.b); }
        if (!STATE_ONLY && any)
          for (int i = 0; i * STAGE < p.n; ++i) put(column(p.ch0, 0), p.first + i * STAGE, p.b);
        any = w.more(a);
        if (any) { p.of(w, TILE); w.next(a, TILE); }
      }
      // the copies still in flight land before this thread ends
      for (uint32_t q = s > SLOTS ? s - SLOTS : 0; q < s; ++q) wait_to_end(&zfull[q % SLOTS], (q / SLOTS) & 1, a.waits);
    }
    return;
  }

  if (warp >= MMA_WARPS) {
    // ================================================ element-wise warps: two groups of four take the stages of 128 tokens in turn;
    // thread = (channel quad, run of 8 tokens)
    regs_down<EW_REGS>();
    const int et = tid - MMA_WARPS * 32, group = et >> 7, quad = et & 7, run = (et >> 3) & 15;
    uint32_t s = 0;                                                     // running slot number (both groups count all slots)
    uint32_t q = 0;                                                     // running tile number
    bool ok = true, any = false;
    Tile p;
    p.of(w, TILE);
    // ten raw rows of this thread's run from slot s, the first two in front of it, as two channel pairs; the slot is then free (and not ok: none)
    auto rows = [&](uint32_t slot, int t, int b, int col, uint32_t (&z)[2][10]) {
      const uint32_t i = slot % SLOTS;
      ok = warp_wait(&zfull[i], (slot / SLOTS) & 1, a.waits);
      if (!ok) return;
      const uint8_t* src = ring + i * SLOT_BYTES + run * 8 * (CH * 2) + quad * 8;
#pragma unroll
      for (int e = 0; e < 10; ++e) { const uint2 v = *reinterpret_cast<const uint2*>(src + e * (CH * 2)); z[0][e] = v.x; z[1][e] = v.y; }
      __syncwarp();
      if (lane == 0) mbar_arrive(&zempty[i]);
      if (t < 2 && a.halo) {
        // in front of a sequence's first token: the carried inputs (the copy filled in zeros)
        const bf16* h = a.halo + (long long)b * 2 * 3 * a.D + col;
        const uint2 v = ldg64(h + t * 3LL * a.D);
        z[0][0] = v.x; z[1][0] = v.y;
        if (t == 0) { const uint2 u = ldg64(h + 3LL * a.D); z[0][1] = u.x; z[1][1] = u.y; }
      }
    };
    while (ok && (w.more(a) || any)) {
      if (w.more(a)) {
        // ---------------- A: x1 * v of tile q
        const int n = w.tokens(TILE), ns = (n + STAGE - 1) / STAGE, ch = w.ch0 + 4 * quad, zc = (ch / HD) * 3 * HD + ch % HD;
        uint8_t* xs = xbuf + (q & 1) * (CH * TILE * 2);
#pragma unroll 1
        for (int i = group; i < TILE / STAGE; i += 2) {
          const int gran = i * (STAGE / 8) + run, row = gran / (2 * R), gr = gran % (2 * R);
          uint32_t x[2][8];
          if (i < ns) {
            const int t = w.first(TILE) + gran * 8;
            uint32_t z[2][10];
            {
              const Taps w1 = load_taps(a.fir_w, a.fir_b, zc + HD);       // (from L1; kept over the stages they would not fit the registers)
              rows(s + 2 * i, t, w.b, zc + HD, z);
              if (!ok) break;
              fir8(w1.w[0], w1.bias.x, z[0], [&](int e, uint32_t f) { x[0][e] = f; });
              fir8(w1.w[1], w1.bias.y, z[1], [&](int e, uint32_t f) { x[1][e] = f; });
            }
            const Taps wv = load_taps(a.fir_w, a.fir_b, zc + 2 * HD);
            rows(s + 2 * i + 1, t, w.b, zc + 2 * HD, z);
            if (!ok) break;
            fir8(wv.w[0], wv.bias.x, z[0], [&](int e, uint32_t f) { x[0][e] = mulbf(x[0][e], f); });
            fir8(wv.w[1], wv.bias.y, z[1], [&](int e, uint32_t f) { x[1][e] = mulbf(x[1][e], f); });
            if (n < TILE) {
#pragma unroll
              for (int e = 0; e < 8; ++e) if (gran * 8 + e >= n) x[0][e] = x[1][e] = 0u;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[0][e] = x[1][e] = 0u;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t (&v)[8] = x[u >> 1];
            const uint32_t sel = (u & 1) ? 0x7632 : 0x5410;
            *reinterpret_cast<uint4*>(xs + cell<R>(4 * quad + u, row, gr)) =
                make_uint4(__byte_perm(v[0], v[1], sel), __byte_perm(v[2], v[3], sel), __byte_perm(v[4], v[5], sel), __byte_perm(v[6], v[7], sel));
          }
        }
        if (!ok) break;                                                 // the tensor-core warps wait in vain and end, too
        s += 2 * ns;
        __syncwarp();
        if (lane == 0) mbar_arrive(&xfull[q & 1]);
      }
      if (any) {
        // ---------------- C: tile q - 1, (convolution + D x) * x2.  The cells are this thread's own: A of tile q + 1 may refill them afterwards
        ok = warp_wait(&xdone[(q - 1) & 1], ((q - 1) >> 1) & 1, a.waits);
        if (!ok) break;
        if (!STATE_ONLY) {
          const int ns = (p.n + STAGE - 1) / STAGE, ch = p.ch0 + 4 * quad, zc = (ch / HD) * 3 * HD + ch % HD;
          const uint8_t* xs = xbuf + ((q - 1) & 1) * (CH * TILE * 2);
#pragma unroll 1
          for (int i = group; i < ns; i += 2) {
            const int gran = i * (STAGE / 8) + run, row = gran / (2 * R), gr = gran % (2 * R);
            const int t = p.first + gran * 8, left = p.n - gran * 8;
            uint32_t z[2][10], o[2][8];
            const Taps w2 = load_taps(a.fir_w, a.fir_b, zc);
            rows(s + i, t, p.b, zc, z);
            if (!ok) break;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              const uint4 lo = *reinterpret_cast<const uint4*>(xs + cell<R>(4 * quad + 2 * v, row, gr)), hi = *reinterpret_cast<const uint4*>(xs + cell<R>(4 * quad + 2 * v + 1, row, gr));
              const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
              fir8(w2.w[v], v ? w2.bias.y : w2.bias.x, z[v], [&](int e, uint32_t f) { o[v][e] = mulbf(__byte_perm(l[e >> 1], h[e >> 1], (e & 1) ? 0x7632 : 0x5410), f); });
            }
            bf16* yr = a.y + ((long long)p.b * a.L + t) * a.D + ch;
            if (left >= 8 && a.y_wide) {
#pragma unroll
              for (int e = 0; e < 8; ++e) *reinterpret_cast<uint2*>(yr + (long long)e * a.D) = make_uint2(o[0][e], o[1][e]);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (e < left) { uint32_t* d = reinterpret_cast<uint32_t*>(yr + (long long)e * a.D); d[0] = o[0][e]; d[1] = o[1][e]; }
            }
          }
          s += ns;
        }
      }
      any = w.more(a);
      if (any) { p.of(w, TILE); w.next(a, TILE); ++q; }
    }
    return;
  }

  // ================================================ tensor-core warps: one channel at a time, channels warp, warp + 8, ..
  regs_up<MMA_REGS>();
  const int g = lane >> 2, tq = lane & 3;
  uint8_t* slot = cons + warp * CONST_BYTES;
  // the constants of the next channel are fetched while the current one is in its last sweep
  auto fetch = [&](int chg) {
    const uint8_t* src = a.consts + (size_t)chg * CONST_BYTES + lane * 16;
    const uint32_t dst = smem_u32(slot) + lane * 16;
#pragma unroll
    for (int i = 0; i < CONST_BYTES / 512; ++i) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512), "l"(src + i * 512) : "memory");
    constexpr int REST = CONST_BYTES % 512 / 16;
    if (lane < REST) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + CONST_BYTES / 512 * 512), "l"(src + CONST_BYTES / 512 * 512) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();                                                           // the constants
  fetch(w.ch0 + warp);
  for (uint32_t q = 0; w.more(a); ++q) {
    const int n = w.tokens(TILE);
    const bool last = w.k == w.n_tiles - 1;
    if (w.k == 0) {
      // carry entering the segment: lane = (one of the warp's four channels, mode)
      const int c = warp + (lane >> 3) * MMA_WARPS, m = lane & 7;
      const long long e = ((long long)w.b * a.D + w.ch0 + c) * NS + m;
      float2 S = make_float2(0.f, 0.f);
      if (!STATE_ONLY) {
        if (a.state_in) S = reinterpret_cast<const float2*>(a.state_in)[e];
        if (w.seg > 0) {
          const float2 pl = a.seg_pow[(long long)(w.ch0 + c) * NS + m];
          for (int k = 0; k < w.seg; ++k) S = cfma(pl, S, reinterpret_cast<const float2*>(a.seg_states)[(((long long)w.b * a.nseg + k) * a.D + w.ch0 + c) * NS + m]);
        }
      }
      carry[c * NS + m] = S;
      __syncwarp();
    }
    uint8_t* xs = xbuf + (q & 1) * (CH * TILE * 2);
    if (!warp_wait(&xfull[q & 1], (q >> 1) & 1, a.waits)) break;
#pragma unroll 1
    for (int c = warp; c < CH; c += MMA_WARPS) {
      const int chg = w.ch0 + c;
      float2 E[R][2][2], F[2][2];                                      // [block][rows g | g + 8][mode tq | tq + 4]
      const uint32_t dsk = STATE_ONLY ? 0u : (uint32_t)__bfloat16_as_ushort(a.Dskip[chg]) * 0x10001u;
      const float2 S0[2] = {carry[c * NS + tq], carry[c * NS + tq + 4]};
      const uint4* tab = reinterpret_cast<const uint4*>(slot) + lane;
      const float2* pw = reinterpret_cast<const float2*>(slot + TAB_WORDS * 128);
      uint32_t T[12], Q[12];
      float2 p16[2];
      // the lane's 8 bytes of block 0 in rows g and g + 8; block j lies at the address with j in bits 5 and 6 exchanged (see cell())
      const uint32_t x0 = smem_u32(xs) + (tq & 1) * 8 + cell<R>(c, g, tq >> 1), x8 = smem_u32(xs) + (tq & 1) * 8 + cell<R>(c, g + 8, tq >> 1);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      bool calm = n > 16;                                              // a short rest costs less token by token
      if (calm) {
        p16[0] = pw[tq]; p16[1] = pw[tq + 4];
        {
          uint32_t P[12];
#pragma unroll
          for (int i = 0; i < 3; ++i) { const uint4 t = tab[i * 32]; P[4 * i] = t.x; P[4 * i + 1] = t.y; P[4 * i + 2] = t.z; P[4 * i + 3] = t.w; }
#pragma unroll
          for (int j = 0; j < R; ++j) {
            uint32_t x[4];
            lds64(x[0], x[2], x0 ^ (j << 5)); lds64(x[1], x[3], x8 ^ (j << 5));
            float e[2][4];
#pragma unroll
            for (int sp = 2; sp >= 0; --sp)
#pragma unroll
              for (int nt = 0; nt < 2; ++nt) {
                if (sp == 2) mma0(e[nt], x, P[(nt * 2) * 3 + sp], P[(nt * 2 + 1) * 3 + sp]);
                else mma(e[nt], x, P[(nt * 2) * 3 + sp], P[(nt * 2 + 1) * 3 + sp]);
              }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
              E[j][0][nt] = make_float2(e[nt][0], e[nt][1]); E[j][1][nt] = make_float2(e[nt][2], e[nt][3]);
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) F[hf][nt] = j == 0 ? E[0][hf][nt] : cfma(p16[nt], F[hf][nt], E[j][hf][nt]);
            }
          }
        }
        if (!STATE_ONLY) {                                             // (under way while the fold waits for its shuffles)
#pragma unroll
          for (int i = 0; i < 3; ++i) { const uint4 t = tab[(3 + i) * 32]; T[4 * i] = t.x; T[4 * i + 1] = t.y; T[4 * i + 2] = t.z; T[4 * i + 3] = t.w; }
#pragma unroll
          for (int i = 0; i < 3; ++i) { const uint4 t = tab[(6 + i) * 32]; Q[4 * i] = t.x; Q[4 * i + 1] = t.y; Q[4 * i + 2] = t.z; Q[4 * i + 3] = t.w; }
        }
        // ---- fold the rows: F[hf][.] becomes the state behind row g (+ 8), then the state in front of it
        float2 S8[2], po[3][2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {                             // a lane without a row that far in front adds nothing
            po[i][nt] = pw[(1 << i) * NS + tq + 4 * nt];
            if (g < (1 << i)) po[i][nt] = make_float2(0.f, 0.f);
          }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) F[hf][nt] = cfma(po[i][nt], shfl_up2(F[hf][nt], 4 << i), F[hf][nt]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float2 pg = pw[(g + 1) * NS + tq + 4 * nt];
          S8[nt] = cfma(pw[8 * NS + tq + 4 * nt], S0[nt], shfl2(F[0][nt], 28 + tq));
          F[0][nt] = cfma(pg, S0[nt], F[0][nt]);
          F[1][nt] = cfma(pg, S8[nt], F[1][nt]);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) calm = calm && fabsf(F[hf][nt].x) < 1e30f && fabsf(F[hf][nt].y) < 1e30f;
        }
        calm = __all_sync(0xffffffffu, calm);
        if (calm) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            if (g == 7) carry[c * NS + tq + 4 * nt] = F[1][nt];
            const float2 u0 = shfl_up2(F[0][nt], 4), u1 = shfl_up2(F[1][nt], 4);
            F[0][nt] = g ? u0 : S0[nt];
            F[1][nt] = g ? u1 : S8[nt];
          }
        }
      }
      __syncwarp();
      {
        int nx = chg + MMA_WARPS;                                      // behind the warp's last channel: its first one of the next tile
        if (c + MMA_WARPS >= CH) {
          const int it = w.item + (int)gridDim.x;
          nx = (w.k + 1 < w.n_tiles || it >= a.items ? w.ch0 : it % (a.D / CH) * CH) + warp;
        }
        fetch(nx);
      }
      if (!calm) {
        // token by token: one mode per lane, four copies
        const int m = lane & 7;
        const float2 p = reinterpret_cast<const float2*>(a.poles)[(long long)chg * NS + m], r = reinterpret_cast<const float2*>(a.residues)[(long long)chg * NS + m];
        const float skip = __bfloat162float(a.Dskip[chg]);
        float2 S = carry[c * NS + m];
#pragma unroll 1
        for (int t = 0; t < n; ++t) {
          bf16* xp = reinterpret_cast<bf16*>(xs + cell<R>(c, t / (BLK * R), (t % (BLK * R)) >> 3)) + (t & 7);
          const float x = __bfloat162float(*xp);
          S = make_float2(fmaf(p.x, S.x, fmaf(-p.y, S.y, x)), fmaf(p.x, S.y, p.y * S.x));
          if (!STATE_ONLY) {
            float o = fmaf(r.x, S.x, -r.y * S.y);
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
            if (lane == 0) *xp = __float2bfloat16_rn(rbf(o) + rbf(x * skip));
          }
        }
        __syncwarp();
        if (lane < 8) { carry[c * NS + m] = S; fin[c * NS + m] = S; }
        if (lane == 0) finm[c] = 0;
        __syncwarp();
        continue;
      }
      const int fq = last ? n >> 4 : -1;                                // the segment's last block, if it ends within this tile
      if (lane == 0 && last) finm[c] = n & 15;
      if (!STATE_ONLY || last) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          uint32_t x[4];
          lds64(x[0], x[2], x0 ^ (j << 5)); lds64(x[1], x[3], x8 ^ (j << 5));
          if (last) {
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
              if (fq == (g + 8 * hf) * R + j) {
                fin[c * NS + tq] = F[hf][0]; fin[c * NS + tq + 4] = F[hf][1];
                xlast[c * 8 + 2 * tq] = x[hf]; xlast[c * 8 + 2 * tq + 1] = x[2 + hf];
              }
          }
          if (!STATE_ONLY) {
            uint32_t sh[4], smd[4], sl[4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) split3(F[hf][nt].x, F[hf][nt].y, sh[nt * 2 + hf], smd[nt * 2 + hf], sl[nt * 2 + hf]);
            // two sums per column group, small products first: what the block itself gives, and what the state gives
            float o[2][4], os[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) { mma0(o[nt], x, T[(nt * 2) * 3 + 2], T[(nt * 2 + 1) * 3 + 2]); mma0(os[nt], sl, Q[(nt * 2) * 3], Q[(nt * 2 + 1) * 3]); }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) { mma(o[nt], x, T[(nt * 2) * 3 + 1], T[(nt * 2 + 1) * 3 + 1]); mma(os[nt], sh, Q[(nt * 2) * 3 + 2], Q[(nt * 2 + 1) * 3 + 2]); }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) { mma(o[nt], x, T[(nt * 2) * 3], T[(nt * 2 + 1) * 3]); mma(os[nt], smd, Q[(nt * 2) * 3 + 1], Q[(nt * 2 + 1) * 3 + 1]); }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma(os[nt], smd, Q[(nt * 2) * 3], Q[(nt * 2 + 1) * 3]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma(os[nt], sh, Q[(nt * 2) * 3 + 1], Q[(nt * 2 + 1) * 3 + 1]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma(os[nt], sh, Q[(nt * 2) * 3], Q[(nt * 2 + 1) * 3]);
            // conv (rounded) + D x (rounded), rounded: tokens 4 tq .. + 3 of rows g and g + 8, back into the place of x
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int e = 0; e < 4; ++e) o[nt][e] += os[nt][e];
            sts64(x0 ^ (j << 5), addbf(pack_bf16(o[0][0], o[0][1]), mulbf(x[0], dsk)), addbf(pack_bf16(o[1][0], o[1][1]), mulbf(x[2], dsk)));
            sts64(x8 ^ (j << 5), addbf(pack_bf16(o[0][2], o[0][3]), mulbf(x[1], dsk)), addbf(pack_bf16(o[1][2], o[1][3]), mulbf(x[3], dsk)));
          }
          if (j + 1 < R) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) F[hf][nt] = cfma(p16[nt], F[hf][nt], E[j][hf][nt]);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&xdone[q & 1]);
    if (last) {
      // ---- the state behind the segment
      float* dst = STATE_ONLY ? a.seg_states + (((long long)w.b * a.nseg + w.seg) * a.D + w.ch0) * NS * 2
                              : (a.state_out && w.seg == a.nseg - 1 ? a.state_out + ((long long)w.b * a.D + w.ch0) * NS * 2 : nullptr);
      if (dst) {
        const int c = warp + (lane >> 3) * MMA_WARPS, m = lane & 7;
        float2 S = n == TILE ? carry[c * NS + m] : fin[c * NS + m];
        const int left = n == TILE ? 0 : finm[c];
        const float2 p = reinterpret_cast<const float2*>(a.poles)[(long long)(w.ch0 + c) * NS + m];
        for (int t = 0; t < left; ++t) {
          const float x = __bfloat162float(reinterpret_cast<const bf16*>(xlast + c * 8)[t]);
          S = make_float2(fmaf(p.x, S.x, fmaf(-p.y, S.y, x)), fmaf(p.x, S.y, p.y * S.x));
        }
        reinterpret_cast<float2*>(dst)[c * NS + m] = S;
      }
      __syncwarp();
    }
    w.next(a, TILE);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace evo_hytc
