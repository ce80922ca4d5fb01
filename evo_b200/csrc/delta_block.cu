// Gated delta rule over prompts by blocks of 64 tokens on the tensor cores (evo_gated_delta_fwd, bf16 activations; matrix_state.cu holds the entry point and the
// token-by-token form).  With the block's decays g, G_i = g_1 .. g_i, Gam_ij = g_{j+1} .. g_i, and the state S in front of it:
//   u_i = beta_i (v_i - G_i S^T k_i - sum_{j<i} Gam_ij (k_i . k_j) u_j)      o_i = G_i S^T q_i + sum_{j<=i} Gam_ij (q_i . k_j) u_j      S' = G_64 S + sum_j Gam_64,j k_j u_j^T
// i.e. U = T diag(beta) (V - diag(G) K S) with T = (1 + A)^-1, A_ij = beta_i Gam_ij (k_i . k_j) below the diagonal; O = diag(G) Q S + P U.
//
// delta_prepare_kernel, one CTA per (block, head, sequence), all in parallel: what does not depend on the state.  k . k and q . k as bf16 products (exact) with fp32
//   sums, norms and gates in fp32, sums of log decays in 64 bits (their differences enter as two floats), T in fp32 by halves: two triangles of 32 by forward
//   substitution (one column per thread), the square between them by products.
//   T diag(beta) and P go to the workspace as three bf16 parts (24 bits), in the order in which the next kernel's lanes read them.
// delta_scan_kernel, one warp per 16 value channels, blocks one after another.  Everything is held transposed (value channels = rows of the mma tiles): the sums of
//   one product are then, lane by lane, the first operand of the next, so the 16 x dk piece of the state stays in the warp's registers and warps exchange nothing:
//     W^T = V^T - S^T K^T (x G rk);  Q^T-part = S^T Q^T;  U^T = W^T T^T;  O^T += U^T P^T;  S'^T = G S^T + (U Gam rk)^T K
//   S, W, U are fp32 and enter as three bf16 parts; K and Q are bf16 as they stand (their norms scale the sums); T, P have three parts and meet W, U in the six products
//   down to 2^-16 of the leading one.  K, Q, V, T, P of the next block arrive by bulk copies while one is in work.
// delta_norm_kernel: head norm, weight and SiLU gate of the fp32 read-outs.
// Measured (B200): 4 x 4096 tokens, 16 heads of 128 x 128: 590 us (token by token 2774), of which the scan 395, bound by the tensor pipe (816 mma of 8.7 cycles per block and
// warp, one warp per scheduler: 7.1 k of 10.4 k cycles) and the splits between its products; 1 x 777 tokens, 32 heads: 110 us (516).
// A block in which W or U is not finite goes token by token: a product with a structural zero would carry a NaN to earlier tokens.
#include "waits.cuh"
#include "mma_sync.cuh"
#include "../../include/evo_b200.h"
#include <algorithm>
#include <math.h>

using namespace evo;

namespace evo {
size_t delta_block_workspace(const evo_gated_delta_params* p);                                   // 0: not taken
int delta_block_fwd(const evo_gated_delta_params* p, void* ws, size_t bytes, cudaStream_t st);    // called by matrix_state.cu
}

namespace {

constexpr int BT = 64;                                  // tokens of a block
constexpr int TILES = 20;                               // 16 x 8 tiles of a lower triangle: k-tile kt with n-tiles 2 kt .. 7
constexpr int PART_BYTES = 256;                         // one part of one tile: 32 lanes x 2 words
constexpr int TRI_BYTES = TILES * 3 * PART_BYTES;       // T or P of a block
enum { V_GK = 0, V_GQ, V_CK, V_RK, V_RQ, V_BETA, V_G, V_ROWS };       // G rk | G rq | Gam_64 rk | rk | rq | beta | g
constexpr int VEC_BYTES = V_ROWS * BT * 4 + 256;        // + the block's decay G_64
constexpr int BLOCK_BYTES = 2 * TRI_BYTES + VEC_BYTES;  // of one (block, head, sequence)
__host__ __device__ constexpr int tile_index(int kt, int nt) { return kt * (9 - kt) + nt - 2 * kt; }

struct Args {
  const bf16* k; const bf16* q; const bf16* v; int64_t ld;
  const bf16* b; const bf16* a; int64_t ldz;
  const bf16* A_log; const bf16* dt_bias;
  float unit_eps, q_scale;
  uint8_t* blocks;                                      // (sequence, head, block of the slab)
  float* state; int zero_start, store_state;
  float* y;                                             // (rows, H * dv) fp32 read-outs
  int B; int64_t L; int H, G, dv;
  int64_t first; int n_blocks;                          // the slab: its first block and its length
  unsigned int* failed;                                 // a wait of this call ran out: later slabs and the states behind them are not computed
  WaitLimit waits;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool on) {       // zero-filled when off
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
// global -> shared memory, bytes and both addresses multiples of 16
__device__ __forceinline__ void bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mma_np(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {       // free to be scheduled
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float softplus_f(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }

// ------------------------------------------------------------------------------------------------ what does not depend on the state
__host__ __device__ constexpr int prepare_rows_bytes(int dk) { return 2 * BT * (2 * dk + 16) > 2 * BT * (BT + 4) * 4 ? 2 * BT * (2 * dk + 16) : 2 * BT * (BT + 4) * 4; }
template <int DK>
__global__ void __launch_bounds__(128) delta_prepare_kernel(const Args p) {
  constexpr int PITCH = 2 * DK + 16, AP = BT + 4;            // bytes of a key row; floats of a row of A (16-byte pieces)
  extern __shared__ __align__(16) uint8_t sm[];
  uint8_t* ks = sm;
  uint8_t* qs = ks + BT * PITCH;
  float* As = reinterpret_cast<float*>(sm);                  // [BT][AP] A, then T, in the place of the keys and queries once they are multiplied
  float* Ps = As + BT * AP;                                  // [BT][AP]
  float* rk = reinterpret_cast<float*>(sm + prepare_rows_bytes(DK));
  float* rq = rk + BT;
  float* beta = rq + BT;
  float* lh = beta + BT;                                     // running log decay, high and low float
  float* ll = lh + BT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z, g = h / (p.H / p.G);
  const int64_t t0 = (p.first + blk) * BT, row0 = (int64_t)b * p.L + t0;
  const int nt = (int)min((int64_t)BT, p.L - t0);
  if (p.first == 0 && (blk | h | b | tid) == 0) *p.failed = 0u;
  for (int e = tid; e < BT * (DK / 8); e += 128) {
    const int r = e / (DK / 8), c = e % (DK / 8);
    const bool on = r < nt;
    const int64_t off = (row0 + (on ? r : 0)) * p.ld + (int64_t)g * DK + c * 8;
    cp16(smem_u32(ks + r * PITCH + c * 16), p.k + off, on);
    cp16(smem_u32(qs + r * PITCH + c * 16), p.q + off, on);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (warp == 0) {
    // gates; the running sum of the log decays in 64 bits, two tokens per lane
    const float A = expf(__bfloat162float(p.A_log[h])), dtb = __bfloat162float(p.dt_bias[h]);
    double l[2];
    float gl[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = 2 * lane + u;
      const bool on = t < nt;
      const float av = on ? __bfloat162float(p.a[(row0 + t) * p.ldz + h]) : 0.f, bv = on ? __bfloat162float(p.b[(row0 + t) * p.ldz + h]) : 0.f;
      gl[u] = on ? -A * softplus_f(av + dtb) : 0.f;
      if (gl[u] < -200.f) gl[u] = -200.f;                                // e^-200 is zero already; the sums stay finite (and a NaN stays one)
      l[u] = gl[u];
      beta[t] = on ? 1.f / (1.f + expf(-bv)) : 0.f;
    }
    double run = l[0] + l[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double u = __shfl_up_sync(0xffffffffu, run, o); if (lane >= o) run += u; }
    const double before = run - (l[0] + l[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double v = u ? run : before + l[0];
      const float hi = (float)v;
      lh[2 * lane + u] = hi; ll[2 * lane + u] = (float)(v - (double)hi);
    }
    float* vec = reinterpret_cast<float*>(p.blocks + (((int64_t)b * p.H + h) * p.n_blocks + blk) * BLOCK_BYTES + 2 * TRI_BYTES);
#pragma unroll
    for (int u = 0; u < 2; ++u) vec[V_G * BT + 2 * lane + u] = expf(gl[u]);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // ---- norms: one warp per 16 tokens, two lanes per token
  {
    const int t = warp * 16 + (lane >> 1);
    const uint8_t* kr = ks + t * PITCH + (lane & 1) * DK;
    const uint8_t* qr = qs + t * PITCH + (lane & 1) * DK;
    float sk = 0.f, sq = 0.f;
#pragma unroll 4
    for (int c = 0; c < DK / 16; ++c) {
      const uint4 x = *reinterpret_cast<const uint4*>(kr + c * 16), y = *reinterpret_cast<const uint4*>(qr + c * 16);
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sk = fmaf(bf_lo(xw[i]), bf_lo(xw[i]), fmaf(bf_hi(xw[i]), bf_hi(xw[i]), sk));
        sq = fmaf(bf_lo(yw[i]), bf_lo(yw[i]), fmaf(bf_hi(yw[i]), bf_hi(yw[i]), sq));
      }
    }
    sk += __shfl_xor_sync(0xffffffffu, sk, 1); sq += __shfl_xor_sync(0xffffffffu, sq, 1);
    if (!(lane & 1)) { rk[t] = 1.0f / sqrtf(sk + p.unit_eps); rq[t] = p.q_scale / sqrtf(sq + p.unit_eps); }
  }
  __syncthreads();
  // ---- k . k and q . k: warp = 16 rows i, tiles of 8 columns j up to the diagonal
  {
    const int gq = lane >> 2, tq = lane & 3, i0 = warp * 16;
    float kk[8][4], qk[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) kk[n][e] = qk[n][e] = 0.f;
    const int arow = i0 + (lane & 15), acol = (lane >> 4) * 16;
    const int brow = (lane & 7) + ((lane >> 4) << 3), bcol = ((lane >> 3) & 1) * 16;
#pragma unroll 2
    for (int kt = 0; kt < DK / 16; ++kt) {
      uint32_t ak[4], aq[4];
      ldmatrix_x4(ak, ks + arow * PITCH + kt * 32 + acol);
      ldmatrix_x4(aq, qs + arow * PITCH + kt * 32 + acol);
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) {
        if (n2 <= warp) {
          uint32_t bk[4];
          ldmatrix_x4(bk, ks + (n2 * 16 + brow) * PITCH + kt * 32 + bcol);
          mma_np(kk[2 * n2], ak, bk[0], bk[1]); mma_np(kk[2 * n2 + 1], ak, bk[2], bk[3]);
          mma_np(qk[2 * n2], aq, bk[0], bk[1]); mma_np(qk[2 * n2 + 1], aq, bk[2], bk[3]);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      if (n / 2 > warp) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + gq + (e >> 1) * 8, j = n * 8 + 2 * tq + (e & 1);
        if (j <= i) {
          const float gam = expf((lh[i] - lh[j]) + (ll[i] - ll[j])) * rk[j];
          Ps[i * AP + j] = gam * rq[i] * qk[n][e];
          if (j < i) As[i * AP + j] = beta[i] * (gam * rk[i] * kk[n][e]);
        }
      }
    }
  }
  __syncthreads();
  // ---- T = (1 + A)^-1 in fp32: the two diagonal blocks of 32 by forward substitution, one column per thread; then T21 = -T22 (A21 T11), with the
  // inner product in the unused upper right block (one block of 64 would be 2016 multiply-adds in a row, an instruction stream no cache holds)
  uint8_t* out = p.blocks + (((int64_t)b * p.H + h) * p.n_blocks + blk) * BLOCK_BYTES;
  float* vec = reinterpret_cast<float*>(out + 2 * TRI_BYTES);
  if (tid < BT) {
    const int d = tid & 32, c = tid & 31;
    const float* Ad = As + d * AP + d;
    float T[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < i; k += 4) {
        const float4 r = *reinterpret_cast<const float4*>(Ad + i * AP + k);          // (what lies on and above the diagonal is not used)
        const float rv[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) if (k + u < i) s[u] = fmaf(rv[u], T[k + u], s[u]);
      }
      T[i] = i < c ? 0.f : (i == c ? 1.f : -((s[0] + s[1]) + (s[2] + s[3])));
    }
    __syncwarp();                                                       // a diagonal block is read and replaced by one warp
#pragma unroll
    for (int i = 0; i < 32; ++i) As[(d + i) * AP + d + c] = T[i];
  } else {
    const int t = tid - BT;
    const float G = expf(lh[t] + ll[t]);
    vec[V_GK * BT + t] = G * rk[t];
    vec[V_GQ * BT + t] = G * rq[t];
    vec[V_CK * BT + t] = expf((lh[BT - 1] - lh[t]) + (ll[BT - 1] - ll[t])) * rk[t];
    vec[V_RK * BT + t] = rk[t]; vec[V_RQ * BT + t] = rq[t]; vec[V_BETA * BT + t] = beta[t];
    if (t == BT - 1) vec[V_ROWS * BT] = G;
  }
  __syncthreads();
  {
    const int r = tid >> 2, c = (tid & 3) * 8;
    // acc[0..7] = sum_k left[k] * right[k][c ..]
    auto row_times = [&](const float* left, const float* right, float (&acc)[8]) {
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] = 0.f;
#pragma unroll 4
      for (int k = 0; k < 32; ++k) {
        const float l = left[k];
        const float4 x = *reinterpret_cast<const float4*>(right + k * AP + c), y = *reinterpret_cast<const float4*>(right + k * AP + c + 4);
        acc[0] = fmaf(l, x.x, acc[0]); acc[1] = fmaf(l, x.y, acc[1]); acc[2] = fmaf(l, x.z, acc[2]); acc[3] = fmaf(l, x.w, acc[3]);
        acc[4] = fmaf(l, y.x, acc[4]); acc[5] = fmaf(l, y.y, acc[5]); acc[6] = fmaf(l, y.z, acc[6]); acc[7] = fmaf(l, y.w, acc[7]);
      }
    };
    float acc[8];
    row_times(As + (32 + r) * AP, As, acc);
#pragma unroll
    for (int u = 0; u < 8; ++u) As[r * AP + 32 + c + u] = acc[u];
    __syncthreads();
    row_times(As + (32 + r) * AP + 32, As + 32, acc);
    // (A21 was read before the barrier)
#pragma unroll
    for (int u = 0; u < 8; ++u) As[(32 + r) * AP + c + u] = -acc[u];
  }
  __syncthreads();
  // ---- as second operands: column n = token i, k = token j; lane (g, tq) of tile (kt, nt): i = 8 nt + g, j = 16 kt + 2 tq + {0, 1} | + 8
  for (int e = warp; e < 2 * TILES; e += 4) {
    const float* src = e < TILES ? As : Ps;
    int kt = 0, x = e % TILES;
    while (x >= 8 - 2 * kt) { x -= 8 - 2 * kt; ++kt; }
    const int i = 8 * (x + 2 * kt) + (lane >> 2), j = 16 * kt + 2 * (lane & 3);
    uint32_t w[2][3];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int jj = j + 8 * u;
      const float2 x = *reinterpret_cast<const float2*>(src + i * AP + jj);
      const float f0 = e < TILES ? beta[jj] : 1.f, f1 = e < TILES ? beta[jj + 1] : 1.f;
      split3(jj <= i ? x.x * f0 : 0.f, jj + 1 <= i ? x.y * f1 : 0.f, w[u][0], w[u][1], w[u][2]);
    }
    uint2* dst = reinterpret_cast<uint2*>(out + (e < TILES ? 0 : TRI_BYTES) + (e % TILES) * 3 * PART_BYTES) + lane;
#pragma unroll
    for (int s = 0; s < 3; ++s) dst[s * 32] = make_uint2(w[0][s], w[1][s]);
  }
}

// ------------------------------------------------------------------------------------------------ the recurrence
template <int DK>
__global__ void __launch_bounds__(256, 1) delta_scan_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmV, const Args p) {
  constexpr int KT = DK / 16, BOX = BT * 128, ROWS_BYTES = DK / 64 * BOX;      // keys and queries: boxes of 64 columns, 16-byte pieces of a row swizzled by row & 7
  extern __shared__ __align__(16) uint8_t sm_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t arrived[2];
  const int nw = blockDim.x >> 5, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int vpitch = nw * 32, stage_bytes = 2 * ROWS_BYTES + BT * vpitch + BLOCK_BYTES;
  const int h = blockIdx.x, b = blockIdx.y, g = h / (p.H / p.G), dv = p.dv;
  const int c0 = blockIdx.z * nw * 16, cw = c0 + warp * 16;            // the CTA's and the warp's first value channel
  const int64_t rowb = (int64_t)b * p.L + p.first * BT, left = p.L - p.first * BT;       // the slab's first row; tokens from there
  const uint8_t* blocks = p.blocks + ((int64_t)b * p.H + h) * p.n_blocks * (int64_t)BLOCK_BYTES;

  // a block's rows of K, Q, V (rows behind the last token arrive as zeros) and its T, P and vectors: one lane
  auto fetch = [&](int blk) {
    uint8_t* st = sm + (blk & 1) * stage_bytes;
    uint64_t* bar = &arrived[blk & 1];
    const int t0 = (int)(p.first + blk) * BT;
    mbar_arrive_expect_tx(bar, stage_bytes);
#pragma unroll
    for (int i = 0; i < DK / 64; ++i) {
      tma_load_3d(st + i * BOX, &tmK, bar, g * DK + i * 64, t0, b);
      tma_load_3d(st + ROWS_BYTES + i * BOX, &tmQ, bar, g * DK + i * 64, t0, b);
    }
    tma_load_3d(st + 2 * ROWS_BYTES, &tmV, bar, h * dv + c0, t0, b);
    bulk(st + 2 * ROWS_BYTES + BT * vpitch, blocks + (int64_t)blk * BLOCK_BYTES, BLOCK_BYTES, bar);
  };
  if (tid == 0) { mbar_init(&arrived[0], 1); mbar_init(&arrived[1], 1); fence_barrier_init(); }
  if (__syncthreads_or(p.first > 0 && tid == 0 && *(volatile unsigned int*)p.failed)) return;

  // ---- S^T: rows = value channels cw + gq (+ 8), columns = state rows: S[n][..] covers state rows 8 n + 2 tq, + 1
  float S[2 * KT][4];
  float* Sg = p.state + ((int64_t)b * p.H + h) * DK * (int64_t)dv;
  const bool live = cw < dv;                                            // (dv is a multiple of 16)
#pragma unroll
  for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[n][e] = (p.zero_start || !live) ? 0.f : Sg[(int64_t)(8 * n + 2 * tq + (e & 1)) * dv + cw + gq + (e >> 1) * 8];

  if (tid == 0) fetch(0);
  for (int blk = 0; blk < p.n_blocks; ++blk) {
    if (tid == 0 && blk + 1 < p.n_blocks) fetch(blk + 1);
    const uint8_t* ks = sm + (blk & 1) * stage_bytes;
    const bool here = wait_or_give_up(&arrived[blk & 1], (blk >> 1) & 1, p.waits);
    if (__syncthreads_or(!here)) {
      // no state is kept; the copies under way land before the CTA ends
      if (tid == 0) {
        *p.failed = 1u;
        wait_to_end(&arrived[blk & 1], (blk >> 1) & 1, p.waits);
        if (blk + 1 < p.n_blocks) wait_to_end(&arrived[(blk + 1) & 1], ((blk + 1) >> 1) & 1, p.waits);
      }
      return;
    }
    const uint8_t* qs = ks + ROWS_BYTES;
    const uint8_t* vs = qs + ROWS_BYTES;
    const uint8_t* tri = vs + BT * vpitch;
    const float* vec = reinterpret_cast<const float*>(tri + 2 * TRI_BYTES);
    const int nt = (int)min((int64_t)BT, left - (int64_t)blk * BT);
    float* yr = p.y + (rowb + (int64_t)blk * BT) * p.H * dv + (int64_t)h * dv + cw + gq;
    if (live) {
      float W[8][4], O[8][4];                                           // columns = tokens 8 n + 2 tq, + 1
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) W[n][e] = O[n][e] = 0.f;
      const uint32_t brow = ((lane & 7) + ((lane >> 4) << 3)) * 128, piece = (lane >> 3) & 1, turn = lane & 7;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        const uint32_t at = (kt >> 2) * BOX + brow + (((2 * (kt & 3) + piece) ^ turn) << 4), kb = smem_u32(ks) + at, qb = smem_u32(qs) + at;
        uint32_t a[3][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          split3(S[2 * kt + u][0], S[2 * kt + u][1], a[0][2 * u], a[1][2 * u], a[2][2 * u]);
          split3(S[2 * kt + u][2], S[2 * kt + u][3], a[0][2 * u + 1], a[1][2 * u + 1], a[2][2 * u + 1]);
        }
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
          uint32_t bk[4], bq[4];
          ldmatrix_x4_at(bk, kb + n2 * 16 * 128);
          ldmatrix_x4_at(bq, qb + n2 * 16 * 128);
#pragma unroll
          for (int s = 2; s >= 0; --s) {
            mma_np(W[2 * n2], a[s], bk[0], bk[1]); mma_np(W[2 * n2 + 1], a[s], bk[2], bk[3]);
            mma_np(O[2 * n2], a[s], bq[0], bq[1]); mma_np(O[2 * n2 + 1], a[s], bq[2], bq[3]);
          }
        }
      }
      // ---- W = V - G rk (K S); O = G rq (Q S)
      float wrong = 0.f;
      {
        const uint32_t vb = smem_u32(vs) + ((lane & 7) + ((lane >> 4) << 3)) * vpitch + warp * 32 + ((lane >> 3) & 1) * 16;
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
          uint32_t v[4];                                                // (tokens 0-7, channels 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15), turned
          ldmatrix_x4_trans_at(v, vb + n2 * 16 * vpitch);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int n = 2 * n2 + u;
            const float2 gk = *reinterpret_cast<const float2*>(vec + V_GK * BT + 8 * n + 2 * tq), gqv = *reinterpret_cast<const float2*>(vec + V_GQ * BT + 8 * n + 2 * tq);
            W[n][0] = fmaf(-gk.x, W[n][0], bf_lo(v[2 * u])); W[n][1] = fmaf(-gk.y, W[n][1], bf_hi(v[2 * u]));
            W[n][2] = fmaf(-gk.x, W[n][2], bf_lo(v[2 * u + 1])); W[n][3] = fmaf(-gk.y, W[n][3], bf_hi(v[2 * u + 1]));
            O[n][0] *= gqv.x; O[n][1] *= gqv.y; O[n][2] *= gqv.x; O[n][3] *= gqv.y;
#pragma unroll
            for (int e = 0; e < 4; ++e) wrong = fmaf(0.f, W[n][e], wrong);
          }
        }
      }
      // second operands of a triangle: the three parts of tile (kt, n)
      auto tri_mul = [&](const uint8_t* base, const float (&X)[8][4], float (&Y)[8][4]) {
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
          uint32_t a[3][4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            split3(X[2 * kt + u][0], X[2 * kt + u][1], a[0][2 * u], a[1][2 * u], a[2][2 * u]);
            split3(X[2 * kt + u][2], X[2 * kt + u][3], a[0][2 * u + 1], a[1][2 * u + 1], a[2][2 * u + 1]);
          }
#pragma unroll
          for (int n0 = 2 * kt; n0 < 8; n0 += 4) {                       // four sums at a time: a sum's next mma is four later (23 cycles of latency, 8.7 of issue)
            uint2 t[4][3];
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (n0 + c < 8)
#pragma unroll
                for (int s = 0; s < 3; ++s) t[c][s] = (reinterpret_cast<const uint2*>(base + tile_index(kt, n0 + c) * 3 * PART_BYTES) + lane)[s * 32];
            const int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};       // small products first
#pragma unroll
            for (int m = 0; m < 6; ++m)
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (n0 + c < 8) mma_np(Y[n0 + c], a[pa[m]], t[c][pb[m]].x, t[c][pb[m]].y);
          }
        }
      };
      float U[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) U[n][e] = 0.f;
      tri_mul(tri, W, U);
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) wrong = fmaf(0.f, U[n][e], wrong);
      if (__all_sync(0xffffffffu, wrong == 0.f)) {
        tri_mul(tri + TRI_BYTES, U, O);
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = 8 * n + 2 * tq + (e & 1);
            if (t < nt) yr[(int64_t)t * p.H * dv + (e >> 1) * 8] = O[n][e];
          }
        // ---- S = G_64 S + (Gam rk U)^T K
        const float G = vec[V_ROWS * BT];
#pragma unroll
        for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[n][e] *= G;
        const uint32_t kt_b = smem_u32(ks) + ((lane & 7) + (((lane >> 3) & 1) << 3)) * 128;
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
          uint32_t a[3][4];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int n = 2 * kt + u;
            const float2 ck = *reinterpret_cast<const float2*>(vec + V_CK * BT + 8 * n + 2 * tq);
            split3(U[n][0] * ck.x, U[n][1] * ck.y, a[0][2 * u], a[1][2 * u], a[2][2 * u]);
            split3(U[n][2] * ck.x, U[n][3] * ck.y, a[0][2 * u + 1], a[1][2 * u + 1], a[2][2 * u + 1]);
          }
#pragma unroll
          for (int n2 = 0; n2 < KT; n2 += 2) {
            uint32_t bk[8];
            ldmatrix_x4_trans_at(bk, kt_b + kt * 16 * 128 + (n2 >> 2) * BOX + (((2 * (n2 & 3) + (lane >> 4)) ^ turn) << 4));
            ldmatrix_x4_trans_at(bk + 4, kt_b + kt * 16 * 128 + (n2 >> 2) * BOX + (((2 * (n2 & 3) + 2 + (lane >> 4)) ^ turn) << 4));
#pragma unroll
            for (int s = 2; s >= 0; --s)
#pragma unroll
              for (int c = 0; c < 4; ++c) mma_np(S[2 * n2 + c], a[s], bk[2 * c], bk[2 * c + 1]);
          }
        }
      } else {
        // token by token, as the recurrence is defined; lanes of a quad share the rows of the state
        for (int t = 0; t < nt; ++t) {
          const float dec = vec[V_G * BT + t], be = vec[V_BETA * BT + t], nk = vec[V_RK * BT + t], nq = vec[V_RQ * BT + t];
          float pk[2] = {0.f, 0.f}, po[2] = {0.f, 0.f}, kq = 0.f;
#pragma unroll
          for (int n = 0; n < 2 * KT; ++n) {
            const uint32_t kw = *reinterpret_cast<const uint32_t*>(ks + (n >> 3) * BOX + t * 128 + (((n & 7) ^ (t & 7)) << 4) + 4 * tq), qw = *reinterpret_cast<const uint32_t*>(qs + (n >> 3) * BOX + t * 128 + (((n & 7) ^ (t & 7)) << 4) + 4 * tq);
            const float k0 = bf_lo(kw) * nk, k1 = bf_hi(kw) * nk, q0 = bf_lo(qw) * nq, q1 = bf_hi(qw) * nq;
            kq = fmaf(k1, q1, fmaf(k0, q0, kq));
#pragma unroll
            for (int e = 0; e < 4; ++e) S[n][e] *= dec;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              pk[u] = fmaf(S[n][2 * u + 1], k1, fmaf(S[n][2 * u], k0, pk[u]));
              po[u] = fmaf(S[n][2 * u + 1], q1, fmaf(S[n][2 * u], q0, po[u]));
            }
          }
          kq = quad_sum(kq);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            pk[u] = be * (__bfloat162float(*reinterpret_cast<const bf16*>(vs + t * vpitch + (warp * 16 + gq + 8 * u) * 2)) - quad_sum(pk[u]));
            po[u] = fmaf(pk[u], kq, quad_sum(po[u]));
            if (tq == 0) yr[(int64_t)t * p.H * dv + 8 * u] = po[u];
          }
#pragma unroll
          for (int n = 0; n < 2 * KT; ++n) {
            const uint32_t kw = *reinterpret_cast<const uint32_t*>(ks + (n >> 3) * BOX + t * 128 + (((n & 7) ^ (t & 7)) << 4) + 4 * tq);
            const float k0 = bf_lo(kw) * nk, k1 = bf_hi(kw) * nk;
#pragma unroll
            for (int u = 0; u < 2; ++u) { S[n][2 * u] = fmaf(k0, pk[u], S[n][2 * u]); S[n][2 * u + 1] = fmaf(k1, pk[u], S[n][2 * u + 1]); }
          }
        }
      }
    }
    __syncthreads();                                                    // the stage may be filled again
  }
  if (p.store_state && live) {
#pragma unroll
    for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) Sg[(int64_t)(8 * n + 2 * tq + (e & 1)) * dv + cw + gq + (e >> 1) * 8] = S[n][e];
  }
}

// head norm, weight and SiLU gate of the read-outs of (row, head): one warp, four channels per lane and step
__global__ void __launch_bounds__(256) delta_norm_kernel(const float* __restrict__ y, const bf16* __restrict__ gate, int64_t ldg, const bf16* __restrict__ w, bf16* __restrict__ out, int64_t ldo,
                                                         int64_t rows, int H, int dv, float eps) {
  const int64_t wid = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= rows * H) return;
  const int64_t row = wid / H;
  const int h = (int)(wid % H);
  const float4* r = reinterpret_cast<const float4*>(y + wid * dv);
  float ss = 0.f;
  for (int c = lane; c < dv / 4; c += 32) { const float4 o = r[c]; ss = fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, fmaf(o.w, o.w, ss)))); }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float rstd = 1.0f / sqrtf(ss / (float)dv + eps);
  const bf16* gr = gate + row * ldg + (int64_t)h * dv;
  bf16* orow = out + row * ldo + (int64_t)h * dv;
  const auto one = [&](float o, bf16 gb, bf16 wb) { const float gv = __bfloat162float(gb); return o * rstd * __bfloat162float(wb) * (gv / (1.f + expf(-gv))); };
  for (int c = lane; c < dv / 4; c += 32) {
    const float4 o = r[c];
    // gate, weight and output rows need not be aligned: single elements
    orow[4 * c] = __float2bfloat16_rn(one(o.x, gr[4 * c], w[4 * c]));
    orow[4 * c + 1] = __float2bfloat16_rn(one(o.y, gr[4 * c + 1], w[4 * c + 1]));
    orow[4 * c + 2] = __float2bfloat16_rn(one(o.z, gr[4 * c + 2], w[4 * c + 2]));
    orow[4 * c + 3] = __float2bfloat16_rn(one(o.w, gr[4 * c + 3], w[4 * c + 3]));
  }
  if (h == H - 1)
    for (int64_t c = (int64_t)H * dv + lane; c < ldo; c += 32) out[row * ldo + c] = __float2bfloat16_rn(0.f);
}
// the same for heads of 32 N channels and rows that start on four elements: eight lanes per (row, head), everything in registers between the two passes
template <int N>
__global__ void __launch_bounds__(256) delta_norm4_kernel(const float* __restrict__ y, const bf16* __restrict__ gate, int64_t ldg, const bf16* __restrict__ w, bf16* __restrict__ out, int64_t ldo,
                                                          int64_t rows, int H, int dv, float eps) {
  const int64_t id = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  const int sub = threadIdx.x & 7;
  const bool on = id < rows * H;
  const int64_t row = on ? id / H : 0;
  const int h = on ? (int)(id - row * H) : 0;
  const float4* r = reinterpret_cast<const float4*>(y + (on ? id : 0) * (32 * N)) + sub;
  const uint2* gr = reinterpret_cast<const uint2*>(gate + row * ldg + (int64_t)h * (32 * N)) + sub;
  const uint2* wr = reinterpret_cast<const uint2*>(w) + sub;
  float4 o[N];
  uint2 gv[N];
#pragma unroll
  for (int i = 0; i < N; ++i) { o[i] = r[8 * i]; gv[i] = gr[8 * i]; }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) ss = fmaf(o[i].x, o[i].x, fmaf(o[i].y, o[i].y, fmaf(o[i].z, o[i].z, fmaf(o[i].w, o[i].w, ss))));
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  const float rstd = 1.0f / sqrtf(ss / (float)(32 * N) + eps);
  if (!on) return;
  uint2* orow = reinterpret_cast<uint2*>(out + row * ldo + (int64_t)h * (32 * N)) + sub;
  const auto one = [&](float v, float g, float wv) { return v * rstd * wv * (g / (1.f + expf(-g))); };
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint2 wv = wr[8 * i];
    orow[8 * i] = make_uint2(pack_bf16(one(o[i].x, bf_lo(gv[i].x), bf_lo(wv.x)), one(o[i].y, bf_hi(gv[i].x), bf_hi(wv.x))),
                             pack_bf16(one(o[i].z, bf_lo(gv[i].y), bf_lo(wv.y)), one(o[i].w, bf_hi(gv[i].y), bf_hi(wv.y))));
  }
  if (h == H - 1)
    for (int64_t c = (int64_t)H * (32 * N) + sub; c < ldo; c += 8) out[row * ldo + c] = __float2bfloat16_rn(0.f);
}

// Blocks whose T and P are in memory at a time: at most 256 MB of them, or one block of every (head, sequence) pair where that is more (32 KB each, above 8192 pairs).
// A longer call runs slab after slab, the state carried in between.
constexpr int64_t SLAB_BYTES = 256ll << 20;

// From how many tokens on the blocks are faster.  Three launches and a 64-token block take 25 us (8 pairs of head and sequence) to 300 (2048 pairs of 128 x 128) whether the block is
// full or not; token by token a call takes 0.5 to 1 us per token while the pairs fit the SMs, in proportion to their number beyond.  Measured (us, token by token / blocks):
//   heads of 64 x 64, 32 pairs: 32 tokens 23 / 26, 40 tokens 27 / 26, 48 tokens 31 / 26;  128 x 128, 128 pairs: 32 / 36, 39 / 37, 45 / 37;  64 x 128, 128 pairs: 25 / 32, 31 / 33, 33 / 33
//   512 pairs, where token by token has more than a wave: 64 x 64: 32 tokens 52 / 51;  128 x 128: 125 / 86
//   few value channels, whose token-by-token CTAs are nearly empty: 128 x 16, 32 pairs: 32 tokens 50 / 29;  but 1024 pairs: 48 tokens 97 / 120
int64_t block_tokens(const evo_gated_delta_params* p) {
  const int64_t pairs = (int64_t)p->B * p->H;
  if (p->dv >= 48) return pairs >= 512 ? 32 : 48;
  if (pairs <= 128) return 32;
  return p->dv < 32 && pairs > 512 ? 128 : 48;
}

// Taken for bf16 heads of 64 or 128 key channels and a multiple of 16 value channels, rows that start on 16 bytes, and enough tokens.
// (The workspace query comes here with shapes that the call has not looked over: an empty batch has no blocks to count.)
bool taken(const evo_gated_delta_params* p) {
  return p->B > 0 && p->H > 0 && p->dv > 0 && p->dtype == 0 && (p->dk == 64 || p->dk == 128) && p->dv % 16 == 0 && p->L >= block_tokens(p) && p->ld % 8 == 0 && p->H <= 65535 && p->B <= 65535 &&
         (((uintptr_t)p->q | (uintptr_t)p->k | (uintptr_t)p->v) & 15) == 0;
}
struct Sizes {
  int64_t blocks, slab; size_t y, tri, state;
  size_t total() const { return y + tri + state + 2 * 256; }         // with the call's `failed` word, and the start moved up to a multiple of 256
};
Sizes sizes(const evo_gated_delta_params* p) {
  Sizes s;
  s.blocks = (p->L + BT - 1) / BT;
  s.slab = std::max<int64_t>(1, std::min<int64_t>(s.blocks, SLAB_BYTES / ((int64_t)BLOCK_BYTES * p->B * p->H)));
  const auto up = [](size_t n) { return (n + 255) / 256 * 256; };
  s.y = up(sizeof(float) * (size_t)p->B * p->L * p->H * p->dv);
  s.tri = up((size_t)BLOCK_BYTES * s.slab * p->B * p->H);
  s.state = p->state || s.slab == s.blocks ? 0 : up(sizeof(float) * (size_t)p->B * p->H * p->dk * p->dv);
  return s;
}

constexpr int scan_smem_bytes(int dk, int warps) { return 1024 + 2 * (2 * BT * dk * 2 + BT * warps * 32 + BLOCK_BYTES); }
static_assert(scan_smem_bytes(128, 8) <= 227 * 1024, "two stages of eight warps");

template <int DK>
int run(const evo_gated_delta_params* p, const Sizes& s, uint8_t* ws, cudaStream_t st) {
  Args a = {};
  if (const int rc = wait_limit(&a.waits)) return rc;
  a.failed = (unsigned int*)(ws + s.y + s.tri + s.state);
  a.k = (const bf16*)p->k; a.q = (const bf16*)p->q; a.v = (const bf16*)p->v; a.ld = p->ld;
  a.b = (const bf16*)p->b; a.a = (const bf16*)p->a; a.ldz = p->ldz;
  a.A_log = (const bf16*)p->A_log; a.dt_bias = (const bf16*)p->dt_bias;
  a.unit_eps = p->unit_eps; a.q_scale = p->q_scale;
  a.y = (float*)ws; a.blocks = ws + s.y;
  a.state = p->state ? p->state : (s.state ? (float*)(ws + s.y + s.tri) : (float*)ws);      // (never read nor written in the last case)
  a.B = p->B; a.L = p->L; a.H = p->H; a.G = p->G; a.dv = p->dv;
  // warps spread over the schedulers: two (32 channels) to eight per CTA, as few as fill the chip (592 schedulers)
  const int64_t warps = (int64_t)p->B * p->H * (p->dv / 16);
  int nw = 2;
  while (nw < 8 && nw * 16 < p->dv && warps > (int64_t)nw * device_sm_count()) nw *= 2;
  const int prep_smem = prepare_rows_bytes(DK) + 5 * BT * 4, scan_smem = scan_smem_bytes(DK, nw);
  CUtensorMap tmK, tmQ, tmV;
  const uint64_t kdims[3] = {(uint64_t)p->G * DK, (uint64_t)p->L, (uint64_t)p->B}, vdims[3] = {(uint64_t)p->H * p->dv, (uint64_t)p->L, (uint64_t)p->B};
  const uint64_t strides[2] = {(uint64_t)p->ld * 2, (uint64_t)p->L * p->ld * 2};
  const uint32_t kbox[3] = {64, BT, 1}, vbox[3] = {(uint32_t)nw * 16, BT, 1};
  int rc;
  if ((rc = make_tmap_nd_bf16(&tmK, p->k, 3, kdims, strides, kbox, true)) || (rc = make_tmap_nd_bf16(&tmQ, p->q, 3, kdims, strides, kbox, true)) ||
      (rc = make_tmap_nd_bf16(&tmV, p->v, 3, vdims, strides, vbox, false))) return rc;
  static unsigned long long done_prep = 0, done_scan = 0;
  if ((rc = ensure_dyn_smem(delta_prepare_kernel<DK>, prep_smem, done_prep)) || (rc = ensure_dyn_smem(delta_scan_kernel<DK>, scan_smem_bytes(DK, 8), done_scan))) return rc;
  for (int64_t first = 0; first < s.blocks; first += s.slab) {
    a.first = first; a.n_blocks = (int)std::min<int64_t>(s.slab, s.blocks - first);
    a.zero_start = first == 0 && (p->zero_start || !p->state);
    a.store_state = p->state || s.state;
    delta_prepare_kernel<DK><<<dim3(a.n_blocks, a.H, a.B), 128, prep_smem, st>>>(a);
    if ((rc = check_launch("evo_gated_delta_fwd(prepare)"))) return rc;
    delta_scan_kernel<DK><<<dim3(a.H, a.B, (a.dv / 16 + nw - 1) / nw), nw * 32, scan_smem, st>>>(tmK, tmQ, tmV, a);
    if ((rc = check_launch("evo_gated_delta_fwd(scan)"))) return rc;
  }
  const int64_t rows = (int64_t)p->B * p->L, w = rows * p->H;
  const bool wide = p->ldz % 4 == 0 && p->ldo % 4 == 0 && (((uintptr_t)p->gate | (uintptr_t)p->out | (uintptr_t)p->norm_w) & 7) == 0;
  auto norm = !wide ? delta_norm_kernel : (p->dv == 128 ? delta_norm4_kernel<4> : (p->dv == 64 ? delta_norm4_kernel<2> : (p->dv == 32 ? delta_norm4_kernel<1> : delta_norm_kernel)));
  const int per_cta = norm == delta_norm_kernel ? 8 : 32;
  norm<<<(unsigned)((w + per_cta - 1) / per_cta), 256, 0, st>>>(a.y, (const bf16*)p->gate, p->ldz, (const bf16*)p->norm_w, (bf16*)p->out, p->ldo, rows, p->H, p->dv, p->eps);
  return check_launch("evo_gated_delta_fwd(norm)");
}

}  // namespace

size_t evo::delta_block_workspace(const evo_gated_delta_params* p) {
  if (!taken(p)) return 0;
  const Sizes s = sizes(p);
  return s.total();
}

int evo::delta_block_fwd(const evo_gated_delta_params* p, void* ws, size_t bytes, cudaStream_t st) {
  const Sizes s = sizes(p);
  EVO_REQUIRE(ws && bytes >= s.total(), "evo_gated_delta_fwd: workspace too small (%zu < %zu)", bytes, s.total());
  uint8_t* base = (uint8_t*)(((uintptr_t)ws + 255) & ~(uintptr_t)255);
  return p->dk == 64 ? run<64>(p, s, base, st) : run<128>(p, s, base, st);
}
