// Gated delta rule over prompts by blocks of 64 tokens on the tensor cores (evo_gated_delta_fwd, bf16 activations; matrix_state.cu holds the entry point and the
// token-by-token form).  With the block's decays g, G_i = g_1 .. g_i, Gam_ij = g_{j+1} .. g_i, and the state S in front of it:
//   u_i = beta_i (v_i - G_i S^T k_i - sum_{j<i} Gam_ij (k_i . k_j) u_j)      o_i = G_i S^T q_i + sum_{j<=i} Gam_ij (q_i . k_j) u_j      S' = G_64 S + sum_j Gam_64,j k_j u_j^T
// i.e. U = T diag(beta) (V - diag(G) K S) with T = (1 + A)^-1, A_ij = beta_i Gam_ij (k_i . k_j) below the diagonal; O = diag(G) Q S + P U.
//
// delta_prepare_kernel, one CTA per (block, head, sequence), all in parallel: what does not depend on the state.  k . k and q . k as bf16 products (exact) with fp32
//   sums, norms and gates in fp32, sums of log decays in 64 bits (their differences enter as two floats), T in fp32 by halves: two triangles of 32 by forward
//   substitution (one column per thread), the square between them by products of three-part splits.
//   T diag(beta) and P go to the workspace as three bf16 parts (24 bits), in the order in which the next kernel's lanes read them.
// delta_single_kernel, the recurrence of a call of one block where there are many (head, sequence) pairs.
// delta_scan_kernel, blocks one after another on the fifth-generation tensor cores, everything transposed (value channels = rows): the sums of one product, split by the warps that
//   read them from TMEM, are the first operand of the next, in TMEM too:
//     W^T = V^T - S^T K^T (x G rk);  Q^T-part = S^T Q^T;  U^T = W^T T^T;  O^T += U^T P^T;  S'^T = G S^T + (U Gam rk)^T K
//   S, W, U are fp32 and enter as three bf16 parts; K and Q are bf16 as they stand (their norms scale the sums); T, P have three parts and meet W, U in the six products
//   down to 2^-16 of the leading one.  K, Q, V, T, P of the next block arrive by bulk copies while one is in work; the read-outs are normed, weighted and gated by warps of their own.
// Measured (B200): 4 x 4096 tokens, 16 heads of 128 x 128: 329 us (token by token 2774; the scan on mma.sync, one warp per 16 channels and a launch of its own for the head norm, 588);
// the kernels by themselves: the scan 224 (395 + 51), delta_prepare_kernel 92 (135 with the norms summed apart, both matrices stored and read again, and the square of T by
// multiply-adds from shared memory: 15.7 k instructions and 5.5 k shared-memory wavefronts an item then, 10.5 k and 2.3 k now; its four warps wait for one another at barriers; six CTAs per
// SM, which spill: 135); 1 x 777 tokens, 32 heads: 60 us (516; 113).  A block takes 6.3 k cycles, 4.1 k of them products (120 of M 64 and 40 or 25
// cycles, by clock stamps); what is left of the chain  state's parts - K S - W's parts - T W - U's parts - K U - state  is the splitting, bound by instructions (11 k warp instructions a
// block and CTA, four per element of W, U and S; three byte permutations of the half-rate integer pipe and four mixed multiply-adds of two numbers).
// A block in which U is not finite goes token by token: a product with a structural zero would carry a NaN to earlier tokens.
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
constexpr int PART_BYTES = 256;                         // one part of one tile: two 8 x 8 matrices, rows of 16 bytes
constexpr int TRI_BYTES = TILES * 3 * PART_BYTES;       // T or P of a block
enum { V_GK = 0, V_GQ, V_CK, V_RK, V_RQ, V_BETA, V_G, V_ROWS };       // -G rk | G rq | Gam_64 rk | rk | rq | beta | g
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
  float* y;                                             // (rows, H * dv) fp32 read-outs, where a norm of its own follows
  int norm, pair, wide;                                 // head norm, weight and gate here; with a second CTA; their rows start on four elements
  const bf16* gate; const bf16* norm_w; bf16* out; int64_t ldo; float eps;
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
// the three parts (split3) of two neighbours of a row, to a lane's place in the tiles of each part
__device__ __forceinline__ void store_parts(uint8_t* dst, float2 x) {
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const uint32_t w = tops(x.x, x.y);
    *reinterpret_cast<uint32_t*>(dst + s * TILES * PART_BYTES) = w;
    if (s < 2) x = take_away(x, w);
  }
}

constexpr int AP = BT + 4;                                   // floats of a row of A (16-byte pieces)
__host__ __device__ constexpr int prepare_smem_bytes(int dk) { return 2 * BT * (2 * dk + 16) + 5 * BT * 4; }
template <int DK>
__global__ void __launch_bounds__(128) delta_prepare_kernel(const Args p) {
  constexpr int PITCH = 2 * DK + 16;                         // bytes of a key row
  static_assert(BT * AP * 4 <= 2 * BT * PITCH, "A fits where the keys and queries were");
  extern __shared__ __align__(16) uint8_t sm[];
  uint8_t* ks = sm;                                          // [BT] keys, [BT] queries
  float* As = reinterpret_cast<float*>(sm);                  // [BT][AP] A, then T, in the place of the keys and queries once they are multiplied
  float* rk = reinterpret_cast<float*>(sm + 2 * BT * PITCH);
  float* rq = rk + BT;
  float* beta = rq + BT;
  float* lh = beta + BT;                                     // running log decay, high and low float
  float* ll = lh + BT;
  pdl_wait();                                                // itself launched dependent: what it writes may still be read, and what the scan reads before its own wait must be there
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x, h = blockIdx.y, b = blockIdx.z, g = h / (p.H / p.G);
  const int64_t t0 = (p.first + blk) * BT, row0 = (int64_t)b * p.L + t0;
  const int nt = (int)min((int64_t)BT, p.L - t0);
  uint8_t* out = p.blocks + (((int64_t)b * p.H + h) * p.n_blocks + blk) * BLOCK_BYTES;
  float* vec = reinterpret_cast<float*>(out + 2 * TRI_BYTES);
  if (p.first == 0 && (blk | h | b | tid) == 0) *p.failed = 0u;
  {
    constexpr int STEP = 128 / (DK / 8);                     // rows that the CTA copies at a time
    const int c = tid % (DK / 8), r0 = tid / (DK / 8);
    const int64_t col = (int64_t)g * DK + c * 8;
    const bf16 *kp = p.k + (row0 + r0) * p.ld + col, *qp = p.q + (row0 + r0) * p.ld + col;
    const uint32_t dst = smem_u32(ks) + r0 * PITCH + c * 16;
#pragma unroll
    for (int i = 0; i < BT / STEP; ++i) {
      const bool on = r0 + i * STEP < nt;
      cp16(dst + i * STEP * PITCH, on ? kp : p.k, on);
      cp16(dst + (BT + i * STEP) * PITCH, on ? qp : p.q, on);
      kp += STEP * p.ld; qp += STEP * p.ld;
    }
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
#pragma unroll
    for (int u = 0; u < 2; ++u) vec[V_G * BT + 2 * lane + u] = expf(gl[u]);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    // ---- k . k and q . k: warp = 16 rows i, the 16 columns of [d] d warps further to the left; and q . q of the rows themselves for their norms (k . k has them on its diagonal)
    const int gq = lane >> 2, tq = lane & 3, i0 = warp * 16;
    float kk[4][2][4], qk[4][2][4], qq[2][4];
#pragma unroll
    for (int d = 0; d < 4; ++d)
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) { kk[d][u][e] = qk[d][u][e] = 0.f; if (d == 0) qq[u][e] = 0.f; }
    const uint32_t arow = smem_u32(ks) + (i0 + (lane & 15)) * PITCH + (lane >> 4) * 16;
    const uint32_t brow = smem_u32(ks) + (i0 + (lane & 7) + ((lane >> 4) << 3)) * PITCH + ((lane >> 3) & 1) * 16;
#pragma unroll 2
    for (int kt = 0; kt < DK / 16; ++kt) {
      uint32_t ak[4], aq[4], bk[4];
      ldmatrix_x4_at(ak, arow + kt * 32);
      ldmatrix_x4_at(aq, arow + BT * PITCH + kt * 32);
      ldmatrix_x4_at(bk, brow + BT * PITCH + kt * 32);
      mma_np(qq[0], aq, bk[0], bk[1]); mma_np(qq[1], aq, bk[2], bk[3]);
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        if (d <= warp) {
          ldmatrix_x4_at(bk, brow - d * 16 * PITCH + kt * 32);
          mma_np(kk[d][0], ak, bk[0], bk[1]); mma_np(kk[d][1], ak, bk[2], bk[3]);
          mma_np(qk[d][0], aq, bk[0], bk[1]); mma_np(qk[d][1], aq, bk[2], bk[3]);
        }
      }
    }
    if (tq == gq >> 1) {
      const bool odd = gq & 1;
      rk[i0 + gq] = 1.0f / sqrtf((odd ? kk[0][0][1] : kk[0][0][0]) + p.unit_eps);
      rk[i0 + gq + 8] = 1.0f / sqrtf((odd ? kk[0][1][3] : kk[0][1][2]) + p.unit_eps);
      rq[i0 + gq] = p.q_scale / sqrtf((odd ? qq[0][1] : qq[0][0]) + p.unit_eps);
      rq[i0 + gq + 8] = p.q_scale / sqrtf((odd ? qq[1][3] : qq[1][2]) + p.unit_eps);
    }
    __syncthreads();
    // ---- A to shared memory; P goes to the workspace from here, as a second operand: column n = token i, k = token j; lane (gq, tq) of tile (kt, nt): i = 8 nt + gq,
    // j = 16 kt + 8 u + 2 tq + {0, 1}
    float lhi[2], lli[2], rqi[2], bri[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) { const int i = i0 + gq + 8 * r; lhi[r] = lh[i]; lli[r] = ll[i]; rqi[r] = rq[i]; bri[r] = beta[i] * rk[i]; }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      if (d > warp) continue;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int kt = warp - d, j = kt * 16 + 8 * u + 2 * tq;
        const float2 lhj = *reinterpret_cast<const float2*>(lh + j), llj = *reinterpret_cast<const float2*>(ll + j), rkj = *reinterpret_cast<const float2*>(rk + j);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = i0 + gq + 8 * r;
          const float g0 = expf((lhi[r] - lhj.x) + (lli[r] - llj.x)) * rkj.x, g1 = expf((lhi[r] - lhj.y) + (lli[r] - llj.y)) * rkj.y;
          float2 P = make_float2(g0 * rqi[r] * qk[d][u][2 * r], g1 * rqi[r] * qk[d][u][2 * r + 1]);
          if (d == 0) { if (j > i) P.x = 0.f; if (j + 1 > i) P.y = 0.f; }
          store_parts(out + TRI_BYTES + (kt * (9 - kt) + 2 * (warp - kt) + r) * PART_BYTES + u * 128 + lane * 4, P);
          // (what lies on and above the diagonal of A is not used)
          *reinterpret_cast<float2*>(As + i * AP + j) = make_float2(bri[r] * (g0 * kk[d][u][2 * r]), bri[r] * (g1 * kk[d][u][2 * r + 1]));
        }
      }
    }
  }
  __syncthreads();
  // ---- T = (1 + A)^-1 in fp32: the two diagonal blocks of 32 by forward substitution, one column per thread (one block of 64 would be 2016 multiply-adds in a row, an instruction
  // stream no cache holds); then the square below them
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
    vec[V_GK * BT + t] = -G * rk[t];
    vec[V_GQ * BT + t] = G * rq[t];
    vec[V_CK * BT + t] = expf((lh[BT - 1] - lh[t]) + (ll[BT - 1] - ll[t])) * rk[t];
    vec[V_RK * BT + t] = rk[t]; vec[V_RQ * BT + t] = rq[t]; vec[V_BETA * BT + t] = beta[t];
    if (t == BT - 1) vec[V_ROWS * BT] = G;
  }
  __syncthreads();
  {
    // T21^T = -(T11^T A21^T) T22^T: the sums of the first product are, lane by lane, the first operand of the second.  A warp has 16 columns c of T11 and 16 rows i of T22
    const int gq = lane >> 2, tq = lane & 3, c = (warp & 1) * 16 + gq, ih = warp >> 1;
    const float* A21 = As + 32 * AP;
    const float* T22 = A21 + 32;
    constexpr int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};       // small products first
    const auto second = [&](const float* at, uint32_t (&w)[3][2]) {             // a column of the second operand: two neighbours, and those eight further on
      const float2 x = *reinterpret_cast<const float2*>(at), y = *reinterpret_cast<const float2*>(at + 8);
      split3(x.x, x.y, w[0][0], w[1][0], w[2][0]);
      split3(y.x, y.y, w[0][1], w[1][1], w[2][1]);
    };
    float X[4][4], Y[2][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) { X[n][e] = 0.f; if (n < 2) Y[n][e] = 0.f; }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k < (warp & 1)) continue;                                             // (T11 is zero there)
      uint32_t a[3][4];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float* at = As + (16 * k + 8 * (v >> 1) + 2 * tq) * AP + c + 8 * (v & 1);
        split3(at[0], at[AP], a[0][v], a[1][v], a[2][v]);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (n >= 2 && !ih) continue;                                            // (nor does T22 have what would meet these)
        uint32_t w[3][2];
        second(A21 + (8 * n + gq) * AP + 16 * k + 2 * tq, w);
#pragma unroll
        for (int m = 0; m < 6; ++m) mma_np(X[n], a[pa[m]], w[pb[m]][0], w[pb[m]][1]);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k > ih) continue;
      uint32_t a[3][4];
#pragma unroll
      for (int v = 0; v < 4; ++v) split3(X[2 * k + (v >> 1)][2 * (v & 1)], X[2 * k + (v >> 1)][2 * (v & 1) + 1], a[0][v], a[1][v], a[2][v]);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        uint32_t w[3][2];
        second(T22 + (16 * ih + 8 * n + gq) * AP + 16 * k + 2 * tq, w);
#pragma unroll
        for (int m = 0; m < 6; ++m) mma_np(Y[n], a[pa[m]], w[pb[m]][0], w[pb[m]][1]);
      }
    }
    __syncthreads();                                                            // A21 has been read
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) As[(32 + 16 * ih + 8 * n + 2 * tq + (e & 1)) * AP + c + 8 * (e >> 1)] = -Y[n][e];
  }
  __syncthreads();
  // ---- T diag(beta), laid down like P
  for (int e = warp; e < TILES; e += 4) {
    int kt = 0, x = e;
    while (x >= 8 - 2 * kt) { x -= 8 - 2 * kt; ++kt; }
    const int i = 8 * (x + 2 * kt) + (lane >> 2), j = 16 * kt + 2 * (lane & 3);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int jj = j + 8 * u;
      const float2 t = *reinterpret_cast<const float2*>(As + i * AP + jj), bt = *reinterpret_cast<const float2*>(beta + jj);
      store_parts(out + e * PART_BYTES + u * 128 + lane * 4, make_float2(jj <= i ? t.x * bt.x : 0.f, jj + 1 <= i ? t.y * bt.y : 0.f));
    }
  }
}

// ------------------------------------------------------------------------------------------------ the recurrence
// A CTA has 64 value channels of a (head, sequence): 16 lanes of each quarter of TMEM (the layout of products with M = 64).  TMEM's lanes belong to
// the schedulers, so a warp instruction on a quarter's 16 lanes (shapes 16x256b and 16x128b, whose fragments are those of mma.sync) does half the work of one on 32, and 128 channels go
// to two CTAs, a cluster (one CTA for 128 channels, 32 lanes an instruction: 13.4 k cycles a block, bound by the issue of 27 k instructions; two: 6.3 k).
// Eight warps split what one product leaves as fp32 sums into the three parts that the next one multiplies; the two warps of a channel hold half of its state each (HC columns, in
// registers) and 32 of the block's tokens of W and U.
// TMEM columns: the state's parts, which the state's update overwrites once they are multiplied (DK = 128; DK = 64 has columns to spare), W (then U) and O as they are summed, the
// parts of W (then U), the parts of U Gam rk
template <int DK> struct Columns {
  static constexpr int HC = DK / 2, S = 0, S_HALF = 3 * HC / 2, DS = DK == 128 ? 0 : 96, DS_HALF = DK == 128 ? S_HALF : HC, W = 192, O = 256, WP = 320, UP = 416;
};
static_assert(Columns<64>::DS + 64 <= Columns<64>::W && Columns<128>::S_HALF * 2 <= Columns<128>::W, "TMEM columns overlap");
constexpr int MMA_M = 64;
constexpr int CH = 64;                                                     // value channels of a CTA
constexpr int SPLIT_WARPS = 8, EPI_WARPS = 4, SCAN_THREADS = 640;         // two groups of read-out warps, which take the blocks in turn; a warp each for the copies and the products
constexpr int COPY_WARP = SPLIT_WARPS + 2 * EPI_WARPS, MMA_WARP = COPY_WARP + 1;
constexpr int SPLIT_REGS = 112, EPI_REGS = 104, OTHER_REGS = 40;          // shares of the launch's 96 a thread
static_assert(SPLIT_WARPS * 32 * SPLIT_REGS + 2 * EPI_WARPS * 32 * EPI_REGS + 128 * OTHER_REGS <= SCAN_THREADS * 96, "register shares exceed the launch");
constexpr int OUT_PITCH = CH + 4;                       // floats of a token's row on its way from lanes to rows
constexpr int OUT_BYTES = BT * OUT_PITCH * 4;           // of a block
constexpr int V_BYTES = BT * CH * 2;
constexpr int NORM_TURNS = 2;                           // places for the other CTA's sums of squares, for the blocks of a parity in turn

// 16 lanes; a thread has row lane / 4 (and + 8), columns 2 (lane & 3) and the next of every eight: [8 columns][row, row + 8][2]
template <int N> __device__ __forceinline__ void tmem_ld(uint32_t taddr, float2 (&x)[N]) {
  static_assert(N == 4 || N == 8, "");
  uint32_t r[2 * N];
  if constexpr (N == 4)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
  else
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// packed pairs of the same thread and columns: four columns of words for every eight
template <int N> __device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[N]) {
  static_assert(N == 2 || N == 4 || N == 8, "");
  if constexpr (N == 2) asm volatile("tcgen05.st.sync.aligned.16x128b.x1.b32 [%2], {%0, %1};" ::"r"(r[0]), "r"(r[1]), "r"(taddr) : "memory");
  else if constexpr (N == 4) asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%4], {%0, %1, %2, %3};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(taddr) : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
// the three parts (split3) of a thread's fragment, `apart` columns from one to the next
template <int N> __device__ __forceinline__ void put_parts(uint32_t at, uint32_t apart, const float2* given) {
  float2 x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = given[i];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    uint32_t w[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      w[i] = tops(x[i].x, x[i].y);
      if (s < 2) x[i] = take_away(x[i], w[i]);
    }
    tmem_st(at + s * apart, w);
  }
}
// a triangle's tiles as delta_prepare_kernel lays them down: 8 x 8 matrices of 128 bytes, two of them a step of 16 tokens j, 256 bytes from eight tokens i to the next
__device__ __forceinline__ uint64_t desc_tri(uint32_t addr) { return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(128 >> 4) << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46; }
// one product, the second operand's descriptor in two words
template <bool ADD> __device__ __forceinline__ void product(uint32_t lead, uint32_t d, uint32_t a, uint32_t lo, uint32_t hi, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred e;\n\t.reg .b64 b;\n\tsetp.ne.b32 e, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, %6;\n\t}\n"
               ::"r"(d), "r"(a), "r"(lo), "r"(hi), "r"(idesc), "r"(lead), "n"(ADD ? 1 : 0) : "memory");
}

__host__ __device__ constexpr int stage_bytes(int dk) { return 2 * BT * dk * 2 + V_BYTES + BLOCK_BYTES; }          // a multiple of 1024
__host__ __device__ constexpr int scan_smem_bytes(int dk) { return 1024 + 2 * stage_bytes(dk) + 2 * OUT_BYTES; }

template <int DK>
__global__ void __launch_bounds__(SCAN_THREADS, 1) delta_scan_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmV, const Args p) {
  using T = Columns<DK>;
  constexpr int BOX = BT * 128, ROWS_BYTES = DK / 64 * BOX, HC = T::HC, STAGE = stage_bytes(DK);      // boxes of 64 columns, 16-byte pieces of a row swizzled by row & 7
  static_assert(STAGE % 1024 == 0, "");
  extern __shared__ __align__(16) uint8_t sm_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[2], empty[2], s_ready, w_done, wp_ready, u_done, up_ready, pu_ready, ds_done[2], qs_done[2], o_done[2], o_free, fixed[2], half_met[4], rows_met[2], norm_met[2][NORM_TURNS], ended;
  __shared__ uint32_t tmem_slot;
  __shared__ int odd[2];                                // W or U of block (parity) holds something that is not finite
  __shared__ float part_sum[2][3][2][CH];               // of a token (parity): S^T k, S^T q, k . q over half the key channels
  __shared__ float norm_sum[2][NORM_TURNS][BT];         // of a block (parity, and its turn among those of that parity): the other CTA's sums of squares
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int h = blockIdx.x, b = blockIdx.y, g = h / (p.H / p.G), dv = p.dv, c0 = blockIdx.z * CH;
  const int64_t rowb = (int64_t)b * p.L + p.first * BT, left = p.L - p.first * BT;       // the slab's first row; tokens from there
  const uint8_t* blocks = p.blocks + ((int64_t)b * p.H + h) * p.n_blocks * (int64_t)BLOCK_BYTES;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1 + SPLIT_WARPS + EPI_WARPS); mbar_init(&ds_done[i], 1); odd[i] = 0;
      mbar_init(&qs_done[i], 1); mbar_init(&o_done[i], 1); mbar_init(&fixed[i], 4); mbar_init(&rows_met[i], EPI_WARPS);
      for (int k = 0; k < NORM_TURNS; ++k) mbar_init(&norm_met[i][k], 1);
    }
    mbar_init(&s_ready, SPLIT_WARPS); mbar_init(&w_done, 1); mbar_init(&wp_ready, SPLIT_WARPS); mbar_init(&u_done, 1); mbar_init(&up_ready, SPLIT_WARPS);
    mbar_init(&pu_ready, SPLIT_WARPS + EPI_WARPS);               // the parts of U, and Q S read
    mbar_init(&o_free, EPI_WARPS); mbar_init(&ended, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&half_met[i], 2);
    fence_barrier_init();
  }
  if (warp == MMA_WARP) { tmem_alloc<1>(&tmem_slot, 512); tmem_relinquish<1>(); }
  const bool given_up = p.first > 0 && *(volatile unsigned int*)p.failed;      // (of the slab in front, which was through before this one's delta_prepare_kernel began)
  tc_fence_before();
  const bool skip = __syncthreads_or(given_up);
  tc_fence_after();
  if (p.pair) cluster_sync_all();                        // the other CTA's barriers are there
  const uint32_t tmem = tmem_slot;
  const int n_blocks = skip ? 0 : p.n_blocks;
  const auto wait = [&](uint64_t* bar, uint32_t parity) { return warp_wait_or_give_up(bar, parity, p.waits); };
  // a warp's report behind its reads (or, after their completion, writes) of TMEM
  const auto report = [&](uint64_t* bar) { tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(bar); __syncwarp(); };
  bool ok = true;

  if (warp < SPLIT_WARPS) {
    regs_up<SPLIT_REGS>();
    const int q = warp & 3, hf = warp >> 2, c = q * 16 + gq;                       // the thread's channels: c and c + 8
    const bool works = c0 + q * 16 < dv;                                   // (dv is a multiple of 16)  a warp without a channel only reports: its lanes' products are read by nobody
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
    float* Sg = p.state + (((int64_t)b * p.H + h) * DK + hf * HC + 2 * tq) * (int64_t)dv + c0 + c;
    float2 S[HC / 4];                                                      // [8 columns][row]
    const auto state_at = [&](int i, int e) -> float& { return Sg[(int64_t)(i / 2 * 8 + e) * dv + (i & 1) * 8]; };
#pragma unroll
    for (int i = 0; i < HC / 4; ++i) S[i] = (p.zero_start || !works || skip) ? make_float2(0.f, 0.f) : make_float2(state_at(i, 0), state_at(i, 1));
    const auto publish = [&] {
      if (works) {
#pragma unroll
        for (int i = 0; i < HC / 32; ++i) put_parts<8>(lanes + T::S + hf * T::S_HALF + 16 * i, HC / 2, S + 8 * i);
        tmem_st_wait();
      }
      report(&s_ready);
    };
    // (with the state's parts a warp reports that it has seen the block's copies land: the products wait for nothing else)
    if (n_blocks) { ok = wait(&full[0], 0); if (ok) publish(); }
#pragma unroll 1
    for (int blk = 0; blk < n_blocks && ok; ++blk) {
      const uint32_t ph = blk & 1;
      const uint8_t* ks = sm + ph * STAGE;
      const uint8_t* vs = ks + 2 * ROWS_BYTES;
      const float* vec = reinterpret_cast<const float*>(vs + V_BYTES + 2 * TRI_BYTES);
      const float* vec2 = vec + 32 * hf + 2 * tq;        // of the thread's tokens 32 hf + 8 n + 2 tq, + 1
      // ---- W = V - G rk (K S)
      ok = wait(&w_done, ph);
      if (!ok) break;
      tc_fence_after();
      if (works) {
        float2 x[8];
        tmem_ld(lanes + T::W + 32 * hf, x);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t v[4];                                 // (tokens 0-7, channels 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15), turned
          ldmatrix_x4_trans_at(v, smem_u32(vs) + (32 * hf + 16 * m + (lane & 7) + ((lane >> 4) << 3)) * 128 + (((2 * q + (lane >> 3 & 1)) ^ (lane & 7)) << 4));
#pragma unroll
          for (int i = 0; i < 4; ++i)
            x[4 * m + i] = __ffma2_rn(*reinterpret_cast<const float2*>(vec2 + V_GK * BT + 16 * m + i / 2 * 8), x[4 * m + i], make_float2(bf_lo(v[i]), bf_hi(v[i])));
        }
        put_parts<8>(lanes + T::WP + 16 * hf, 32, x);
        tmem_st_wait();
      }
      report(&wp_ready);
      // ---- U, first weighted for the state, then as it is for the read-outs
      ok = wait(&u_done, ph);
      if (!ok) break;
      tc_fence_after();
      if (works) {
        float2 u[8], x[8], wrong = make_float2(0.f, 0.f);
        tmem_ld(lanes + T::W + 32 * hf, u);
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          x[n] = __fmul2_rn(u[n], *reinterpret_cast<const float2*>(vec2 + V_CK * BT + n / 2 * 8));
          wrong = __ffma2_rn(make_float2(0.f, 0.f), u[n], wrong);          // (a W that is not finite leaves no U that is: T's diagonal times a NaN among its parts)
        }
        if (wrong.x + wrong.y != 0.f) odd[ph] = 1;
        __syncwarp();
        put_parts<8>(lanes + T::UP + 16 * hf, 32, x);
        tmem_st_wait();
        report(&up_ready);
        put_parts<8>(lanes + T::WP + 16 * hf, 32, u);
        tmem_st_wait();
      } else report(&up_ready);
      report(&pu_ready);
      // ---- S = G_64 S + (U Gam rk)^T K
      const float G = vec[V_ROWS * BT];
      ok = wait(&ds_done[hf], ph);
      if (!ok) break;
      tc_fence_after();
      if (*(volatile int*)&odd[ph] == 0) {
        if (works) {
#pragma unroll
          for (int n = 0; n < HC / 4; n += 8) {
            float2 x[8];
            tmem_ld(lanes + T::DS + hf * T::DS_HALF + 4 * n, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) S[n + i] = __ffma2_rn(make_float2(G, G), S[n + i], x[i]);
          }
        }
      } else {
        // token by token, as the recurrence is defined; a channel's quads and halves exchange their sums.  The read-outs go to the columns of O once the products there are through.
        ok = wait(&o_done[ph], (blk >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const int nt = (int)min((int64_t)BT, left - (int64_t)blk * BT);
        float kept[2] = {0.f, 0.f};
#pragma unroll 1
        for (int t = 0; t < BT; ++t) {
          const float dec = t < nt ? vec[V_G * BT + t] : 1.f, be = vec[V_BETA * BT + t], nk = vec[V_RK * BT + t], nq = vec[V_RQ * BT + t];
          const auto two = [&](int side, int n, float norm) {            // keys (side 0) or queries hf HC + 8 n + 2 tq and the next
            const int d = hf * HC + 8 * n;
            const uint32_t w = *reinterpret_cast<const uint32_t*>(ks + side * ROWS_BYTES + (d >> 6) * BOX + t * 128 + ((((d >> 3) & 7) ^ (t & 7)) << 4) + 4 * tq);
            return make_float2(bf_lo(w) * norm, bf_hi(w) * norm);
          };
          float pk[2] = {0.f, 0.f}, po[2] = {0.f, 0.f}, kq = 0.f;
#pragma unroll
          for (int n = 0; n < HC / 8; ++n) {
            const float2 kv = two(0, n, nk), qv = two(1, n, nq);
            kq = fmaf(kv.y, qv.y, fmaf(kv.x, qv.x, kq));
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              float2& s = S[2 * n + u];
              s.x *= dec; s.y *= dec;
              pk[u] = fmaf(s.y, kv.y, fmaf(s.x, kv.x, pk[u]));
              po[u] = fmaf(s.y, qv.y, fmaf(s.x, qv.x, po[u]));
            }
          }
          kq = quad_sum(kq);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            pk[u] = quad_sum(pk[u]); po[u] = quad_sum(po[u]);
            if (tq == 0) { part_sum[t & 1][0][hf][c + 8 * u] = pk[u]; part_sum[t & 1][1][hf][c + 8 * u] = po[u]; part_sum[t & 1][2][hf][c + 8 * u] = kq; }
          }
          report(&half_met[q]);
          ok = wait(&half_met[q], t & 1);                                // (64 meetings a block: the parity starts anew)
          if (!ok) break;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const auto sum = [&](int k) { return part_sum[t & 1][k][0][c + 8 * u] + part_sum[t & 1][k][1][c + 8 * u]; };
            const int col = c + 8 * u;
            const float x = be * (__bfloat162float(*reinterpret_cast<const bf16*>(vs + t * 128 + (((col >> 3) ^ (t & 7)) << 4) + (col & 7) * 2)) - sum(0));
            if ((t & 3) == tq) kept[u] = fmaf(x, sum(2), sum(1));
            if (t < nt) {
#pragma unroll
              for (int n = 0; n < HC / 8; ++n) { const float2 kv = two(0, n, nk); float2& s = S[2 * n + u]; s.x = fmaf(kv.x, x, s.x); s.y = fmaf(kv.y, x, s.y); }
            }
          }
          __syncwarp();
          if (hf == 0 && (t & 3) == 3) { const uint32_t w[2] = {__float_as_uint(kept[0]), __float_as_uint(kept[1])}; tmem_st(lanes + T::O + (t & ~3), w); }
        }
        if (!ok) break;
        if (hf == 0) { tmem_st_wait(); report(&fixed[ph]); }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[ph]);
      if (tid == 0 && blk) odd[ph ^ 1] = 0;              // the last block's: everyone has read it (the read-outs' warps before this block's Q S could be asked for)
      __syncwarp();
      if (blk + 1 < n_blocks) { ok = wait(&full[ph ^ 1], ((blk + 1) >> 1) & 1); if (ok) publish(); }
    }
    const bool lost = __syncthreads_or(!ok);
    if (lost) { if (tid == 0) { pdl_wait(); *p.failed = 1u; } }            // (delta_prepare_kernel, which clears the word, may still be running)
    else if (p.store_state && works && !skip) {
      asm volatile("" : "+l"(Sg));                       // (or the compiler keeps the addresses of the loads above, two registers each, over the whole recurrence)
#pragma unroll
      for (int i = 0; i < HC / 4; ++i) { state_at(i, 0) = S[i].x; state_at(i, 1) = S[i].y; }
    }
  } else if (warp < COPY_WARP) {
    // ================================================ read-outs: O = G rq (Q S) + P U, turned from lanes to rows, normed and gated
    regs_up<EPI_REGS>();
    const int q = warp & 3, c = q * 16 + gq, group = (warp - SPLIT_WARPS) >> 2;          // the group's blocks: those of its parity
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
    float* rows_out = reinterpret_cast<float*>(sm + 2 * STAGE + group * OUT_BYTES);
    int repaired = 0, met = 0;
    const auto meet = [&] { __syncwarp(); if (lane == 0) mbar_arrive(&rows_met[group]); __syncwarp(); const bool all = wait(&rows_met[group], met & 1); ++met; return all; };
    // rows: half a warp per token, four channels per lane; tokens 16 q + 2 u + side, u = 0..7
    const int side = lane >> 4, e0 = c0 + 4 * (lane & 15);
    const bool mine = e0 < dv;
    float2 w01 = make_float2(0.f, 0.f), w23 = w01;
    if (p.norm && mine) {
      const bf16* w = p.norm_w + e0;
      w01 = make_float2(__bfloat162float(w[0]), __bfloat162float(w[1])); w23 = make_float2(__bfloat162float(w[2]), __bfloat162float(w[3]));
    }
#pragma unroll 1
    for (int blk = group; blk < n_blocks; blk += 2) {
      const uint32_t ph = group, turn = (blk >> 1) & 1;
      const float* vec = reinterpret_cast<const float*>(sm + ph * STAGE + 2 * ROWS_BYTES + V_BYTES + 2 * TRI_BYTES);
      const int nt = (int)min((int64_t)BT, left - (int64_t)blk * BT), mine_nt = mine ? nt - q * 16 - side : 0;      // (the thread's tokens 2 u < mine_nt)
      const int64_t row0 = rowb + (int64_t)blk * BT + q * 16 + side;
      uint2 gates[8];
      if (p.norm) {
        const bf16* gr = p.gate + row0 * p.ldz + (int64_t)h * dv + e0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          gates[u] = make_uint2(0u, 0u);
          const bf16* r = gr + 2 * u * p.ldz;
          if (2 * u < mine_nt) {
            if (p.wide) gates[u] = __ldg(reinterpret_cast<const uint2*>(r));
            else gates[u] = make_uint2((uint32_t)__bfloat16_as_ushort(r[0]) | (uint32_t)__bfloat16_as_ushort(r[1]) << 16, (uint32_t)__bfloat16_as_ushort(r[2]) | (uint32_t)__bfloat16_as_ushort(r[3]) << 16);
          }
        }
      }
      ok = wait(&full[ph], turn) && wait(&qs_done[ph], turn);
      if (!ok) break;
      tc_fence_after();
      float2 o[16];                                      // [8 tokens][channel c, c + 8]
#pragma unroll
      for (int i = 0; i < 16; i += 8) {
        float2 x[8];
        tmem_ld(lanes + T::O + 4 * i, x);
#pragma unroll
        for (int n = 0; n < 8; ++n) o[i + n] = __fmul2_rn(x[n], *reinterpret_cast<const float2*>(vec + V_GQ * BT + 4 * i + n / 2 * 8 + 2 * tq));
      }
      report(&pu_ready);
      if (lane == 0) mbar_arrive(&empty[ph]);
      __syncwarp();
      if (blk >= 2 && p.norm) { ok = meet(); if (!ok) break; }           // the rows of the group's last block are read
      // The exchange of the sums of squares: each CTA writes a block's into the other, where they are read behind the barrier of their place.  The blocks of a parity take two places in turn,
      // so that no sum is written over one that is still to be read, and no two blocks' bytes meet at a barrier: the other CTA sends block n + 4's, the next into block n's place, when its
      // warps have met at block n + 4, each with every sum of block n + 2 from here; and a warp here sends those of n + 2 when all have met there, with block n's read.  (With one place the
      // other CTA goes on to block n + 2 once block n's sums have left here, read or not.)
      const int place = (blk >> 1) % NORM_TURNS;
      if (p.pair && q == 0 && lane == 0) mbar_arrive_expect_tx(&norm_met[ph][place], BT * 4);
      __syncwarp();
      ok = wait(&o_done[ph], turn);
      if (!ok) break;
      const bool anew = *(volatile int*)&odd[ph] != 0;   // the split warps computed this block's token by token
      if (anew) {
        ok = wait(&fixed[ph], repaired & 1);
        if (!ok) break;
        ++repaired;
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = make_float2(0.f, 0.f);
      }
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 16; i += 8) {
        float2 x[8];
        tmem_ld(lanes + T::O + 4 * i, x);
#pragma unroll
        for (int n = 0; n < 8; ++n) o[i + n] = __fadd2_rn(o[i + n], x[n]);
      }
      report(&o_free);
      if (!p.norm) {
        if (c0 + q * 16 < dv) {
          float* yr = p.y + (rowb + (int64_t)blk * BT) * p.H * dv + (int64_t)h * dv + c0 + c;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int t = i / 4 * 8 + 2 * tq + (i & 1);
            if (t < nt) yr[(int64_t)t * p.H * dv + (i >> 1 & 1) * 8] = (i & 1) ? o[i / 2].y : o[i / 2].x;
          }
        }
        continue;
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) rows_out[(i / 4 * 8 + 2 * tq + (i & 1)) * OUT_PITCH + c + (i >> 1 & 1) * 8] = (i & 1) ? o[i / 2].y : o[i / 2].x;
      ok = meet();
      if (!ok) break;
      float4 x[8];
      float ss[8];
      const float* src = rows_out + (q * 16 + side) * OUT_PITCH + 4 * (lane & 15);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = mine ? *reinterpret_cast<const float4*>(src + 2 * u * OUT_PITCH) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 a = make_float2(x[u].x, x[u].y), c2 = make_float2(x[u].z, x[u].w), sq = __ffma2_rn(a, a, __fmul2_rn(c2, c2));
        ss[u] = sq.x + sq.y;
      }
      // eight sums over 16 lanes: a lane keeps half of them at each of three steps and ends with that of u = (lane >> 1) & 7
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int n = 4 >> k, d = 8 >> k;
        const bool up = lane & d;
#pragma unroll
        for (int u = 0; u < n; ++u) {
          const float keep = up ? ss[u + n] : ss[u], give = up ? ss[u] : ss[u + n];
          ss[u] = keep + __shfl_xor_sync(0xffffffffu, give, d);
        }
      }
      ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
      if (p.pair) {
        // the head's other channels are the other CTA's
        const uint32_t other = cluster_ctarank() ^ 1;
        const int t = q * 16 + (lane & 14) + side;
        if (!(lane & 1))
          asm volatile("{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
                       "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [ra], %3, [rb];\n\t}\n"
                       ::"r"(smem_u32(&norm_sum[ph][place][t])), "r"(smem_u32(&norm_met[ph][place])), "r"(other), "r"(__float_as_uint(ss[0])) : "memory");
        __syncwarp();
        ok = wait(&norm_met[ph][place], ((blk >> 1) / NORM_TURNS) & 1);
        if (!ok) break;
        ss[0] += norm_sum[ph][place][t];
      }
      const float rstd = 1.0f / sqrtf(ss[0] / (float)dv + p.eps);
      bf16* orow = p.out + row0 * p.ldo + (int64_t)h * dv + e0;
#pragma unroll
      for (int u = 0; u < 8; ++u, orow += 2 * p.ldo) {
        const float r1 = __shfl_sync(0xffffffffu, rstd, (lane & 16) + 2 * u);
        const float2 r2 = make_float2(r1, r1);
        const float2 a01 = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(x[u].x, x[u].y), r2), w01), silu2_bf16(make_float2(bf_lo(gates[u].x), bf_hi(gates[u].x))));
        const float2 a23 = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(x[u].z, x[u].w), r2), w23), silu2_bf16(make_float2(bf_lo(gates[u].y), bf_hi(gates[u].y))));
        const uint2 r = make_uint2(pack_bf16(a01.x, a01.y), pack_bf16(a23.x, a23.y));
        if (2 * u < mine_nt) {
          if (p.wide) *reinterpret_cast<uint2*>(orow) = r;
          else {
            orow[0] = __ushort_as_bfloat16((unsigned short)(r.x & 0xffffu)); orow[1] = __ushort_as_bfloat16((unsigned short)(r.x >> 16));
            orow[2] = __ushort_as_bfloat16((unsigned short)(r.y & 0xffffu)); orow[3] = __ushort_as_bfloat16((unsigned short)(r.y >> 16));
          }
        }
      }
      if (h == p.H - 1 && c0 == 0 && p.ldo > (int64_t)p.H * dv)
        for (int t = q * 16; t < min(nt, q * 16 + 16); ++t)
          for (int64_t e = (int64_t)p.H * dv + lane; e < p.ldo; e += 32) p.out[(rowb + (int64_t)blk * BT + t) * p.ldo + e] = __float2bfloat16_rn(0.f);
    }
    __syncthreads_or(!ok);
  } else {
    regs_down<OTHER_REGS>();
    if (warp == COPY_WARP) {
      // ================================================ copies: a block's rows of K, Q, V (rows behind the last token arrive as zeros) and its T, P and vectors
      if (lane == 0 && n_blocks) {
        tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmV);
        int blk = 0;
        pdl_wait();                                      // T, P and vectors; nothing else of this kernel, which may be launched dependent, comes from delta_prepare_kernel
        for (; blk < n_blocks; ++blk) {
          const int s = blk & 1;
          if (blk >= 2 && !wait_or_give_up(&empty[s], ((blk >> 1) - 1) & 1, p.waits)) { ok = false; break; }
          uint8_t* st = sm + s * STAGE;
          const int t0 = (int)(p.first + blk) * BT;
          mbar_arrive_expect_tx(&full[s], STAGE);
#pragma unroll
          for (int i = 0; i < DK / 64; ++i) {
            tma_load_3d(st + i * BOX, &tmK, &full[s], g * DK + i * 64, t0, b);
            tma_load_3d(st + ROWS_BYTES + i * BOX, &tmQ, &full[s], g * DK + i * 64, t0, b);
          }
          tma_load_3d(st + 2 * ROWS_BYTES, &tmV, &full[s], h * dv + c0, t0, b);            // (columns behind the head's own are multiplied and not read)
          bulk(st + 2 * ROWS_BYTES + V_BYTES, blocks + (int64_t)blk * BLOCK_BYTES, BLOCK_BYTES, &full[s]);
        }
        // every copy has landed before this thread ends
        for (int i = max(0, blk - 2); i < blk; ++i) wait_to_end(&full[i & 1], (i >> 1) & 1, p.waits);
      }
    } else if (warp == MMA_WARP) {
      // ================================================ products, issued by one lane of a converged warp, in small loops
      const uint32_t lead = elect_one();
      constexpr uint32_t id64 = umma_idesc_bf16(MMA_M, BT), id_mn = umma_idesc_bf16(MMA_M, 64) | (1u << 16);
#pragma unroll 1
      for (int blk = 0; blk < n_blocks && ok; ++blk) {
        const uint32_t ph = blk & 1, base = smem_u32(sm + ph * STAGE);
        // (descriptors' low words; the high ones do not change)
        const uint32_t kd = (uint32_t)umma_desc_k_sw128(base), qd = (uint32_t)umma_desc_k_sw128(base + ROWS_BYTES), td = (uint32_t)desc_tri(base + 2 * ROWS_BYTES + V_BYTES);
        constexpr uint32_t ROWS_HI = (uint32_t)(1024 >> 4) | 1u << 14 | 2u << 29, TRI_HI = (uint32_t)(256 >> 4) | 1u << 14;
        // half of K S or Q S, the small parts first
        const auto state_times = [&](uint32_t d, uint32_t rows, int hf, bool add) {
          const uint32_t at = tmem + T::S + hf * T::S_HALF, from = rows + hf * (DK == 128 ? BOX >> 4 : 4);
#pragma unroll
          for (int s = 2; s >= 0; --s)
#pragma unroll
            for (int i = 0; i < DK / 32; ++i) {
              const int col = s * (HC / 2) + i * 8;
              if (s < 2 || i > 0) product<true>(lead, d, at + col, from + i * 2, ROWS_HI, id64);
              else if (add) product<true>(lead, d, at + col, from + i * 2, ROWS_HI, id64);
              else product<false>(lead, d, at + col, from + i * 2, ROWS_HI, id64);
            }
        };
        // sums over a triangle: parts (0, 2) (2, 0) (1, 1) (0, 1) (1, 0) (0, 0), the small products first
        const auto tri_times = [&](uint32_t d, uint32_t tri) {
          constexpr int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
          for (int m = 0; m < 6; ++m)
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
              const uint32_t a = tmem + T::WP + pa[m] * 32 + kt * 8, from = tri + (pb[m] * TILES * PART_BYTES + tile_index(kt, 2 * kt) * PART_BYTES) / 16;
              if (m || kt) product<true>(lead, d + 16 * kt, a, from, TRI_HI, umma_idesc_bf16(MMA_M, BT - 16 * kt));
              else product<false>(lead, d, a, from, TRI_HI, umma_idesc_bf16(MMA_M, BT));
            }
        };
        ok = wait(&s_ready, ph);
        if (!ok) break;
        tc_fence_after();
        state_times(tmem + T::W, kd, 0, false);
        state_times(tmem + T::W, kd, 1, true);
        if (lead) umma_commit(&w_done);
        ok = wait(&wp_ready, ph);
        if (!ok) break;
        tc_fence_after();
        tri_times(tmem + T::W, td);
        if (lead) umma_commit(&u_done);
        // Q S fills the time in which U is split, P U that of the state
        if (blk) { ok = wait(&o_free, (blk - 1) & 1); if (!ok) break; tc_fence_after(); }
        state_times(tmem + T::O, qd, 0, false);
        state_times(tmem + T::O, qd, 1, true);
        if (lead) umma_commit(&qs_done[ph]);
        ok = wait(&up_ready, ph);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int hf = 0; hf < DK / 64; ++hf) {
#pragma unroll
          for (int s = 2; s >= 0; --s)
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
              const uint32_t d = tmem + T::DS + hf * T::DS_HALF, a = tmem + T::UP + s * 32 + kt * 8, from = kd + hf * (BOX >> 4) + kt * (16 * 128 >> 4);
              if (s < 2 || kt) product<true>(lead, d, a, from, ROWS_HI, id_mn);
              else product<false>(lead, d, a, from, ROWS_HI, id_mn);
            }
          if (lead) umma_commit(&ds_done[hf]);
        }
        if (DK == 64 && lead) umma_commit(&ds_done[1]);
        // (the next block's copies are looked for here, off the chain from the state's parts to the next products)
        ok = wait(&pu_ready, ph);
        if (!ok) break;
        tc_fence_after();
        tri_times(tmem + T::O, td + TRI_BYTES / 16);
        if (lead) { umma_commit(&o_done[ph]); umma_commit(&empty[ph]); }
      }
      if (lead) umma_commit(&ended);                     // every product has been summed before TMEM is given back
      wait_to_end(&ended, 0, p.waits);
    }
    __syncwarp();
    __syncthreads_or(!ok);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc<1>(tmem, 512);
  if (p.pair) { __syncwarp(); cluster_sync_all(); }      // the other CTA may still write its sums here
}

// ------------------------------------------------------------------------------------------------ a call of one block, on more CTAs than the chip takes at once
// delta_scan_kernel is alone on its SM, so that nothing covers what surrounds a block there: its copies, the state's way in and out, the start of the next CTA, 5 of 8 us.  Here a warp has 16
// value channels (again the rows of the products, on mma.sync: the sums of one are, lane by lane, the first operand of the next, and warps exchange nothing) and two to eight warps make a CTA,
// several of which share an SM; the state is in registers, the read-outs are left to a norm of their own.  single() says where it is taken.
template <int DK>
__global__ void __launch_bounds__(256, 1) delta_single_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmV, const Args p) {
  pdl_wait();
  constexpr int KT = DK / 16, BOX = BT * 128, ROWS_BYTES = DK / 64 * BOX;      // keys and queries: boxes of 64 columns, 16-byte pieces of a row swizzled by row & 7
  extern __shared__ __align__(16) uint8_t sm_raw[];
  uint8_t* ks = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t arrived;
  const int nw = blockDim.x >> 5, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int vpitch = nw * 32, h = blockIdx.x, b = blockIdx.y, dv = p.dv, nt = (int)p.L;
  const int c0 = blockIdx.z * nw * 16, cw = c0 + warp * 16;            // the CTA's and the warp's first value channel
  const uint8_t* qs = ks + ROWS_BYTES;
  const uint8_t* vs = qs + ROWS_BYTES;
  const uint8_t* tri = vs + BT * vpitch;
  const float* vec = reinterpret_cast<const float*>(tri + 2 * TRI_BYTES);
  if (tid == 0) {
    mbar_init(&arrived, 1);
    fence_barrier_init();
    const int g = h / (p.H / p.G);
    mbar_arrive_expect_tx(&arrived, 2 * ROWS_BYTES + BT * vpitch + BLOCK_BYTES);       // (rows behind the last token arrive as zeros)
#pragma unroll
    for (int i = 0; i < DK / 64; ++i) {
      tma_load_3d(ks + i * BOX, &tmK, &arrived, g * DK + i * 64, 0, b);
      tma_load_3d(ks + ROWS_BYTES + i * BOX, &tmQ, &arrived, g * DK + i * 64, 0, b);
    }
    tma_load_3d(ks + 2 * ROWS_BYTES, &tmV, &arrived, h * dv + c0, 0, b);
    bulk(ks + 2 * ROWS_BYTES + BT * vpitch, p.blocks + ((int64_t)b * p.H + h) * (int64_t)BLOCK_BYTES, BLOCK_BYTES, &arrived);
  }
  // ---- S^T: rows = value channels cw + gq (+ 8), columns = state rows: S[n][..] covers state rows 8 n + 2 tq, + 1
  float S[2 * KT][4];
  float* Sg = p.state + ((int64_t)b * p.H + h) * DK * (int64_t)dv;
  const bool live = cw < dv;                                            // (dv is a multiple of 16)
#pragma unroll
  for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[n][e] = (p.zero_start || !live) ? 0.f : Sg[(int64_t)(8 * n + 2 * tq + (e & 1)) * dv + cw + gq + (e >> 1) * 8];
  __syncthreads();
  if (__syncthreads_or(!wait_or_give_up(&arrived, 0, p.waits))) {
    if (tid == 0) wait_to_end(&arrived, 0, p.waits);                    // no state is kept; the copies under way land before the CTA ends
    return;
  }
  if (!live) return;
  float* yr = p.y + (int64_t)b * p.L * p.H * dv + (int64_t)h * dv + cw + gq;
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
        W[n][0] = fmaf(gk.x, W[n][0], bf_lo(v[2 * u])); W[n][1] = fmaf(gk.y, W[n][1], bf_hi(v[2 * u]));
        W[n][2] = fmaf(gk.x, W[n][2], bf_lo(v[2 * u + 1])); W[n][3] = fmaf(gk.y, W[n][3], bf_hi(v[2 * u + 1]));
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
            for (int s = 0; s < 3; ++s) {
              const uint32_t* part = reinterpret_cast<const uint32_t*>(base + (s * TILES + tile_index(kt, n0 + c)) * PART_BYTES) + lane;
              t[c][s] = make_uint2(part[0], part[32]);
            }
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
  if (p.store_state) {
#pragma unroll
    for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) Sg[(int64_t)(8 * n + 2 * tq + (e & 1)) * dv + cw + gq + (e >> 1) * 8] = S[n][e];
  }
}
constexpr int single_smem_bytes(int dk, int warps) { return 1024 + 2 * BT * dk * 2 + BT * warps * 32 + BLOCK_BYTES; }

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

// From how many tokens on the blocks are taken.  A call of one block takes 22 us (8 pairs of head and sequence, 64 x 64) to 290 (2048 pairs of 128 x 128), nearly whatever its number of tokens;
// token by token it takes 0.6 to 1.2 us per token while the pairs fit the SMs, in proportion to their number beyond.  Measured (us, cold L2, token by token / blocks):
//   64 x 64, 8 to 128 pairs: 16 tokens 18 / 23, 24 tokens 25 / 23, 32 tokens 31 / 23, 47 tokens 41 / 23;  128 x 128, 32 pairs: 16: 25 / 29, 32: 39 / 30;  128 pairs: 24: 37 / 38, 32: 41 / 40,
//   47: 55 / 40;  64 x 128, 128 pairs: 24: 29 / 32, 32: 33 / 32, 47: 43 / 34
//   512 pairs, where token by token has more than a wave: 64 x 64: 16: 39 / 48, 32: 65 / 48;  128 x 128: 16: 84 / 81, 32: 141 / 85;  2048 pairs of 128 x 128: 32: 479 / 261
//   few value channels, whose token-by-token CTAs are nearly empty: 128 x 16, 32 pairs: 16: 37 / 28;  1024 pairs: 24: 66 / 73, 32: 82 / 77, 47: 117 / 83;  64 x 16, 1024 pairs: 32: 70 / 67
// The lines are those of the blocks' former kernels, which were slower: by these figures the blocks could be taken from 32 tokens on throughout.  What lies between would then be rounded elsewhere.
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
  // The read-outs' place is asked for in any case, so that a call takes the workspace it always took.  Where the scan norms them itself (up to 128 channels, more than one block) it is left alone.
  s.y = up(sizeof(float) * (size_t)p->B * p->L * p->H * p->dv);
  s.tri = up((size_t)BLOCK_BYTES * s.slab * p->B * p->H);
  s.state = p->state || s.slab == s.blocks ? 0 : up(sizeof(float) * (size_t)p->B * p->H * p->dk * p->dv);
  return s;
}

// One block, and so many CTAs of the scan (64 channels) that they take more than a wave: delta_single_kernel.  Measured, 64 tokens with a state (us, scan launched dependent / single):
//   64 x 32, 160 pairs: 31.6 / 27.6, 1024: 85 / 62;  128 x 32, 160: 35.9 / 33.8, 1024: 101 / 77;  (read-outs of more than 128 channels need a norm of their own in any case) 64 x 192, 64: 37.9 /
//   33.8, 512: 124 / 101;  128 x 192, 64: 44 / 40;  else only from more waves on: 64 x 128, 128: 33.8 / 33.9, 256: 52 / 46, 1024: 159 / 124;  128 x 128, 160: 48 / 54, 256: 60 / 54, 1024: 185 /
//   159;  64 x 16, 160: 29.7 / 31.8, 512: 49 / 48.  Heads of 48 and 64 channels fill the scan's lanes and stay there (64 x 64, 512: 50 / 58, 2048: 161 / 163).
bool single(const evo_gated_delta_params* p, const Sizes& s) {
  const int64_t ctas = (int64_t)p->B * p->H * ((p->dv + CH - 1) / CH), sms = device_sm_count();
  if (s.blocks > 1 || (p->dv > 32 && p->dv <= 64)) return false;
  return 2 * ctas > (p->dv > 128 || p->dv == 32 ? 2 * sms : 5 * sms);
}

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
  a.gate = (const bf16*)p->gate; a.norm_w = (const bf16*)p->norm_w; a.out = (bf16*)p->out; a.ldo = p->ldo; a.eps = p->eps;
  const bool one = single(p, s);
  a.norm = !one && p->dv <= 2 * CH; a.pair = a.norm && p->dv > CH;
  a.wide = p->ldz % 4 == 0 && p->ldo % 4 == 0 && (((uintptr_t)p->gate | (uintptr_t)p->out) & 7) == 0;
  constexpr int prep_smem = prepare_smem_bytes(DK), scan_smem = scan_smem_bytes(DK);
  CUtensorMap tmK, tmQ, tmV;
  const uint64_t kdims[3] = {(uint64_t)p->G * DK, (uint64_t)p->L, (uint64_t)p->B}, vdims[3] = {(uint64_t)p->H * p->dv, (uint64_t)p->L, (uint64_t)p->B};
  const uint64_t strides[2] = {(uint64_t)p->ld * 2, (uint64_t)p->L * p->ld * 2};
  // delta_single_kernel: two warps (32 channels) to eight per CTA, as few as fill the chip
  int nw = 2;
  while (nw < 8 && nw * 16 < p->dv && (int64_t)p->B * p->H * (p->dv / 16) > (int64_t)nw * device_sm_count()) nw *= 2;
  const uint32_t kbox[3] = {64, BT, 1}, vbox[3] = {one ? (uint32_t)nw * 16 : CH, BT, 1};
  int rc;
  if ((rc = make_tmap_nd_bf16(&tmK, p->k, 3, kdims, strides, kbox, true)) || (rc = make_tmap_nd_bf16(&tmQ, p->q, 3, kdims, strides, kbox, true)) ||
      (rc = make_tmap_nd_bf16(&tmV, p->v, 3, vdims, strides, vbox, !one))) return rc;
  static unsigned long long done_prep = 0, done_scan = 0, done_single = 0;
  if ((rc = ensure_dyn_smem(delta_prepare_kernel<DK>, prep_smem, done_prep)) || (rc = ensure_dyn_smem(delta_scan_kernel<DK>, scan_smem, done_scan)) ||
      (rc = ensure_dyn_smem(delta_single_kernel<DK>, single_smem_bytes(DK, 8), done_single))) return rc;
  for (int64_t first = 0; first < s.blocks; first += s.slab) {
    a.first = first; a.n_blocks = (int)std::min<int64_t>(s.slab, s.blocks - first);
    a.zero_start = first == 0 && (p->zero_start || !p->state);
    a.store_state = p->state || s.state;
    EVO_CUDA(launch_dependent(delta_prepare_kernel<DK>, dim3(a.n_blocks, a.H, a.B), dim3(128), prep_smem, st, a));
    if ((rc = check_launch("evo_gated_delta_fwd(prepare)"))) return rc;
    if (one) {
      EVO_CUDA(launch_dependent(delta_single_kernel<DK>, dim3(a.H, a.B, (a.dv / 16 + nw - 1) / nw), dim3(nw * 32), single_smem_bytes(DK, nw), st, tmK, tmQ, tmV, a));
      if ((rc = check_launch("evo_gated_delta_fwd(single)"))) return rc;
      break;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.H, a.B, (a.dv + CH - 1) / CH); cfg.blockDim = dim3(SCAN_THREADS); cfg.dynamicSmemBytes = scan_smem; cfg.stream = st;
    cudaLaunchAttribute attrs[2] = {};
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension; attrs[1].val.clusterDim = {1, 1, 2};
    // Launched dependent, the scan's CTAs are set up while the last of delta_prepare_kernel's run, which is worth 2 to 4 us: normal / dependent (us) 1 x 300 tokens, 8 heads of 64 x 64
    // 28.8 / 26.7, 1 x 777, 32 heads of 128 x 128 62.9 / 60.4, 1 x 4096 253 / 249.  But CTAs that come to most of the SMs one by one are placed worse: 64 pairs, 128 CTAs, 4 x 4096 tokens
    // 329 / 340, 4 x 1024 95 / 99; 128 pairs of 128 x 64 67.0 / 67.6.  For one or two blocks the early start is worth more than the place: 48 tokens, 128 pairs of 64 x 128 37.9 / 33.8,
    // 160 of 64 x 32 33.8 / 31.6; 128 tokens, 128 pairs of 128 x 128 50 / 48, 1024 249 / 245.
    const bool dependent = !pdl_off() && ((int64_t)cfg.gridDim.x * cfg.gridDim.y * cfg.gridDim.z * 2 <= device_sm_count() || s.blocks <= 2);
    cfg.attrs = dependent ? attrs : attrs + 1; cfg.numAttrs = (dependent ? 1 : 0) + (a.pair ? 1 : 0);
    EVO_CUDA(cudaLaunchKernelEx(&cfg, delta_scan_kernel<DK>, tmK, tmQ, tmV, a));
    if ((rc = check_launch("evo_gated_delta_fwd(scan)"))) return rc;
  }
  if (a.norm) return 0;
  const int64_t rows = (int64_t)p->B * p->L, w = rows * p->H;
  const bool wide = a.wide && ((uintptr_t)p->norm_w & 7) == 0;
  const auto norm = wide && p->dv == 128 ? delta_norm4_kernel<4> : (wide && p->dv == 32 ? delta_norm4_kernel<1> : delta_norm_kernel);
  const int per_cta = norm == delta_norm_kernel ? 8 : 32;
  norm<<<(unsigned)((w + per_cta - 1) / per_cta), 256, 0, st>>>(a.y, a.gate, p->ldz, a.norm_w, a.out, p->ldo, rows, p->H, p->dv, p->eps);
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
