// The usual windowed attention of a prompt -- one map, causal or with a window, optional sink, gate per head or channel, heads of 64 or 128 -- on the fifth-generation
// tensor cores (evo_window_attn_fwd; window_attention_mma.cu has the form for everything else).
//
// A CTA takes two tiles of 128 queries of one head, so that one tile's softmax runs while the tensor pipe works on the other's products:
//   warps 0-7, 8-15  softmax and epilogue of the tiles: query r <-> TMEM lane r, its keys' two halves with two threads that exchange their maxima through shared memory
//   warp  16         copies: both query tiles once, keys and values through two-deep rings that both tiles read
//   warp  17         the products, TMEM (the warps of its warpgroup give their registers to the softmax)
// A tile pair of 128 queries and 128 keys costs the tensor pipe 1536 cycles; 4 x 4096 queries, 16 heads of 128, window 1024, in a warm loop: 727 us in the mma.sync form, 335 with
// one thread per query and a single issuing thread (by clock stamps the softmax then waited for scores more than half of the time; its products in a loop of eight: 288), 260 with
// a converged issuing warp, 237 with two threads per query (without a window 1518 / 535 / 393 / 362; 16 heads, 300 tokens 31 / 23 / 22 / 20).  With cold L2 257 us.
// The scores (fp32, 128 columns of TMEM) are read once into registers; each probability goes back as a bf16 high part (columns 0-63 of its scores) plus a bf16 low part
// (64-127), and two products with the values add them up in fp32: relative error 2^-17 per weight, as in the mma.sync form.  The exponents' reference follows the
// running maximum lazily (weights stay below 2^8).  A key tile is counted from the first key that the first query tile sees, so the second tile's first key is a tile
// boundary too and both walk window/128 + 1 tiles.
//
// A masked probability is 0, and 0 x inf or 0 x NaN from a value that the row does not see would spoil the row (up to 127 tokens away).  A row whose sums are not finite
// although its denominator is, is therefore summed again over the keys that it sees alone, on the CUDA cores.
//
// Every wait has a limit; a role that gives up ends, and the CTA ends when its copies and products have.
#include "waits.cuh"
#include <algorithm>
#include "../../include/evo_b200.h"

using namespace evo;

namespace {

constexpr int BQ = 128, BKV = 128, KV_STAGES = 2, THREADS = 640;
constexpr int HALF_BYTES = 128 * 64 * 2;         // 128 rows of 64 channels: one copy, 128-byte swizzled rows
constexpr int WARPS = 16, HK = BKV / 2;         // softmax warps; keys of a tile per thread
// registers per thread: the launch's 96 shared out again, the softmax warps' from the other four's
constexpr int SOFTMAX_REGS = 112, OTHER_REGS = 32;
static_assert(WARPS * 32 * SOFTMAX_REGS + 128 * OTHER_REGS <= THREADS * 96, "register shares exceed the launch");
constexpr uint32_t TM_S = 0, TM_O = 256;         // + 128 * tile

struct Args {
  const bf16 *q, *k, *v, *gate, *sink;
  bf16* out;
  long long q_tok, k_tok, v_tok, k_batch, v_batch, gate_tok, ldo, Lq, pos;
  int B, H, G, n_qblk, window, gate_per_head, tail;
  float scale2;
  WaitLimit waits;
};

__device__ __forceinline__ float ex2(float x) { float y; asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// values as the second operand: rows are keys, 64-channel halves HALF_BYTES apart
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(HALF_BYTES >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
window_attn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const Args a) {
  constexpr int TILE_BYTES = BQ * HD * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sQ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);   // [2 tiles]
  uint8_t* sK = sQ + 2 * TILE_BYTES;                // [KV_STAGES]
  uint8_t* sV = sK + KV_STAGES * TILE_BYTES;        // [KV_STAGES]
  __shared__ uint64_t q_full[2], k_full[KV_STAGES], k_empty[KV_STAGES], v_full[KV_STAGES], v_empty[KV_STAGES], s_full[2], p_full[2], o_full[2], ended;
  __shared__ uint32_t tmem_slot;
  __shared__ float side[2][2][2 * BQ];               // [parity][half][tile, row]: a half's maximum, in the end its sum

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (head, sequence) by (head, sequence), the last queries first; the last `tail` of them together, the pairs with the most keys of all first (see the launcher)
  const int pairs = (a.n_qblk + 1) / 2, bulk = (a.B * a.H - a.tail) * pairs, at = (int)blockIdx.x;
  const int pair = pairs - 1 - (at < bulk ? at % pairs : (at - bulk) / a.tail), hb = at < bulk ? at / pairs : a.B * a.H - a.tail + (at - bulk) % a.tail;
  const int h = hb % a.H, b = hb / a.H, g = h / (a.H / a.G);
  const int win = a.window > 0 ? a.window : 1 << 30;
  // keys and queries are counted from the first key that the first tile sees
  const long long rel0 = (long long)pair * 2 * BQ, key0 = a.window > 0 ? max(0ll, a.pos + rel0 - a.window + 1) : 0ll;
  const int row0 = (int)(a.pos + rel0 - key0);       // the first tile's first query
  int j0[2], j1[2];                                  // key tiles of the two query tiles
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int live = (int)min((long long)BQ, a.Lq - rel0 - t * BQ);                  // queries of the tile
    j0[t] = j1[t] = 0;
    if (live > 0) {
      j0[t] = max(0, row0 + t * BQ - win + 1) / BKV;
      j1[t] = (row0 + t * BQ + live - 1) / BKV + 1;
    }
  }
  const int n_kv = max(j1[0], j1[1]);

  if (warp == WARPS && lane == 0) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
  if (warp == WARPS + 1 && lane == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 256); mbar_init(&o_full[i], 1); }
    for (int i = 0; i < KV_STAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(&ended, 1);
    fence_barrier_init();
  }
  if (warp == WARPS + 1) { __syncwarp(); tmem_alloc<1>(&tmem_slot, 512); tmem_relinquish<1>(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();              // launched dependent: nothing in front of this touches what a kernel before may write or read

  if (warp >= WARPS) {
    regs_down<OTHER_REGS>();
    if (warp == WARPS) {
      if (lane == 0) {
        const auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int head, long long tok) {
          mbar_arrive_expect_tx(bar, TILE_BYTES);
#pragma unroll
          for (int c = 0; c < HD; c += 64) tma_load_4d(dst + c / 64 * HALF_BYTES, map, bar, c, head, (int)tok, b);
        };
        load(sQ, &tmQ, &q_full[0], h, rel0);
        if (j1[1] > 0) load(sQ + TILE_BYTES, &tmQ, &q_full[1], h, rel0 + BQ);
        int kn = 0, vn = 0;                            // tiles asked for
        for (int j = 0; j < n_kv; ++j) {
          const int st = j % KV_STAGES;
          const uint32_t ph = (uint32_t)(j / KV_STAGES) & 1;
          if (!wait_or_give_up(&k_empty[st], ph ^ 1, a.waits)) break;
          load(sK + st * TILE_BYTES, &tmK, &k_full[st], g, key0 + (long long)j * BKV);
          ++kn;
          if (!wait_or_give_up(&v_empty[st], ph ^ 1, a.waits)) break;
          load(sV + st * TILE_BYTES, &tmV, &v_full[st], g, key0 + (long long)j * BKV);
          ++vn;
        }
        // every copy has landed before this thread ends
        wait_to_end(&q_full[0], 0, a.waits);
        if (j1[1] > 0) wait_to_end(&q_full[1], 0, a.waits);
        for (int j = max(0, kn - KV_STAGES); j < kn; ++j) wait_to_end(&k_full[j % KV_STAGES], (uint32_t)(j / KV_STAGES) & 1, a.waits);
        for (int j = max(0, vn - KV_STAGES); j < vn; ++j) wait_to_end(&v_full[j % KV_STAGES], (uint32_t)(j / KV_STAGES) & 1, a.waits);
      }
    } else if (warp == WARPS + 1) {
      // one copy of each product, in a small loop (see above)
      constexpr uint32_t idesc_qk = umma_idesc_bf16(BQ, BKV);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(BQ, HD) | (1u << 16);     // the values are MN-major
      const uint64_t q_desc = umma_desc_k_sw128(smem_u32(sQ)), k_desc = umma_desc_k_sw128(smem_u32(sK)), v_desc = desc_mn_sw128(smem_u32(sV));
      const uint32_t lead = elect_one();
      bool ok = true;
#pragma unroll 1
      for (int j = -1; j < n_kv && ok; ++j) {
#pragma unroll 1
        for (int t = 0; t < 2; ++t) {
          const int first = t ? j0[1] : j0[0], last = t ? j1[1] : j1[0];      // of the tile's key tiles, exclusive
          const uint32_t s_tm = tmem_base + TM_S + t * BKV, o_tm = tmem_base + TM_O + t * 128;
          if (j >= first && j < last) {
            const int st = j % KV_STAGES;
            ok = wait_or_give_up(&v_full[st], (uint32_t)(j / KV_STAGES) & 1, a.waits) && wait_or_give_up(&p_full[t], (uint32_t)(j - first) & 1, a.waits);
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = v_desc + st * (TILE_BYTES >> 4);
#pragma unroll 1
            for (int part = 0; part < 2; ++part)                              // high parts, then low parts
#pragma unroll 8
              for (int kk = 0; kk < BKV / 16; ++kk)
                umma_ts_if(lead, o_tm, s_tm + part * (BKV / 2) + kk * 8, vd + kk * (16 * 128 >> 4), idesc_pv, j != first || part != 0 || kk != 0);
            if (lead && (t == 1 || !(j >= j0[1] && j < j1[1]))) umma_commit(&v_empty[st]);
            if (lead && j == last - 1) umma_commit(&o_full[t]);
          }
          if (j + 1 >= first && j + 1 < last) {
            const int st = (j + 1) % KV_STAGES;
            ok = (j + 1 != first || wait_or_give_up(&q_full[t], 0, a.waits)) && wait_or_give_up(&k_full[st], (uint32_t)((j + 1) / KV_STAGES) & 1, a.waits);
            if (!ok) break;
            tc_fence_after();
            const uint64_t qd = q_desc + t * (TILE_BYTES >> 4), kd = k_desc + st * (TILE_BYTES >> 4);
#pragma unroll 8
            for (int kk = 0; kk < HD / 16; ++kk) {
              const int off = (kk >> 2) * (HALF_BYTES >> 4) + (kk & 3) * 2;
              umma_ss_if(lead, s_tm, qd + off, kd + off, idesc_qk, kk != 0);
            }
            if (lead && (t == 1 || !(j + 1 >= j0[1] && j + 1 < j1[1]))) umma_commit(&k_empty[st]);
            if (lead) umma_commit(&s_full[t]);
          }
        }
      }
      if (lead) umma_commit(&ended);                 // every product has been summed before TMEM is given back
      wait_to_end(&ended, 0, a.waits);
    }
  } else {
    regs_up<SOFTMAX_REGS>();
    const int t = warp >> 3, half = warp >> 2 & 1, w = warp & 3;       // a row's two threads are four warps apart and meet at a barrier of their own
    if (j1[t] > 0) {
      const int r = w * 32 + lane, row = row0 + t * BQ + r;
      const uint32_t lane_addr = tmem_base + ((uint32_t)(w * 32) << 16);
      const uint32_t s_addr = lane_addr + TM_S + t * BKV, o_addr = lane_addr + TM_O + t * 128 + half * (HD / 2);
      const auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + w) : "memory"); };
      float m = -INFINITY, l = 0.f;                  // the exponents' reference (-inf: no key yet), the sum of this half's weights
      bool ok = true;
      for (int j = j0[t]; j < j1[t]; ++j) {
        // a wait that runs out ends both halves: the maximum's place says so
        ok = __all_sync(0xffffffffu, wait_or_give_up(&s_full[t], (uint32_t)(j - j0[t]) & 1, a.waits));
        tc_fence_after();
        const int key = j * BKV + half * HK, top_row = row0 + t * BQ + w * 32 + 31;
        const bool some = ok && key <= top_row && top_row - 31 - (key + HK - 1) < win;      // does any row of the warp see any key of the half
        float sc[HK], mx = -INFINITY;
        if (some) {
          {
            uint32_t t0[32], t1[32];
            tmem_ld_32x32(s_addr + half * HK, t0); tmem_ld_32x32(s_addr + half * HK + 32, t1);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) { sc[i] = __uint_as_float(t0[i]); sc[32 + i] = __uint_as_float(t1[i]); }
          }
          const int d0 = row - key;                  // the distance to the half's first key
          if (d0 < HK - 1 || d0 >= win) {
#pragma unroll
            for (int i = 0; i < HK; ++i) if ((unsigned)(d0 - i) >= (unsigned)win) sc[i] = -INFINITY;
          }
          float mxs[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) mxs[i] = fmaxf(sc[i], sc[4 + i]);
#pragma unroll
          for (int i = 8; i < HK; i += 8)
#pragma unroll
            for (int c = 0; c < 4; ++c) mxs[c] = fmaxf(mxs[c], fmaxf(sc[i + c], sc[i + 4 + c]));
          mx = fmaxf(fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * a.scale2, -INFINITY);      // (a number in any case)
        }
        const int par = (j - j0[t]) & 1, mine = t * BQ + r;
        side[par][half][mine] = ok ? mx : __int_as_float(0x7fc00000);
        meet();                                      // both halves have their scores in registers now: the columns may be written
        const float other = side[par][half ^ 1][mine];
        if (!__all_sync(0xffffffffu, ok && other == other)) { ok = false; break; }
        mx = fmaxf(mx, other);
        const bool grow = mx > m + 8.f;              // also true for a row's first keys
        float alpha = 1.f;
        if (grow) { alpha = m == -INFINITY ? 0.f : ex2(m - mx); m = mx; l *= alpha; }
        // the scores are there, so the sums with the last tile's values are too: they were asked for before
        if (j > j0[t] && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
          for (int c = 0; c < HD / 2; c += 32) {
            uint32_t tt[32];
            tmem_ld_32x32(o_addr + c, tt);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) tt[i] = __float_as_uint(__uint_as_float(tt[i]) * alpha);
            tmem_st_32x32(o_addr + c, tt);
          }
        }
        const uint32_t p_addr = s_addr + half * (HK / 2);
        if (some) {
          const float ref = m == -INFINITY ? 0.f : m;
          const float2 scale2 = make_float2(a.scale2, a.scale2), ref2 = make_float2(-ref, -ref);
          float2 la = make_float2(0.f, 0.f), lb = la;
#pragma unroll
          for (int c = 0; c < HK; c += 16) {
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 x = __ffma2_rn(make_float2(sc[c + 2 * i], sc[c + 2 * i + 1]), scale2, ref2);
              const float2 p = make_float2(ex2(x.x), ex2(x.y));
              if (i & 1) lb = __fadd2_rn(lb, p); else la = __fadd2_rn(la, p);
              hi[i] = pack_bf16(p.x, p.y);
              const float2 rest = __fadd2_rn(p, make_float2(-bf_lo(hi[i]), -bf_hi(hi[i])));
              lo[i] = pack_bf16(rest.x, rest.y);
            }
            tmem_st_x8(p_addr + c / 2, hi);
            tmem_st_x8(p_addr + BKV / 2 + c / 2, lo);
          }
          l += (la.x + lb.x) + (la.y + lb.y);
        } else {
          const uint32_t zero[8] = {};
#pragma unroll
          for (int c = 0; c < HK; c += 16) { tmem_st_x8(p_addr + c / 2, zero); tmem_st_x8(p_addr + BKV / 2 + c / 2, zero); }
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&p_full[t]);
      }
      const int par = (j1[t] - j0[t]) & 1, mine = t * BQ + r;
      if (ok) {                                      // the same in both halves; the place was last read for the last tile but one
        side[par][half][mine] = l;
        meet();
        l = side[par][0][mine] + side[par][1][mine];
        ok = __all_sync(0xffffffffu, wait_or_give_up(&o_full[t], 0, a.waits));
      }
      if (ok) {
        tc_fence_after();
        const long long rel = rel0 + t * BQ + r, orow = (long long)b * a.Lq + rel;
        const bool live = rel < a.Lq;
        float mul = 1.f / l;
        if (a.sink) {                                // e^sink joins the denominator
          const float sk = __bfloat162float(a.sink[h]) * 1.4426950408889634f, top = fmaxf(m, sk), num = ex2(m - top);
          mul = num / fmaf(l, num, ex2(sk - top));
        }
        const bf16* grow = a.gate && live ? a.gate + orow * a.gate_tok + (a.gate_per_head ? h : (long long)h * HD + half * (HD / 2)) : nullptr;
        if (grow && a.gate_per_head) mul *= 1.f / (1.f + expf(-__bfloat162float(*grow)));
        const bool chan = grow && !a.gate_per_head;
        bf16* dst = a.out + orow * a.ldo + (long long)h * HD + half * (HD / 2);
        float odd = 0.f;
#pragma unroll 1
        for (int c = 0; c < HD / 2; c += 32) {
          uint32_t tt[32];
          tmem_ld_32x32(o_addr + c, tt);
          uint4 gw[4] = {};
          if (chan) {
#pragma unroll
            for (int i = 0; i < 4; ++i) gw[i] = reinterpret_cast<const uint4*>(grow + c)[i];
          }
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t gp[4] = {gw[i].x, gw[i].y, gw[i].z, gw[i].w};
            uint32_t ow[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float x = __uint_as_float(tt[8 * i + 2 * e]), y = __uint_as_float(tt[8 * i + 2 * e + 1]);
              odd = fmaf(x, 0.f, fmaf(y, 0.f, odd));
              x *= mul; y *= mul;
              if (chan) { x *= __fdividef(1.f, 1.f + __expf(-bf_lo(gp[e]))); y *= __fdividef(1.f, 1.f + __expf(-bf_hi(gp[e]))); }
              ow[e] = pack_bf16(x, y);
            }
            if (live) reinterpret_cast<uint4*>(dst + c)[i] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
          }
        }
        if (live && h == a.H - 1 && half)
          for (long long c = (long long)a.H * HD; c < a.ldo; ++c) a.out[orow * a.ldo + c] = __float2bfloat16_rn(0.f);
        // rows to be summed again over the keys that they see: a warp takes them one by one, a lane QC channels of the scores and CH of its half's sums
        __syncwarp();
        for (unsigned todo = __ballot_sync(0xffffffffu, live && odd != odd && l == l); todo; todo &= todo - 1) {
          const int src = __ffs(todo) - 1;
          constexpr int QC = HD / 32, CH = HD / 64;
          const float mr = __shfl_sync(0xffffffffu, m == -INFINITY ? 0.f : m, src), mulr = __shfl_sync(0xffffffffu, mul, src);
          const long long relr = rel0 + t * BQ + w * 32 + src, last = a.pos + relr, first = a.window > 0 ? max(0ll, last - a.window + 1) : 0ll;
          const long long row_out = (long long)b * a.Lq + relr, ch0 = (long long)half * (HD / 2) + lane * CH;
          const bf16* qp = a.q + row_out * a.q_tok + (long long)h * HD + lane * QC;
          float qv[QC], o[CH];
#pragma unroll
          for (int c = 0; c < QC; ++c) qv[c] = __bfloat162float(qp[c]);
#pragma unroll
          for (int c = 0; c < CH; ++c) o[c] = 0.f;
#pragma unroll 1
          for (long long key = first; key <= last; ++key) {
            const bf16* kp = a.k + (long long)b * a.k_batch + key * a.k_tok + (long long)g * HD + lane * QC;
            const bf16* vp = a.v + (long long)b * a.v_batch + key * a.v_tok + (long long)g * HD + ch0;
            float s = 0.f;
#pragma unroll
            for (int c = 0; c < QC; ++c) s = fmaf(qv[c], __bfloat162float(kp[c]), s);
#pragma unroll
            for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
            const float p = ex2(fmaf(s, a.scale2, -mr));
#pragma unroll
            for (int c = 0; c < CH; ++c) o[c] = fmaf(p, __bfloat162float(vp[c]), o[c]);
          }
          const bf16* gr = a.gate && !a.gate_per_head ? a.gate + row_out * a.gate_tok + (long long)h * HD + ch0 : nullptr;
          bf16* op = a.out + row_out * a.ldo + (long long)h * HD + ch0;
#pragma unroll
          for (int c = 0; c < CH; ++c) op[c] = __float2bfloat16_rn(o[c] * mulr * (gr ? __fdividef(1.f, 1.f + __expf(-__bfloat162float(gr[c]))) : 1.f));
        }
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == WARPS + 1) tmem_dealloc<1>(tmem_base, 512);
}

template <int HD>
int launch(const evo_window_attn_params* p, cudaStream_t st) {
  Args a;
  a.q = (const bf16*)p->q; a.k = (const bf16*)p->k; a.v = (const bf16*)p->v; a.gate = (const bf16*)p->gate; a.sink = (const bf16*)p->sink; a.out = (bf16*)p->out;
  a.q_tok = p->q_tok_stride; a.k_tok = p->k_tok_stride; a.v_tok = p->v_tok_stride; a.k_batch = p->k_batch_stride; a.v_batch = p->v_batch_stride;
  a.gate_tok = p->gate_tok_stride; a.ldo = p->ldo; a.Lq = p->Lq; a.pos = p->q_pos0;
  a.B = p->B; a.H = p->H; a.G = p->G; a.n_qblk = (int)((p->Lq + BQ - 1) / BQ); a.gate_per_head = p->gate_per_head;
  a.window = p->window > 0 ? (int)std::min<int64_t>(p->window, 1 << 30) : 0;
  a.scale2 = p->scale * 1.4426950408889634f;
  if (const int rc_ = wait_limit(&a.waits)) return rc_;
  const int64_t heads = (int64_t)p->B * p->H, pairs = (a.n_qblk + 1) / 2, Lk = p->q_pos0 + p->Lq;
  // without a window the last heads' longest blocks would start when everything else is done: as many heads as keep their keys and values in half the L2 go together
  a.tail = p->window > 0 ? 1 : (int)std::min<int64_t>(heads, std::max<int64_t>(1, (64ll << 20) / (Lk * 4 * HD)));
  EVO_REQUIRE(heads * pairs < (1ll << 31), "evo_window_attn_fwd: too many blocks");
  CUtensorMap tmQ, tmK, tmV;
  const uint32_t box[4] = {64, 1, 128, 1};
  const uint64_t qd[4] = {(uint64_t)HD, (uint64_t)p->H, (uint64_t)p->Lq, (uint64_t)p->B}, kd[4] = {(uint64_t)HD, (uint64_t)p->G, (uint64_t)Lk, (uint64_t)p->B};
  const auto strides = [&](uint64_t (&s)[3], int64_t tok, int64_t batch, int64_t rows) {
    s[0] = HD * 2; s[1] = (uint64_t)tok * 2; s[2] = (uint64_t)(p->B > 1 ? batch : tok * rows) * 2;
  };
  uint64_t s[3];
  int rc;
  strides(s, p->q_tok_stride, p->Lq * p->q_tok_stride, p->Lq);
  if ((rc = make_tmap_nd_bf16(&tmQ, p->q, 4, qd, s, box, true))) return rc;
  strides(s, p->k_tok_stride, p->k_batch_stride, Lk);
  if ((rc = make_tmap_nd_bf16(&tmK, p->k, 4, kd, s, box, true))) return rc;
  strides(s, p->v_tok_stride, p->v_batch_stride, Lk);
  if ((rc = make_tmap_nd_bf16(&tmV, p->v, 4, kd, s, box, true))) return rc;
  constexpr int smem = BQ * HD * 2 * (2 + 2 * KV_STAGES) + 1024;
  static unsigned long long done = 0;
  if ((rc = ensure_dyn_smem(window_attn_tc_kernel<HD>, smem, done))) return rc;
  EVO_CUDA(launch_dependent(window_attn_tc_kernel<HD>, dim3((unsigned)(heads * pairs)), dim3(THREADS), smem, st, tmQ, tmK, tmV, a));
  return check_launch("evo_window_attn_fwd");
}

}  // namespace

namespace evo {

// 16 query rows or more, the host knows the position (the maps' extents), and every row of every operand starts on 16 bytes.  Fewer rows -- a step, the rest of a
// portion -- go to the CUDA-core kernels, which keep their weights and gate in fp32, spread up to four queries' keys over the warps of a CTA, and also serve the captured
// step: a call's result must not depend on where its position is kept.  One query behind 1000 keys, window 256, 16 heads of 128: 10.6 us there, 14.6 here; behind 4000 without
// a window 65.7 / 74.  (5 to 15 queries behind 1000 keys take 195 us there and 26 here, with 2e-3 of the bf16 results rounded to the other side instead of 3e-4.)
bool window_attn_tc_takes(const evo_window_attn_params* p) {
  if (p->Lq < 16) return false;
  const auto a16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
  const auto tok = [](int64_t s) { return s > 0 && s % 8 == 0 && s < (1ll << 31); };
  const auto batch = [&](int64_t s) { return p->B == 1 || (s > 0 && s % 8 == 0 && s < (1ll << 38)); };
  if (p->dtype != 0 || p->n_maps != 1 || p->dk != p->dv || (p->dk != 64 && p->dk != 128) || p->pos_dev || p->q_pos0 < 0 || p->q_pos0 + p->Lq >= (1 << 30)) return false;
  if (p->keep_first > 0 || p->pool > 0 || p->softcap > 0.f || p->dist_r1 || p->head_norm || !(p->scale > 0.f)) return false;
  if (!tok(p->q_tok_stride) || !tok(p->k_tok_stride) || !tok(p->v_tok_stride) || !batch(p->k_batch_stride) || !batch(p->v_batch_stride)) return false;
  if (p->Lq * p->q_tok_stride >= (1ll << 38) || (p->q_pos0 + p->Lq) * std::max(p->k_tok_stride, p->v_tok_stride) >= (1ll << 38)) return false;
  if (!a16(p->q) || !a16(p->k) || !a16(p->v) || !a16(p->out) || p->ldo % 8 != 0) return false;
  if (p->gate && !p->gate_per_head && (!a16(p->gate) || p->gate_tok_stride % 8 != 0)) return false;
  // Narrow heads with at most 192 keys: three blocks of 64 queries end before one pair of 128, most of whose second tile is empty (16 heads of 64, 130 tokens: 14 us
  // there, 16 here; 200 tokens 16 / 16, 300 20 / 16; heads of 128 win from 16 tokens on: 18 / 16).
  if (p->dk == 64 && p->Lq > 128 && p->q_pos0 + p->Lq <= 192) return false;
  return true;
}

int window_attn_tc(const evo_window_attn_params* p, cudaStream_t st) { return p->dk == 128 ? launch<128>(p, st) : launch<64>(p, st); }

}  // namespace evo
