// Causal attention of a prompt portion over keys and values expanded from latent cache rows: one pass over the keys, running
// maximum and sum (rescaled only when a weight would exceed 2^8, the conditional rescaling that FlashAttention 4 describes),
// probabilities rounded to bf16 before the division by the row sum, fp32 sums.  The layer's prompt form without a window
// (models/decoder_blocks.py, LatentAttention).
//
//   q    bf16 [token][head][dn + dr]   the last dr rotated
//   k    bf16 [key][head][dn]          expanded from the latent; the rotated part of a key is shared by the heads and read
//   kr   bf16 [key][dr]                where it is cached (dr may be 0)
//   v    bf16 [key][head][dv]
//
// Why expanded: with the query absorbed (q W_uk, 512 + 64 wide) scores and weighted sum of a head take 2 (576 + 512) flops
// a pair of tokens, here 2 (192 + 128), and the output of a head fits the tensor memory beside two score tiles.
//
// One CTA = 128 queries of one head, key tiles of 128:
//   warps 0..7   two groups of 128 threads, thread = query row: group g takes the tiles j = g mod 2 with its own score tile,
//                accumulator, maximum and sum, so one group exponentiates while the tensor core works for the other; a row's
//                128 scores are in registers, P goes back over them in tensor memory (the A operand of P.V).  At the end the
//                groups' outputs are merged.
//   warp 8       TMA: Q once, a ring of key tiles and one of value tiles
//   warps 9, 10  issue the products of group 0 / 1: Q.K^T of tile j, then, once P of it is stored, P.V and Q.K^T of j + 2
//                (P.V reads P before Q.K^T overwrites it: one thread's products run in order)
//   warp 11      allocates the tensor memory
// Bound by the chain of a tile (scores -> registers -> maximum -> exponentials -> P -> product), 1.8 us where its exponentials
// are 0.55: 2048 tokens, 16 heads of 128 + 64 / 128, 41 us with the SFU at 22 %, the tensor pipe at 29 % and the issue slots at
// 25 % of their peaks.  The absorbed form's products over the whole square, its softmax and conversions took 390 us, the
// expansion (a product of 4096 rows) and this kernel some 65; the layer 526 -> 164 us (149 with its launches in one call).
// 128 scores a thread in registers are all that 384 threads may have (168 registers, 48 bytes of spills).
#include <mutex>

#include "common.cuh"
#include "decode.cuh"

namespace b200 {

namespace {

constexpr int LP_TQ = 128, LP_TK = 128;
constexpr int LP_BLK = 16 * 1024;       // 128 rows x 64 columns of bf16
constexpr int LP_THREADS = 384;
constexpr int LP_MAX_STAGES = 4;
constexpr int LP_MAX_SMEM = 226 * 1024;   // (227 KB a block, less what is static)
constexpr int LP_O0 = 256;              // TMEM columns: S / P of the groups 0, 128 | O 256, 384
constexpr float LP_LAZY = 8.f;          // log2 of what a weight may exceed 1 by before the row is rescaled

struct LpParams {
  void* out;
  long o_ts;
  int out32;
  int dn, dr, dv, dvp, n_q, S, stages;
  float c;             // scale * log2(e): exponents are of two
  int flags;
};

struct LpBars {
  uint64_t q_full, k_full[LP_MAX_STAGES], k_empty[LP_MAX_STAGES], v_full[LP_MAX_STAGES], v_empty[LP_MAX_STAGES], s_full[2],
      p_full[2], o_full[2], dropped, drained[2];
};

__device__ int g_lp_wait_failed;   // a wait ran out: B200_WAIT_LATENT

__device__ __forceinline__ uint32_t l_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void l_init(uint64_t* bar, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(l_u32(bar)), "r"(n));
}
__device__ __forceinline__ void l_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(l_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void l_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(l_u32(bar)) : "memory");
}
__device__ __forceinline__ void l_tma_3d(void* dst, const CUtensorMap* tmap, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(l_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(l_u32(bar))
      : "memory");
}
__device__ __forceinline__ void l_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void l_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void l_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(l_u32(bar)) : "memory");
}
// 128-byte swizzle, groups of 8 rows 1024 bytes apart; K-major, or (values: dims contiguous) MN-major with 64-element blocks
// LP_BLK bytes apart
constexpr uint32_t L_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t l_desc_k(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t l_desc_mn(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | ((uint32_t)(LP_BLK >> 4) << 16); }
__device__ __forceinline__ void l_mma_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
               "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d),
               "r"(a), "r"(b), "r"(L_DESC_HI), "r"(idesc), "r"(acc)
               : "memory");
}
__device__ __forceinline__ void l_mma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tmov.b64 db, {%2, %3};\n\t"
               "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d),
               "r"(a), "r"(b), "r"(L_DESC_HI), "r"(idesc), "r"(acc)
               : "memory");
}
// (the values may be used after l_ld_wait of the same registers)
__device__ __forceinline__ void l_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
#define LP_R16(r)                                                                                                            \
  "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),    \
      "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
__device__ __forceinline__ void l_ld_wait16(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : LP_R16(r)::"memory");
}
// (16 more registers of a load that a wait before has covered)
__device__ __forceinline__ void l_ld_also16(uint32_t* r) { asm volatile("" : LP_R16(r)::"memory"); }
__device__ __forceinline__ void l_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void l_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 2^x on the SFU (relative error 2^-22)
__device__ __forceinline__ float l_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void l_bar256() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// a ring slot and the parity of its current round, counted along
struct LpSlot {
  int i;
  uint32_t par;
  __device__ __forceinline__ void step(int by, int n) {
    i += by;
    if (i >= n) {
      i -= n;
      par ^= 1u;
    }
  }
};

__global__ void __launch_bounds__(LP_THREADS, 1)
attention_latent_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmQr,
                        const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmKr,
                        const __grid_constant__ CUtensorMap tmV, const LpParams p) {
  extern __shared__ uint8_t lp_raw[];
  __shared__ LpBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  const int kbn = (p.dn + 63) >> 6, kb = kbn + (p.dr > 0 ? 1 : 0), vb = (p.dvp + 63) >> 6, nst = p.stages;
  uint8_t* Qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lp_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* Ks = Qs + kb * LP_BLK;
  uint8_t* Vs = Ks + nst * kb * LP_BLK;
  float2* stat = reinterpret_cast<float2*>(Qs);     // [group][query], after the last product
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x;
  const int row0 = (gridDim.y - 1 - blockIdx.y) * LP_TQ;    // the query tiles with the most keys start first
  const int q_last = min(row0 + LP_TQ, p.n_q) - 1;
  const int S = p.S;
  const int end = S - p.n_q + q_last + 1;           // keys that the tile's last query sees
  const int n_tiles = (end + LP_TK - 1) / LP_TK;

  if (threadIdx.x == 0) {
    l_init(&bars.q_full, 1);
    for (int i = 0; i < LP_MAX_STAGES; ++i) {
      l_init(&bars.k_full[i], 1);
      l_init(&bars.k_empty[i], 1);
      l_init(&bars.v_full[i], 1);
      l_init(&bars.v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      l_init(&bars.s_full[i], 1);
      l_init(&bars.p_full[i], 128);
      l_init(&bars.o_full[i], 1);
      l_init(&bars.drained[i], 1);
    }
    l_init(&bars.dropped, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 11) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(l_u32(&tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  l_fence_before();
  __syncthreads();
  l_fence_after();
  const uint32_t tmem = tmem_slot;
  // (the next kernel may start from here on, not before: it may ask for tensor memory too, and would hold what this one still needs)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int k_loads = 0, v_loads = 0;   // of the loading thread

  if (warp >= 8) {
    if (warp == 8) {
      if (lane == 0 && !(p.flags & 1)) {  // ===== loads (flags 1: none, every wait for them runs out) =====
        l_expect_tx(&bars.q_full, (uint32_t)kb * LP_BLK);
        for (int c = 0; c < kbn; ++c) l_tma_3d(Qs + c * LP_BLK, &tmQ, &bars.q_full, c * 64, h, row0);
        if (p.dr) l_tma_3d(Qs + kbn * LP_BLK, &tmQr, &bars.q_full, 0, h, row0);
        LpSlot sk{0, 1u}, sv{0, 1u};
        bool ok = true;
        for (int j = 0; j < n_tiles + 1 && ok; ++j) {   // K of tile j, then V of j - 1 (a tile ahead of its product)
          if (j < n_tiles) {
            if (!(ok = mbar_wait(&bars.k_empty[sk.i], sk.par, &failed))) break;
            ++k_loads;
            l_expect_tx(&bars.k_full[sk.i], (uint32_t)kb * LP_BLK);
            uint8_t* d = Ks + sk.i * kb * LP_BLK;
            for (int c = 0; c < kbn; ++c) l_tma_3d(d + c * LP_BLK, &tmK, &bars.k_full[sk.i], c * 64, h, j * LP_TK);
            if (p.dr) l_tma_3d(d + kbn * LP_BLK, &tmKr, &bars.k_full[sk.i], 0, 0, j * LP_TK);
            sk.step(1, nst);
          }
          if (j >= 1) {
            if (!(ok = mbar_wait(&bars.v_empty[sv.i], sv.par, &failed))) break;
            ++v_loads;
            l_expect_tx(&bars.v_full[sv.i], (uint32_t)vb * LP_BLK);
            for (int c = 0; c < vb; ++c)
              l_tma_3d(Vs + (sv.i * vb + c) * LP_BLK, &tmV, &bars.v_full[sv.i], c * 64, h, (j - 1) * LP_TK);
            sv.step(1, nst);
          }
        }
      }
    } else if (warp < 11) {
      const int g = warp - 9;
      if (lane == 0 && g < n_tiles) {  // ===== products of group g =====
        // D = f32, A = B = bf16, M = 128; bit 16: B is MN-major
        constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);
        const uint32_t id_o = ID | (1u << 16) | ((uint32_t)(p.dvp >> 3) << 17);
        const int kn = (p.dn + 15) >> 4, kr = (p.dr + 15) >> 4;
        const uint32_t q_lo = l_desc_k(l_u32(Qs)), k_lo = l_desc_k(l_u32(Ks)), v_lo = l_desc_mn(l_u32(Vs));
        const uint32_t d_s = tmem + (uint32_t)g * 128u, d_o = tmem + LP_O0 + (uint32_t)g * 128u;
        bool dead = false;
        LpSlot sk{0, 0u}, sv{0, 0u};
        if (g) { sk.step(1, nst); sv.step(1, nst); }
        auto keys16 = [&](int j) { return min(LP_TK, (end - j * LP_TK + 15) & ~15); };
        auto scores = [&](int j) {
          mbar_wait_issuer(&bars.k_full[sk.i], sk.par, dead);
          l_fence_after();
          const uint32_t id_s = ID | ((uint32_t)(keys16(j) >> 3) << 17);
          const uint32_t ka = k_lo + (uint32_t)(sk.i * kb * (LP_BLK >> 4));
#pragma unroll 4
          for (int i = 0; i < kn; ++i) {
            const uint32_t off = (uint32_t)((i >> 2) * (LP_BLK >> 4) + (i & 3) * 2);
            l_mma_ss(d_s, q_lo + off, ka + off, id_s, i > 0 ? 1u : 0u);
          }
#pragma unroll 4
          for (int i = 0; i < kr; ++i) {
            const uint32_t off = (uint32_t)(kbn * (LP_BLK >> 4) + i * 2);
            l_mma_ss(d_s, q_lo + off, ka + off, id_s, 1u);
          }
          l_commit(dead ? &bars.dropped : &bars.k_empty[sk.i]);
          l_commit(dead ? &bars.dropped : &bars.s_full[g]);
          sk.step(2, nst);
        };
        mbar_wait_issuer(&bars.q_full, 0, dead);
        scores(g);
        uint32_t par = 0;
        for (int j = g; j < n_tiles; j += 2, par ^= 1u) {
          mbar_wait_issuer(&bars.v_full[sv.i], sv.par, dead);
          mbar_wait_issuer(&bars.p_full[g], par, dead);
          l_fence_after();
          const uint32_t va = v_lo + (uint32_t)(sv.i * vb * (LP_BLK >> 4));
          const int n = keys16(j) >> 4;   // (groups of 16 keys that no query of the tile sees are left out; rows behind the last key
                                          //  are zeros: the tensor maps end there)
#pragma unroll
          for (int i = 0; i < LP_TK / 16; ++i) {
            if (i >= n) break;
            l_mma_ts(d_o, d_s + (uint32_t)(i * 8), va + (uint32_t)(i * (2048 >> 4)), id_o, (j > g || i > 0) ? 1u : 0u);
          }
          l_commit(dead ? &bars.dropped : &bars.v_empty[sv.i]);
          l_commit(dead ? &bars.dropped : &bars.o_full[g]);
          sv.step(2, nst);
          if (j + 2 < n_tiles) scores(j + 2);
        }
        if (dead) *static_cast<volatile int*>(&failed) = 1;
      }
    }
  } else {
    // ===== softmax: thread = query row of group g =====
    const int g = warp >> 2, q4 = warp & 3, row = q4 * 32 + lane, qi = row0 + row;
    const int vis = S - p.n_q + min(qi, p.n_q - 1) + 1;   // (rows behind the last query repeat it)
    const int vis_lo = __shfl_sync(0xffffffffu, vis, 0), vis_hi = __shfl_sync(0xffffffffu, vis, 31);
    const uint32_t t_row = tmem + ((uint32_t)(q4 * 32) << 16), t_s = t_row + (uint32_t)g * 128u;
    const uint32_t t_o = t_row + LP_O0 + (uint32_t)g * 128u;
    const uint64_t c2 = f2(p.c, p.c);
    float m = -INFINITY, l = 0.f;
    bool ok = true;     // (the same in a warp)
    int t = 0;
    for (int j = g; j < n_tiles; j += 2, ++t) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.s_full[g], t & 1, &failed));
      if (!ok) break;
      l_fence_after();
      uint32_t x[128];
      const int v0 = vis - j * LP_TK;
      const int nch = min(4, max(0, (vis_hi - j * LP_TK + 31) >> 5));    // groups of 32 columns that some row of the warp sees
      const bool whole = vis_lo - j * LP_TK >= LP_TK;
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (nch > 0) {
        l_ld16(t_s, x);
        l_ld16(t_s + 16, x + 16);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c < nch) {
          l_ld_wait16(x + c * 32);
          l_ld_also16(x + c * 32 + 16);
          if (c < 3 && c + 1 < nch) {
            l_ld16(t_s + (c + 1) * 32, x + (c + 1) * 32);
            l_ld16(t_s + (c + 1) * 32 + 16, x + (c + 1) * 32 + 16);
          }
          if (!whole) {
#pragma unroll
            for (int e = c * 32; e < c * 32 + 32; ++e) x[e] = e < v0 ? x[e] : 0xff800000u;
          }
#pragma unroll
          for (int e = c * 32; e < c * 32 + 32; e += 2)
            mx[(e >> 1) & 3] = fmaxf(fmaxf(mx[(e >> 1) & 3], __uint_as_float(x[e])), __uint_as_float(x[e + 1]));
        }
      }
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      // the row's reference moves only when a weight would exceed 2^8 (and on the first visible key)
      const bool grow = mt > -INFINITY && !((mt - m) * p.c <= LP_LAZY);
      if (__any_sync(0xffffffffu, grow)) {
        const float mn = fmaxf(m, mt);
        const float f = m > -INFINITY ? l_ex2((m - mn) * p.c) : (mn > -INFINITY ? 0.f : 1.f);
        m = mn;
        l *= f;
        if (t > 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(&bars.o_full[g], (t - 1) & 1, &failed));
          if (!ok) break;
          l_fence_after();
          for (int c = 0; c < p.dvp; c += 16) {
            uint32_t r[16];
            l_ld16(t_o + (uint32_t)c, r);
            l_ld_wait16(r);
#pragma unroll
            for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * f);
            l_st16(t_o + (uint32_t)c, r);
          }
        }
      }
      const float ref = m > -INFINITY ? -m * p.c : 0.f;
      const uint64_t ref2 = f2(ref, ref);
      uint64_t sum[2] = {0ull, 0ull};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c < nch) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const uint64_t y = fma2(f2(__uint_as_float(x[c * 32 + 2 * e]), __uint_as_float(x[c * 32 + 2 * e + 1])), c2, ref2);
            const float a = l_ex2(f2_lo(y)), b = l_ex2(f2_hi(y));
            sum[e & 1] = add2(sum[e & 1], f2(a, b));
            x[c * 16 + e] = pack2(a, b);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) x[c * 16 + e] = 0u;
        }
        l_st16(t_s + c * 16, x + c * 16);
      }
      sum[0] = add2(sum[0], sum[1]);
      l += f2_lo(sum[0]) + f2_hi(sum[0]);
      l_st_wait();
      l_fence_before();
      l_arrive(&bars.p_full[g]);
    }
    if (ok && t > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.o_full[g], (t - 1) & 1, &failed));
      l_fence_after();
    }
    // ---- merge: out = (O0 2^(m0 - m) + O1 2^(m1 - m)) / l, 16 columns at a time, the groups in turn; a thread reads the other
    //      group's accumulator too, for whose products only that group has waited ----
    l_fence_before();
    l_bar256();     // (no product reads Q any more)
    stat[g * LP_TQ + row] = make_float2(m, l);
    l_bar256();
    l_fence_after();
    const bool whole = !*static_cast<volatile int*>(&failed);
    const float2 a = stat[row], b = stat[LP_TQ + row];
    const float mm = fmaxf(a.x, b.x);
    const float fa = a.x > -INFINITY ? l_ex2((a.x - mm) * p.c) : 0.f, fb = b.x > -INFINITY ? l_ex2((b.x - mm) * p.c) : 0.f;
    const float inv = 1.0f / (a.y * fa + b.y * fb);
    const float ia = fa * inv, ib = fb * inv;
    const bool two = n_tiles > 1;
    for (int c = g * 16; c < p.dvp; c += 32) {
      uint32_t u[16], w[16];
      l_ld16(t_row + LP_O0 + (uint32_t)c, u);
      if (two) l_ld16(t_row + LP_O0 + 128u + (uint32_t)c, w);
      l_ld_wait16(u);
      if (two) l_ld_also16(w);
      float o[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        o[e] = __uint_as_float(u[e]) * ia;
        if (two) o[e] = fmaf(__uint_as_float(w[e]), ib, o[e]);
        if (!whole) o[e] = __uint_as_float(0x7FC00000u);
      }
      if (qi >= p.n_q) continue;
      const long at = (long)qi * p.o_ts + (long)h * p.dv + c;
      if (p.out32) {
        float* d = static_cast<float*>(p.out) + at;
#pragma unroll
        for (int e = 0; e < 16; e += 4)
          if (c + e < p.dv) *reinterpret_cast<float4*>(d + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
      } else {
        bf16* d = static_cast<bf16*>(p.out) + at;
#pragma unroll
        for (int e = 0; e < 16; e += 8)
          if (c + e < p.dv)
            *reinterpret_cast<uint4*>(d + e) = make_uint4(pack2(o[e], o[e + 1]), pack2(o[e + 2], o[e + 3]), pack2(o[e + 4], o[e + 5]),
                                                          pack2(o[e + 6], o[e + 7]));
      }
    }
  }
  l_fence_before();
  __syncthreads();
  if (failed) {   // nothing is left in flight: the last loads of every slot, the products of each issuer
    if (lane == 0 && warp >= 8 && warp < 11) {
      if (warp == 8) {
        g_lp_wait_failed = B200_WAIT_LATENT;
        if (!(p.flags & 1)) mbar_drain(&bars.q_full, 0);
        for (int i = max(0, k_loads - nst); i < k_loads; ++i) mbar_drain(&bars.k_full[i % nst], (i / nst) & 1);
        for (int i = max(0, v_loads - nst); i < v_loads; ++i) mbar_drain(&bars.v_full[i % nst], (i / nst) & 1);
      } else {
        l_commit(&bars.drained[warp - 9]);
        mbar_drain(&bars.drained[warp - 9], 0);
      }
    }
    __syncthreads();
  }
  if (warp == 11) {
    l_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

}  // namespace

static WaitWord g_lp_wait_word([](int* v) -> int {
  B200_CUDA(cudaMemcpyFromSymbol(v, g_lp_wait_failed, sizeof(int)));
  return B200_OK;
});

// ---- host: 3-D tensor maps ----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn tmap_encoder() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}
// dims (d0 contiguous, d1 with stride s1 elements, d2 with stride s2), box (b0, b1, b2); made anew on each call (half a microsecond)
static int tmap_bf16_3d(const void* ptr, int d0, int d1, long s1, int d2, long s2, int b0, int b1, int b2, CUtensorMap* out) {
  EncodeTiledFn enc = tmap_encoder();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled unavailable");
    return B200_ERR_CUDA;
  }
  const cuuint64_t gdim[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
  const cuuint64_t gstr[2] = {(cuuint64_t)s1 * 2, (cuuint64_t)s2 * 2};
  const cuuint32_t box[3] = {(cuuint32_t)b0, (cuuint32_t)b1, (cuuint32_t)b2}, estr[3] = {1, 1, 1};
  const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), gdim, gstr, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled(3d) failed (%d) ptr=%p dims=(%d,%d,%d) strides=(%ld,%ld) box=(%d,%d,%d)", (int)r, ptr,
              d0, d1, d2, s1, s2, b0, b1, b2);
    return B200_ERR_CUDA;
  }
  return B200_OK;
}

static int attention_latent(const void* q, long q_ts, const void* k, long k_ts, const void* kr, long kr_ts, const void* v, long v_ts,
                     void* out, long o_ts, int out32, int n_heads, int dn, int dr, int dv, int n_q, int S, float scale, int flags,
                     cudaStream_t st) {
  auto al = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
  B200_REQUIRE(n_heads > 0 && n_q > 0 && S >= n_q, "attention_latent: heads=%d queries=%d keys=%d", n_heads, n_q, S);
  B200_REQUIRE(dn > 0 && dn % 8 == 0 && dr >= 0 && dr <= 64 && dr % 8 == 0 && dv > 0 && dv % 8 == 0 && dv <= 128 &&
                   cdiv(dn, 64) + (dr > 0) <= 3,
               "attention_latent: head dims %d + %d, %d", dn, dr, dv);
  B200_REQUIRE(q && k && v && out && (kr || !dr) && al(q) && al(k) && al(kr) && al(v) && al(out) && q_ts % 8 == 0 && k_ts % 8 == 0 &&
                   kr_ts % 8 == 0 && v_ts % 8 == 0 && o_ts % 8 == 0,
               "attention_latent: operands need 16-byte rows");
  B200_REQUIRE(scale > 0.f, "attention_latent: scale %g", scale);
  const int kb = cdiv(dn, 64) + (dr > 0), dvp = (dv + 15) & ~15, vb = cdiv(dvp, 64);
  CUtensorMap tq, tqr, tk, tkr, tv;
  int rc;
  if ((rc = tmap_bf16_3d(q, dn, n_heads, dn + dr, n_q, q_ts, 64, 1, LP_TQ, &tq))) return rc;
  if ((rc = tmap_bf16_3d(k, dn, n_heads, dn, S, k_ts, 64, 1, LP_TK, &tk))) return rc;
  if ((rc = tmap_bf16_3d(v, dv, n_heads, dv, S, v_ts, 64, 1, LP_TK, &tv))) return rc;
  tqr = tq;
  tkr = tk;
  if (dr) {
    if ((rc = tmap_bf16_3d((const bf16*)q + dn, dr, n_heads, dn + dr, n_q, q_ts, 64, 1, LP_TQ, &tqr))) return rc;
    if ((rc = tmap_bf16_3d(kr, dr, 1, dr, S, kr_ts, 64, 1, LP_TK, &tkr))) return rc;
  }
  LpParams p;
  p.out = out; p.o_ts = o_ts; p.out32 = out32;
  p.dn = dn; p.dr = dr; p.dv = dv; p.dvp = dvp; p.n_q = n_q; p.S = S;
  p.c = scale * 1.4426950408889634f;
  p.flags = flags;
  // As many ring slots as fit beside Q, an even number: a slot belongs to one of the two issuing threads, which then sees every
  // round of it (with an odd number it would meet each second round, and the parity of the one before the last passes for it)
  p.stages = min(LP_MAX_STAGES, (LP_MAX_SMEM - 1024 - kb * LP_BLK) / ((kb + vb) * LP_BLK)) & ~1;
  B200_REQUIRE(p.stages >= 2, "attention_latent: %d key and %d value blocks", kb, vb);
  static unsigned long long set_mask = 0ull;
  if (FirstUse first{&set_mask})
    B200_CUDA(cudaFuncSetAttribute(attention_latent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LP_MAX_SMEM));
  const size_t smem = (size_t)(kb + p.stages * (kb + vb)) * LP_BLK + 1024;
  B200_CUDA(launch_pdl(attention_latent_kernel, dim3(n_heads, cdiv(n_q, LP_TQ)), dim3(LP_THREADS), smem, st, tq, tqr, tk, tkr, tv, p));
  return B200_OK;
}

}  // namespace b200

extern "C" int b200_lm_latent_expanded_attention(const void* q, long q_ts, const void* k, long k_ts, const void* kr, long kr_ts,
                                                 const void* v, long v_ts, void* out, long o_ts, int out32, int n_heads, int dn,
                                                 int dr, int dv, int n_q, int S, float scale, int flags, void* stream) {
  return b200::attention_latent(q, q_ts, k, k_ts, kr, kr_ts, v, v_ts, out, o_ts, out32, n_heads, dn, dr, dv, n_q, S, scale, flags,
                                (cudaStream_t)stream);
}
