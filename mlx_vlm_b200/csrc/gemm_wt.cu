// gemm_wt: the Linear layers of the prefill / vision / batched-decode paths as a WEIGHT-MAJOR
// tcgen05 GEMM:   D[n, t] = sum_k W[n, k] * X[t, k]      (C[t, n] = D[n, t])
//
// Why weight-major ("swap AB"): the token count of this path is small and awkward for the
// tensor core's M = 128 side (T = 272 -> 3 tiles, one of them 88 % padding; T = 576 -> 4.5
// tiles; batched decode T <= 16), while the weight rows are many and regular.  So the
// weight rows take the UMMA M side (128 rows per CTA, streamed exactly once per token tile)
// and the tokens the N side, whose width TN is any multiple of 16 up to 256 and is chosen per
// problem (T = 272 -> 2 x 144, T = 576 -> 3 x 192, decode batch -> 16): no padded MMA rows,
// 2-3x less weight re-streaming than 128-row token tiles.
//
//   * TMA (cp.async.bulk.tensor, 128B swizzle) feeds a shared-memory ring of `n_stages` stages
//     of KS k-blocks (64 columns each); one elected thread issues tcgen05.mma (fp32 accumulators
//     in TMEM: 128 lanes = weight rows x TN columns = tokens);
//   * programmatic dependent launch: the weight tiles of the first stages do not depend on the
//     previous kernel and are requested BEFORE griddepcontrol.wait, so the cold-HBM latency of a
//     layer's weights overlaps the previous kernel's tail; shared memory is kept <= 113 KB where
//     that does not hurt so that two CTAs (of this or the next kernel) share an SM;
//   * split-K over gridDim.z for the GEMMs with few weight rows and long K (o_proj, down, fc2):
//     fp32 partial tiles, summed in a FIXED order by the row-op kernel that follows
//     (finish_rows: bias + residual + RMSNorm / LayerNorm of the next block, fused);
//   * epilogue: TMEM -> registers (lane = weight row) -> rows of C (bias / GELU / residual, or SwiGLU of gate and up rows that
//     the TMA box interleaves: 64 channels per tile) or fp32 partial tiles; nothing goes through shared memory.
//
// Replaces nn.Linear of the reference (models/qwen2_vl/vision.py:83-102,108-119,132-133,168-169;
// language.py:52-55; mlp.py:9-15; activations.py:8-10).  Rounding points follow
// oracle/mlx_semantics.py::linear (+ activations, residual add).
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "decode.cuh"

namespace b200 {

namespace {

constexpr int WT_ROWS = 128;        // weight rows per CTA (UMMA M)
constexpr int WT_BK = 64;           // one k-block: 64 bf16 = 128 B = one swizzle row
constexpr int WT_WBLK = WT_ROWS * 128;  // bytes of one weight k-block tile
constexpr int WT_MAX_STAGES = 16;

struct WtParams {
  const bf16* bias;
  const bf16* residual;
  bf16* C;
  float* partial;
  long ldc, ldr;
  int T, N, K;
  int TN, KS, n_stages;
  int kb_per_split;
  int epilogue, mode;
  int inter;
  unsigned flags;  // debug: 1 = no MMA (loads only), 2 = no loads (MMA on stale smem; CTA pairs: the waits run out), 4 = no epilogue stores
  // fp32-accurate towers (LLaVA / Idefics2: the reference runs them in fp32 with bf16-valued weights):
  // X is a SPLIT operand [x_hi | x_lo] (n parts of K_w columns, each padded to 64) multiplied by the SAME
  // weight k-blocks (kb_w of them): D = W.x_hi + W.x_lo in fp32 — exact to ~2^-17 relative.
  int kb_w;          // > 0: weight k-block = k-block % kb_w
  float* C32;        // B200_WT_F32: fp32 output (bias, activation, fp32 residual)
  const float* res32;
  long ldc32, ldr32;
  bf16* Csplit;      // B200_WT_SPLIT: output written as [hi | lo] bf16 halves, n_pad columns apart
  long ld_split;
  int n_pad;
  const int* tile_group;  // grouped products: token tile y multiplies the weight rows of group tile_group[y] (< 0: empty)
  int col_groups, x_group_cols;  // column groups: blockIdx.y = group x token tile; X columns / C32 columns move with the group
  long c_group_cols;
  int w_group_cols;  // > 0: the groups' weights are column ranges of the SAME rows, this many columns apart (else rows g N .. of W)
};

__device__ __forceinline__ uint32_t w_smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void w_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(w_smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void w_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void w_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(w_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void w_mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = w_smem_u32(bar);
  uint32_t done = mbar_test(addr, parity);
  while (!done) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
  }
}
__device__ __forceinline__ void w_tma_2d(void* dst, const CUtensorMap* tmap, uint64_t* bar, int c0,
                                         int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(w_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(w_smem_u32(bar))
      : "memory");
}
// SwiGLU's weights as [channel][gate, up][k]: 64 channels are 128 rows of the tile
__device__ __forceinline__ void w_tma_3d(void* dst, const CUtensorMap* tmap, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(w_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(w_smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void w_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void w_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// descriptors as (lo, hi) words: walking an operand is one 32-bit add per MMA
__device__ __forceinline__ void w_umma(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t hi,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void w_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   w_smem_u32(bar))
               : "memory");
}
// K-major, 128B swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint32_t w_desc_lo(uint32_t addr) {
  return ((addr & 0x3FFFFu) >> 4) | (1u << 16);
}
constexpr uint32_t W_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);

// (its values may be used after w_ld_wait)
__device__ __forceinline__ void w_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void w_ld_wait(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])::"memory");
}
__device__ __forceinline__ void w_pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void w_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- the accumulator tile (128 weight rows x TN tokens, fp32 in TMEM) -> its outputs, by 256 threads (tid; warp tid / 32 reads
// TMEM lane quarter (tid / 32) mod 4, which must be its own, and every other group of 8 tokens).
// Outputs go from the registers to memory as they are: a lane has a weight row, so a warp's store of a token is 32 consecutive
// features: 128 bytes of fp32, and of bf16, two tokens at a time, 64 bytes of each.  Through a staging tile in shared memory, as
// 16-byte rows, the warps waited for one another twice per 64 tokens, which every product pays at its end and those of short k
// of pairs all along.  Staged -> direct, calls of several products and what lies between them: one picture through four vision
// blocks 287 -> 269 us, 6012 patches through two 1001 -> 981, eight pictures through three CLIP blocks (fp32) 1234 -> 1199, 2048
// tokens through a latent attention block (fp32) 149 -> 140, 272 through four 2B layers 249 -> 243.
// The loops are small on purpose: a launch fetches its code anew, and 32 tokens unrolled were 1 - 2 us of fetching at the end of
// every product (stamps of one CTA, 576 x 5120 x 1280 with GELU: 2.1 us for the first 32 tokens, 1.0 for the next; the exact GELU
// 15 and 4.2).
struct WtTile {
  uint32_t tmem;
  int n0, t0;     // first output feature and token
  long cg;        // first C32 column (column groups)
  int split, tid;
  float bias;     // of the thread's weight row: loaded before the products are waited for
  bool dead;      // a wait of this CTA ended without its data: NaN is stored
};

// the bias of a thread's weight row (SwiGLU: rows are gate and up of the channels in turn)
template <bool TOWER>
__device__ __forceinline__ float wt_bias(const WtParams& p, int n0, int tid) {
  const int row = (tid >> 5 & 3) * 32 + (tid & 31);
  if (TOWER && p.mode == B200_WT_SWIGLU_SPLIT) return p.bias && n0 + (row >> 1) < p.inter ? bf2f(p.bias[(row & 1) * p.inter + n0 + (row >> 1)]) : 0.f;
  return p.bias && (TOWER || p.mode == B200_WT_BF16) && n0 + row < p.N ? bf2f(p.bias[n0 + row]) : 0.f;
}

// bias + activation of two tokens of one weight row, rounded to bf16 before and after the activation
template <int EPI>
__device__ __forceinline__ uint32_t wt_act_bf16(uint32_t a0, uint32_t a1, float bias) {
  const uint32_t v = pack_bf2(add2(f2(__uint_as_float(a0), __uint_as_float(a1)), f2(bias, bias)));
  if constexpr (EPI == B200_EPI_GELU_FAST) return gelu_fast_bf2(v);
  if constexpr (EPI == B200_EPI_GELU_EXACT) return pack2(gelu_exact_bf(__uint_as_float(v << 16)), gelu_exact_bf(__uint_as_float(v & 0xffff0000u)));
  return v;
}
// the fp32-accurate paths: no rounding anywhere
template <int EPI>
__device__ __forceinline__ void wt_act_f32(uint32_t& a0, uint32_t& a1, float bias) {
  uint64_t v = add2(f2(__uint_as_float(a0), __uint_as_float(a1)), f2(bias, bias));
  if constexpr (EPI == B200_EPI_GELU_FAST) v = mul2(v, sigmoid2(mul2(v, f2(1.702f, 1.702f))));
  float x[2] = {f2_lo(v), f2_hi(v)};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if constexpr (EPI == B200_EPI_GELU_EXACT) x[e] = x[e] * (1.0f + erff(x[e] / 1.41421356237309515f)) * 0.5f;
    if constexpr (EPI == B200_EPI_GELU_TANH) {
      const float u = 0.7978845608028654f * (x[e] + 0.044715f * x[e] * x[e] * x[e]);
      x[e] = 0.5f * x[e] * (1.0f + tanhf(u));
    }
  }
  a0 = __float_as_uint(x[0]);
  a1 = __float_as_uint(x[1]);
}
// Lanes of a pair (by apart) hold two tokens (low, high half) each of their row; the first gets both rows of the low token, the
// second those of the high one.
__device__ __forceinline__ uint32_t wt_swap(uint32_t v, int by, uint32_t sel) {
  return __byte_perm(v, __shfl_xor_sync(0xffffffffu, v, by), sel);
}

// The warp's groups of 8 tokens in turn: body(first token, accumulators, residuals); the accumulators of the next group, and what
// its residual(first token, words) asks for, are on their way meanwhile.
template <class Residual, class Body>
__device__ __forceinline__ void wt_groups(const WtTile& c, int tokens, Residual residual, Body body) {
  const int warp = c.tid >> 5;
  const uint32_t taddr = c.tmem + ((uint32_t)((warp & 3) * 32) << 16);
  uint32_t next[8], a[8], r_next[8], r[8];
  int cc = (warp >> 2) * 8;
  if (cc >= tokens) return;
  w_ld8(taddr + (uint32_t)cc, next);
  residual(cc, r_next);
#pragma unroll 1
  for (; cc < tokens; cc += 16) {
    w_ld_wait(next);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = c.dead ? 0x7FC00000u : next[j], r[j] = r_next[j];
    if (cc + 16 < tokens) {
      w_ld8(taddr + (uint32_t)cc + 16, next);
      residual(cc + 16, r_next);
    }
    body(cc, a, r);
  }
}

// Does the warp's last feature stand alone (an odd number of features, two to a word)?  It has a loop of its own: one more predicate per
// store in the other's is 2 - 3 % of a vision block.  (Rows of an odd number element by element took 11 - 20 % longer where the
// stores show: 300 x 32003 x 1024 31.5 us, 25.8 so; 600 x 1153 x 1152 18.0 and 15.0.)
__device__ __forceinline__ bool wt_odd_end(const WtParams& p, const WtTile& c) {
  return (p.N & 1) && c.n0 + (c.tid >> 5 & 3) * 32 + 32 > p.N;
}
template <bool TAIL>
__device__ __forceinline__ void wt_put_word(bf16* d, uint32_t v, bool both) {
  if (!TAIL || both) *reinterpret_cast<uint32_t*>(d) = v;
  else *reinterpret_cast<unsigned short*>(d) = (unsigned short)v;
}

// bf16 rows, two features of a token as one word
template <int EPI, bool TAIL>
__device__ __forceinline__ void wt_store_words(const WtParams& p, const WtTile& c, int tokens) {
  const int lane = c.tid & 31, n = c.n0 + (c.tid >> 5 & 3) * 32 + (lane & ~1), odd = lane & 1;
  const uint32_t sel = odd ? 0x3276u : 0x5410u;
  const bool store = n < p.N && !(p.flags & 4u), both = n + 1 < p.N;
  bf16* const d0 = p.C + (long)(c.t0 + odd) * p.ldc + n;
  const bf16* const s0 = p.residual + (long)(c.t0 + odd) * p.ldr + n;
  auto body = [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8], auto with_res) {
    const int nv = store ? tokens - cc - odd : 0;
    bf16* d = d0 + (long)cc * p.ldc;
#pragma unroll
    for (int i = 0; i < 4; ++i, d += 2 * p.ldc) {
      uint32_t v = wt_swap(wt_act_bf16<EPI>(a[2 * i], a[2 * i + 1], c.bias), 1, sel);
      if constexpr (decltype(with_res)::value) v = pack_bf2(add2(unpack_bf2(r[i]), unpack_bf2(v)));
      if (2 * i < nv) wt_put_word<TAIL>(d, v, both);
    }
  };
  if (p.residual) {
    wt_groups(c, tokens, [&](int cc, uint32_t (&r)[8]) {
      const int nv = store ? tokens - cc - odd : 0;
      const bf16* s = s0 + (long)cc * p.ldr;
#pragma unroll
      for (int i = 0; i < 4; ++i, s += 2 * p.ldr) {
        r[i] = 0u;
        if (2 * i < nv) r[i] = !TAIL || both ? *reinterpret_cast<const uint32_t*>(s) : *reinterpret_cast<const unsigned short*>(s);
      }
    }, [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8]) { body(cc, a, r, std::true_type{}); });
  } else {
    wt_groups(c, tokens, [](int, uint32_t (&)[8]) {}, [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8]) { body(cc, a, r, std::false_type{}); });
  }
}

template <int EPI>
__device__ __forceinline__ void wt_store_bf16(const WtParams& p, const WtTile& c, int tokens) {
  const bool res = p.residual != nullptr;
  if (((p.ldc | (res ? p.ldr : 0)) & 1) == 0 &&
      ((reinterpret_cast<uintptr_t>(p.C) | (res ? reinterpret_cast<uintptr_t>(p.residual) : 0)) & 3) == 0) {
    if (wt_odd_end(p, c)) wt_store_words<EPI, true>(p, c, tokens);
    else wt_store_words<EPI, false>(p, c, tokens);
    return;
  }
  // odd strides or bases: element by element, the residuals on their way like the accumulators (read where they are added, 2048 x 4608 x
  // 3584 on pairs took 115 us and 576 x 3840 x 1280 31; so 51 and 13)
  const int n = c.n0 + (c.tid >> 5 & 3) * 32 + (c.tid & 31);
  const bool store = n < p.N && !(p.flags & 4u);
  wt_groups(c, tokens, [&](int cc, uint32_t (&r)[8]) {
    const int nv = store && res ? tokens - cc : 0;
    const bf16* s = p.residual + (long)(c.t0 + cc) * p.ldr + n;
#pragma unroll
    for (int j = 0; j < 8; ++j, s += p.ldr) r[j] = j < nv ? *reinterpret_cast<const unsigned short*>(s) : 0u;
  }, [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8]) {
    const int nv = store ? tokens - cc : 0;
    bf16* d = p.C + (long)(c.t0 + cc) * p.ldc + n;
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      uint32_t v = wt_act_bf16<EPI>(a[j], a[j + 1], c.bias);
      if (res) v = pack_bf2(add2(unpack_bf2(r[j] | (r[j + 1] << 16)), unpack_bf2(v)));
#pragma unroll
      for (int e = 0; e < 2; ++e, d += p.ldc)
        if (j + e < nv) *reinterpret_cast<unsigned short*>(d) = (unsigned short)(v >> (16 * e));
    }
  });
}

// [hi | lo]: hi = bf16(v), lo = bf16(v - hi), two features to a word (rows and parts lie 8-feature aligned)
template <int EPI, bool TAIL>
__device__ __forceinline__ void wt_store_split(const WtParams& p, const WtTile& c, int tokens) {
  const int lane = c.tid & 31, n = c.n0 + (c.tid >> 5 & 3) * 32 + (lane & ~1), odd = lane & 1;
  const uint32_t sel = odd ? 0x3276u : 0x5410u;
  const bool store = n < p.N && !(p.flags & 4u), both = n + 1 < p.N;
  bf16* const d0 = p.Csplit + (long)(c.t0 + odd) * p.ld_split + n;
  wt_groups(c, tokens, [](int, uint32_t (&)[8]) {}, [&](int cc, uint32_t (&a)[8], uint32_t (&)[8]) {
    const int nv = store ? tokens - cc - odd : 0;
    bf16* d = d0 + (long)cc * p.ld_split;
#pragma unroll
    for (int i = 0; i < 4; ++i, d += 2 * p.ld_split) {
      wt_act_f32<EPI>(a[2 * i], a[2 * i + 1], c.bias);
      const float x0 = __uint_as_float(a[2 * i]), x1 = __uint_as_float(a[2 * i + 1]);
      uint32_t hi = pack2(x0, x1);
      uint32_t lo = pack2(x0 - __uint_as_float(hi << 16), x1 - __uint_as_float(hi & 0xffff0000u));
      hi = wt_swap(hi, 1, sel);
      lo = wt_swap(lo, 1, sel);
      if (2 * i < nv) {
        wt_put_word<TAIL>(d, hi, both);
        wt_put_word<TAIL>(d + p.n_pad, lo, both);
      }
    }
  });
}

// fp32 rows, or [hi | lo]
template <int EPI>
__device__ __forceinline__ void wt_store_f32(const WtParams& p, const WtTile& c, int tokens) {
  const int n = c.n0 + (c.tid >> 5 & 3) * 32 + (c.tid & 31);
  const bool store = n < p.N && !(p.flags & 4u);
  auto none = [](int, uint32_t (&)[8]) {};
  if (p.mode == B200_WT_F32) {
    float* const d0 = p.C32 + (long)c.t0 * p.ldc32 + c.cg + n;
    auto body = [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8], auto with_res) {
      const int nv = store ? tokens - cc : 0;
      float* d = d0 + (long)cc * p.ldc32;
#pragma unroll
      for (int j = 0; j < 8; j += 2) wt_act_f32<EPI>(a[j], a[j + 1], c.bias);
#pragma unroll
      for (int j = 0; j < 8; ++j, d += p.ldc32) {
        float v = __uint_as_float(a[j]);
        if constexpr (decltype(with_res)::value) v += __uint_as_float(r[j]);
        if (j < nv) *d = v;
      }
    };
    if (p.res32) {
      const float* const s0 = p.res32 + (long)c.t0 * p.ldr32 + n;
      wt_groups(c, tokens, [&](int cc, uint32_t (&r)[8]) {
        const int nv = store ? tokens - cc : 0;
        const float* s = s0 + (long)cc * p.ldr32;
#pragma unroll
        for (int j = 0; j < 8; ++j, s += p.ldr32) r[j] = j < nv ? __float_as_uint(*s) : 0u;
      }, [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8]) { body(cc, a, r, std::true_type{}); });
    } else {
      wt_groups(c, tokens, none, [&](int cc, uint32_t (&a)[8], uint32_t (&r)[8]) { body(cc, a, r, std::false_type{}); });
    }
    return;
  }
  if (wt_odd_end(p, c)) wt_store_split<EPI, true>(p, c, tokens);
  else wt_store_split<EPI, false>(p, c, tokens);
}

// SwiGLU: the tile's rows are gate and up of its channels in turn (w_tma_3d), so neighbouring lanes hold a channel: one swap gives
// each both of them for one token, another one, of two tokens between channels, two channels to a word.  Gate and up as blocks of
// 64 rows each, which met in shared memory: eight prompts of 608 tokens through two Llama-7B layers 4120 us, so 4080; 272 tokens
// through four 2B layers 243 and 241; five lock-step rows 172 and 160; four pictures through the SigLIP projection 2734 and 2702.
template <bool TOWER, int EPI>
__device__ __forceinline__ void wt_store_swiglu(const WtParams& p, const WtTile& c, int tokens) {
  const int lane = c.tid & 31, i0 = c.n0 + (c.tid >> 5 & 3) * 16 + (lane >> 1);   // channel
  const int odd = lane & 1, later = lane & 2;                                      // which tokens it gets and stores
  const uint32_t sel = odd ? 0x3276u : 0x5410u, sel2 = later ? 0x3276u : 0x5410u;
  const bool store = i0 < p.inter && !(p.flags & 4u);
  auto none = [](int, uint32_t (&)[8]) {};
  const long ld = TOWER ? p.ld_split : p.ldc;
  bf16* const d0 = (TOWER ? p.Csplit : p.C) + (long)(c.t0 + odd + later) * ld + (i0 & ~1);
  wt_groups(c, tokens, none, [&](int cc, uint32_t (&a)[8], uint32_t (&)[8]) {
    const int nv = store ? tokens - cc - odd - later : 0;
    bf16* d = d0 + cc * ld;
#pragma unroll
    for (int i = 0; i < 8; i += 4, d += 4 * ld) {   // tokens i + odd and two on
      if constexpr (!TOWER) {
        const uint32_t x = wt_swap(wt_act_bf16<EPI>(a[i], a[i + 1], 0.f), 1, sel), y = wt_swap(wt_act_bf16<EPI>(a[i + 2], a[i + 3], 0.f), 1, sel);
        const uint32_t r = wt_swap(swiglu_bf2(__byte_perm(x, y, 0x5410), __byte_perm(x, y, 0x7632)), 2, sel2);
        if (i < nv) *reinterpret_cast<uint32_t*>(d) = r;
      } else {
        // silu(gate) * up in fp32, as the next product's operand: the [T, 2 inter] fp32 rows between the two never reach memory.
        // 4096 tokens x 28672 rows x 1152 (two parts) with a kernel of its own behind it 399 + 115 us (and 60 to clear its rows), this 396.
        float g[2], u[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t &a0 = a[i + 2 * e], &a1 = a[i + 2 * e + 1];
          wt_act_f32<EPI>(a0, a1, c.bias);
          const uint32_t mine = odd ? a1 : a0, its = __shfl_xor_sync(0xffffffffu, odd ? a0 : a1, 1);
          g[e] = __uint_as_float(odd ? its : mine);
          u[e] = __uint_as_float(odd ? mine : its);
        }
        const uint64_t g2 = f2(g[0], g[1]), v = mul2(mul2(g2, sigmoid2(g2)), f2(u[0], u[1]));
        const uint32_t h = pack_bf2(v);
        const uint32_t l = pack2(f2_lo(v) - __uint_as_float(h << 16), f2_hi(v) - __uint_as_float(h & 0xffff0000u));
        const uint32_t hi = wt_swap(h, 2, sel2), lo = wt_swap(l, 2, sel2);
        if (i < nv) {
          *reinterpret_cast<uint32_t*>(d) = hi;
          *reinterpret_cast<uint32_t*>(d + p.n_pad) = lo;
        }
      }
    }
  });
}

template <bool TOWER>
__device__ __forceinline__ void wt_store_tile(const WtParams& p, const WtTile& c) {
  if (p.flags & 1u) return;
  const int tokens = min(p.TN, p.T - c.t0), q = c.tid >> 5 & 3;
  // one loop per epilogue kind, chosen OUTSIDE the loop: left to itself the compiler merged the
  // three kinds into one predicated body of ~90 instructions per element (6-7 us per launch, A/B measured)
  if (p.mode == (TOWER ? B200_WT_SWIGLU_SPLIT : B200_WT_SWIGLU)) {
    if (c.n0 + q * 16 >= p.inter) return;
    if constexpr (TOWER) {
      wt_store_swiglu<true, B200_EPI_NONE>(p, c, tokens);
    } else {
      if (p.epilogue == B200_EPI_GELU_FAST) wt_store_swiglu<false, B200_EPI_GELU_FAST>(p, c, tokens);
      else if (p.epilogue == B200_EPI_GELU_EXACT) wt_store_swiglu<false, B200_EPI_GELU_EXACT>(p, c, tokens);
      else wt_store_swiglu<false, B200_EPI_NONE>(p, c, tokens);
    }
    return;
  }
  if (c.n0 + q * 32 >= p.N) return;
  if constexpr (TOWER) {
    if (p.epilogue == B200_EPI_GELU_FAST) wt_store_f32<B200_EPI_GELU_FAST>(p, c, tokens);
    else if (p.epilogue == B200_EPI_GELU_EXACT) wt_store_f32<B200_EPI_GELU_EXACT>(p, c, tokens);
    else if (p.epilogue == B200_EPI_GELU_TANH) wt_store_f32<B200_EPI_GELU_TANH>(p, c, tokens);
    else wt_store_f32<B200_EPI_NONE>(p, c, tokens);
  } else if (p.mode == B200_WT_PARTIAL) {   // fp32 partial tile -> P[split][t][n]
    const int n = c.n0 + q * 32 + (c.tid & 31);
    const bool store = n < p.N && !(p.flags & 4u);
    float* const d0 = p.partial + ((long)c.split * p.T + c.t0) * p.N + n;
    wt_groups(c, tokens, [](int, uint32_t (&)[8]) {}, [&](int cc, uint32_t (&a)[8], uint32_t (&)[8]) {
      const int nv = store ? tokens - cc : 0;
      float* d = d0 + (long)cc * p.N;
#pragma unroll
      for (int j = 0; j < 8; ++j, d += p.N)
        if (j < nv) *d = __uint_as_float(a[j]);
    });
  } else {
    if (p.epilogue == B200_EPI_GELU_FAST) wt_store_bf16<B200_EPI_GELU_FAST>(p, c, tokens);
    else if (p.epilogue == B200_EPI_GELU_EXACT) wt_store_bf16<B200_EPI_GELU_EXACT>(p, c, tokens);
    else wt_store_bf16<B200_EPI_NONE>(p, c, tokens);
  }
}

// TOWER = false: the bf16 paths (B200_WT_BF16 / PARTIAL / SWIGLU); TOWER = true: the fp32-accurate paths
// (B200_WT_F32 / SPLIT / SWIGLU_SPLIT).  Two instantiations keep each one's code small.
template <bool TOWER>
__global__ void __launch_bounds__(256, 2)
gemm_wt_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
               const WtParams p) {
  extern __shared__ uint8_t wt_smem_raw[];
  __shared__ uint64_t full_bar[WT_MAX_STAGES], empty_bar[WT_MAX_STAGES];
  __shared__ uint64_t tmem_full;
  __shared__ uint32_t tmem_slot;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wt_smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool swiglu = p.mode == (TOWER ? B200_WT_SWIGLU_SPLIT : B200_WT_SWIGLU);
  const int rb = blockIdx.x;
  const int n0 = rb * (swiglu ? 64 : WT_ROWS);  // first output feature (SwiGLU: channel) of the tile
  int n0w = n0;                                 // first weight row of the tile (grouped: inside the tile's group)
  int ty = blockIdx.y, xk0 = 0, wk0 = 0;        // token tile; first X and W column (column groups)
  long cg = 0;                                  // first C32 column (column groups)
  if (p.tile_group) {
    const int g = p.tile_group[blockIdx.y];
    if (g < 0) return;                          // an empty token tile: nothing is allocated yet
    n0w += g * p.N;
  } else if (p.col_groups > 0) {
    const int tpg = gridDim.y / p.col_groups, g = ty / tpg;
    ty -= g * tpg;
    if (p.w_group_cols > 0) wk0 = g * p.w_group_cols;
    else n0w += g * p.N;
    xk0 = g * p.x_group_cols;
    cg = (long)g * p.c_group_cols;
  }
  const int t0 = ty * p.TN;
  const int split = blockIdx.z;
  const int kb_total = (p.K + WT_BK - 1) / WT_BK;
  const int kb0 = split * p.kb_per_split;
  const int kb1 = min(kb_total, kb0 + p.kb_per_split);
  const int n_it = (kb1 - kb0 + p.KS - 1) / p.KS;
  const int xblk = p.TN * 128;                      // bytes of one token k-block tile
  const int stage_bytes = p.KS * (WT_WBLK + xblk);
  const int NS = p.n_stages;
  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < p.TN) tmem_cols <<= 1;

  auto issue_w = [&](int it, int s) {
    uint8_t* sW = ring + (long)s * stage_bytes;
    const int cnt = min(p.KS, kb1 - kb0 - it * p.KS);
    if (p.flags & 2u) {  // debug: no loads at all, the MMAs run on whatever the ring holds
      w_mbar_arrive(&full_bar[s]);
      return;
    }
    w_mbar_expect_tx(&full_bar[s], (uint32_t)cnt * (WT_WBLK + xblk));
    for (int j = 0; j < cnt; ++j) {
      int kbw = kb0 + it * p.KS + j;
      if (p.kb_w > 0) kbw %= p.kb_w;
      const int kc = kbw * WT_BK + wk0;
      if (swiglu) w_tma_3d(sW + j * WT_WBLK, &tmW, &full_bar[s], kc, 0, n0);
      else w_tma_2d(sW + j * WT_WBLK, &tmW, &full_bar[s], kc, n0w);
    }
  };
  auto issue_x = [&](int it, int s) {
    if (p.flags & 2u) return;
    uint8_t* sX = ring + (long)s * stage_bytes + p.KS * WT_WBLK;
    const int cnt = min(p.KS, kb1 - kb0 - it * p.KS);
    for (int j = 0; j < cnt; ++j)
      w_tma_2d(sX + j * xblk, &tmX, &full_bar[s], (kb0 + it * p.KS + j) * WT_BK + xk0, t0);
  };

  const int pre = n_it < NS ? n_it : NS;
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmX)) : "memory");
    for (int s = 0; s < NS; ++s) {
      w_mbar_init(&full_bar[s], 1);
      w_mbar_init(&empty_bar[s], 1);
    }
    w_mbar_init(&tmem_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // weights never depend on the previous kernel: request them before waiting for it
    for (int it = 0; it < pre; ++it) issue_w(it, it);
  }
  if (warp == 2) {  // whole warp: tcgen05.alloc is .sync.aligned
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     w_smem_u32(&tmem_slot)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  w_fence_before();
  __syncthreads();
  w_fence_after();
  const uint32_t tmem_base = tmem_slot;
  w_pdl_wait();  // everything the previous kernels wrote (X, residual, the bias) is visible from here on

  if (warp == 0) {
    if (lane == 0) {  // ===== TMA producer =====
      for (int it = 0; it < pre; ++it) issue_x(it, it);
      int s = 0;   // (slot and parity are counted along: no division per stage)
      uint32_t parity = 0;
      for (int it = pre; it < n_it; ++it) {
        w_mbar_wait(&empty_bar[s], parity);
        issue_w(it, s);
        issue_x(it, s);
        if (++s == NS) s = 0, parity ^= 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ===== MMA issuer =====
      // D = f32, A = B = bf16, both K-major; M = 128 weight rows, N = TN tokens
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.TN >> 3) << 17) |
                             ((uint32_t)(WT_ROWS >> 4) << 24);
      uint32_t acc = 0, parity = 0;
      int s = 0;
      for (int it = 0; it < n_it; ++it) {
        w_mbar_wait(&full_bar[s], parity);
        w_fence_after();
        if (!(p.flags & 1u)) {
          const uint32_t w_lo = w_desc_lo(w_smem_u32(ring + (long)s * stage_bytes));
          const uint32_t x_lo = w_desc_lo(w_smem_u32(ring + (long)s * stage_bytes + p.KS * WT_WBLK));
          const int cnt = min(p.KS, kb1 - kb0 - it * p.KS);
          for (int j = 0; j < cnt; ++j) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              w_umma(tmem_base, w_lo + (uint32_t)(j * (WT_WBLK >> 4) + kk * 2),
                     x_lo + (uint32_t)(j * (xblk >> 4) + kk * 2), W_DESC_HI, idesc, acc);
              acc = 1;
            }
          }
        }
        w_commit(&empty_bar[s]);  // frees the ring slot when these MMAs retire
        if (++s == NS) s = 0, parity ^= 1;
      }
      w_commit(&tmem_full);
      // The next kernel may start its set-up and weight loads as SM resources free up: not before this tile's products are issued,
      // for its blocks hold shared memory and registers while they wait, which other streams' kernels could use.  Signalled when
      // the block starts instead: 272 tokens through four 2B layers, three such sequences in flight, 241 us a call, so 231;
      // one at a time 439, 432; eight lock-step rows 377 and 375, one picture 259 and 261.
      w_pdl_launch();
    }
  }
  __syncwarp();

  // ===== epilogue (all 8 warps): warp w reads TMEM lane quarter w % 4, token half w / 4 =====
  const float bias = wt_bias<TOWER>(p, n0, threadIdx.x);   // (on its way while the products are)
  w_mbar_wait(&tmem_full, 0);
  w_fence_after();
  wt_store_tile<TOWER>(p, WtTile{tmem_base, n0, t0, cg, split, (int)threadIdx.x, bias, false});
  w_fence_before();
  __syncthreads();
  if (warp == 2) {
    w_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// The same product for many tokens: CTA PAIRS (cta_group::2), persistent.  A pair multiplies 256 weight rows by TN tokens:
// each CTA keeps 128 weight rows and HALF of the tokens of a k-block in its shared memory and the tensor cores of both read
// both halves, so a 128 x 256 share of the output costs 32 KB of fill per k-block instead of 48: what bounds the one-CTA
// kernel at these sizes is the fill (all SMs together take 11.5 - 12 TB/s out of the L2: 1,050 TFLOP/s at 48 KB).  Two
// accumulators in TMEM: the epilogue warps store a tile while the next one is multiplied, and the ring never drains between
// tiles.
// Measured, one CTA -> pairs: 4896 tokens x 22016 rows x 4096 (SwiGLU) 878 -> 629 us (1,404 TFLOP/s), x 12288 x 4096 479 -> 335,
// x 4096 x 11008 427 -> 332; 2048 x 37888 x 3584 588 -> 418; 6012 x 3840 x 1280 64 -> 52; below a wave of pairs it loses
// (576 x 3840 x 1280 11.8 -> 14.7), so it is one more candidate of the measured choice.
//   warp 0  TMA producer of this CTA's operands; the bytes of both CTAs count on the leader's (rank 0) full barrier
//   warp 1  leader only: MMA issuer; its commits free the slot / hand the accumulator over in both CTAs
//   warp 2  TMEM
//   warps 4..11  epilogue of this CTA's 128 weight rows (wide: of the first 128, warps 12..19 of the others)
// Tiles are dealt out round robin, token tile first, so that the pairs of a wave share weight rows in the L2.
// Up to about 3600 columns of k the epilogue's arithmetic shows: its eight warps have as long as the products of a tile take.  In
// pairs of tokens (packed additions and bf16 products, ex2 and rcp without their slow ranges: about 9 instructions an element for
// the fast GELU instead of some 45): 6012 x 5120 x 1280 with GELU 91 -> 66 us (65 without GELU, 54 without any epilogue).
// HALVES = 2, "wide": 512 weight rows a pair, 256 of each CTA as two accumulators of 128 x TN that share the token operand.  What
// bounds the pairs of 256 rows with long k is their fill, 32 KB of each CTA for 512 cycles of products (64 bytes a cycle, where
// all SMs together got 42 - 53 out of the L2); here 48 KB serve 1024 cycles.  All of the tensor memory is taken, so
// a tile's accumulators are read while the tensor core works on the other half: the second half's products run WP_LAG k-blocks
// behind the first's where a tile begins and ends, and eight epilogue warps belong to each half.  256 -> 512 rows, back to back:
// 2048 tokens x 3584 rows x 18944 207 -> 188 us, 4864 x 4096 x 11008 324 -> 300, 4096 x 4096 x 28672 675 -> 623 (under the
// power limit 243 -> 222, 376 -> 353, 776 -> 728; one-CTA tiles 273, 465, 861).  With k below some 3000 the ends of a tile cost
// more than the fill saves (6012 x 3840 x 1280 45 -> 56, 4096 x 28672 x 2304 367 -> 390).  WP_LAG 0 / 1 / 2 / 3 / 4:
// 2048 x 37888 x 3584 371 / 375 / 365 / 363 / 363, 6012 x 5120 x 1280 93 / 92 / 88 / 84 / 83.
// ---------------------------------------------------------------------------------------------
constexpr int WP_THREADS = 384, WP_WIDE_THREADS = 640;
constexpr int WP_LAG = 3;                                   // (at most the ring's stages, which are held meanwhile)
constexpr int WP_MAX_STAGES = 12;

struct WpBars {
  uint64_t full[WP_MAX_STAGES], empty[WP_MAX_STAGES], acc_full[2], acc_empty[2], dropped, drained;
};

__device__ int g_pair_wait_failed;   // a wait of gemm_wt_pair_kernel ran out: B200_WAIT_PAIR

__device__ __forceinline__ uint32_t wp_leader(const void* p) {   // shared::cluster address of *p in the pair's rank 0
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(w_smem_u32(p)));
  return r;
}
__device__ __forceinline__ void wp_tma_2d(void* dst, const CUtensorMap* tmap, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(w_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void wp_tma_3d(void* dst, const CUtensorMap* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(w_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void wp_umma(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(W_DESC_HI), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void wp_commit(uint64_t* bar) {   // arrives on *bar of both CTAs when the MMAs so far have retired
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(w_smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void wp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <bool TOWER, int HALVES>
__global__ void __launch_bounds__(HALVES == 2 ? WP_WIDE_THREADS : WP_THREADS, 1)
gemm_wt_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const WtParams p) {
  extern __shared__ uint8_t wt_smem_raw[];
  __shared__ WpBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wt_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const bool swiglu = p.mode == (TOWER ? B200_WT_SWIGLU_SPLIT : B200_WT_SWIGLU);
  const int xhalf = p.TN / 2, stage_bytes = HALVES * WT_WBLK + xhalf * 128, NS = p.n_stages;
  const int kb_total = (p.K + WT_BK - 1) / WT_BK;
  const int unit = swiglu ? 64 : WT_ROWS;   // output features of 128 weight rows
  const int row_tiles = ((swiglu ? 2 * p.inter : p.N) + 2 * HALVES * WT_ROWS - 1) / (2 * HALVES * WT_ROWS), tok_tiles = (p.T + p.TN - 1) / p.TN;
  const int splits = (kb_total + p.kb_per_split - 1) / p.kb_per_split;
  const int n_tiles = row_tiles * tok_tiles * splits;
  int s_next = 0;             // the producer's next slot
  uint32_t free_parity = 1;   // and the phase in which it is free
  // tile -> this CTA's first output feature, its first token, its k-blocks
  auto tile_at = [&](int tile, int& n0, int& t0, int& split, int& kb0, int& kb1) {
    t0 = tile % tok_tiles * p.TN;
    tile /= tok_tiles;
    n0 = (tile % row_tiles * 2 * HALVES + rank) * unit;   // (the second half's: 2 units on)
    split = tile / row_tiles;
    kb0 = split * p.kb_per_split;
    kb1 = min(kb_total, kb0 + p.kb_per_split);
  };

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmW)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmX)) : "memory");
    for (int s = 0; s < NS; ++s) {
      w_mbar_init(&bars.full[s], 1);
      w_mbar_init(&bars.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      w_mbar_init(&bars.acc_full[b], 1);
      w_mbar_init(&bars.acc_empty[b], 16);   // eight epilogue warps of each CTA
    }
    w_mbar_init(&bars.dropped, 1);
    w_mbar_init(&bars.drained, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(w_smem_u32(&tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  w_fence_before();
  __syncthreads();
  wp_cluster_sync();   // the peer's barriers exist before anything arrives on them
  w_fence_after();
  const uint32_t tmem = tmem_slot;
  w_pdl_launch();   // (not before all columns are this pair's: the next kernel may ask for some)

  if (warp == 0) {
    if (lane == 0 && !(p.flags & 2u)) {  // ===== TMA producer (flags 2: nothing is loaded; a test in its loop cost 2 %) =====
      const uint32_t full0 = wp_leader(&bars.full[0]);
      auto load_w = [&](int s, int kb, int n0) {
        if (p.kb_w > 0) kb %= p.kb_w;
        uint8_t* sW = ring + (long)s * stage_bytes;
        const uint32_t bar = full0 + s * 8;
        if (rank == 0) w_mbar_expect_tx(&bars.full[s], 2u * (uint32_t)stage_bytes);
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          const int n = n0 + h * 2 * unit;
          if (swiglu) wp_tma_3d(sW + h * WT_WBLK, &tmW, bar, kb * WT_BK, 0, n);
          else wp_tma_2d(sW + h * WT_WBLK, &tmW, bar, kb * WT_BK, n);
        }
      };
      auto load_x = [&](int s, int kb, int t0) {
        wp_tma_2d(ring + (long)s * stage_bytes + HALVES * WT_WBLK, &tmX, full0 + s * 8, kb * WT_BK, t0 + rank * xhalf);
      };
      int n0, t0, split, kb0, kb1;
      // weights never depend on the previous kernel: those of the first slots are requested before waiting for it
      int pre = 0;
      if (pair < n_tiles) {
        tile_at(pair, n0, t0, split, kb0, kb1);
        pre = min(NS, kb1 - kb0);
        for (int i = 0; i < pre; ++i) load_w(i, kb0 + i, n0);
      }
      w_pdl_wait();
      int s = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
        tile_at(tile, n0, t0, split, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (pre > 0) {
            --pre;
          } else {
            ok = mbar_wait(&bars.empty[s], free_parity, &failed);
            if (!ok) break;
            load_w(s, kb, n0);
          }
          load_x(s, kb, t0);
          if (++s == NS) s = 0, free_parity ^= 1;
        }
      }
      s_next = s;
    }
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {  // ===== MMA issuer =====
      // D = f32, A = B = bf16, both K-major; M = 256 weight rows, N = TN tokens
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.TN >> 3) << 17) | (16u << 24);
      // (slot and parity are counted along: a division per k-block would cost more than its four products)
      const uint32_t w_first = w_desc_lo(w_smem_u32(ring)), x_first = w_desc_lo(w_smem_u32(ring + HALVES * WT_WBLK));
      const uint32_t step = (uint32_t)stage_bytes >> 4;
      int s = 0, j = 0, n0, t0, split, kb0, kb1;
      uint32_t w_lo = w_first, x_lo = x_first, parity = 0;
      bool dead = false;
      w_pdl_wait();   // (the time of a wait starts when the tokens can be on their way)
      if constexpr (HALVES == 2) {
        // the products of k-block s with one half of the weight rows
        auto half = [&](int h, uint32_t acc) {
#pragma unroll
          for (int k = 0; k < 4; ++k) wp_umma(tmem + h * 256u, w_lo + h * (WT_WBLK >> 4) + k * 2, x_lo + k * 2, idesc, k > 0 ? 1u : acc);
        };
        auto next = [&] {
          w_lo += step;
          x_lo += step;
          if (++s == NS) s = 0, w_lo = w_first, x_lo = x_first, parity ^= 1;
        };
        auto arrived = [&] {
          mbar_wait_issuer(&bars.full[s], parity, dead);
          w_fence_after();
        };
        for (int tile = pair; tile < n_tiles; tile += n_pairs, ++j) {
          tile_at(tile, n0, t0, split, kb0, kb1);
          const int nk = kb1 - kb0, lag = min(min(WP_LAG, NS), nk >> 1);
          const uint32_t free_par = (j & 1) ^ 1;
          mbar_wait_issuer(&bars.acc_empty[0], free_par, dead);
          w_fence_after();
          // the first k-blocks: the second half lags behind, its accumulator is still being read (their slots are full: no waits)
          int s0 = s;
          uint32_t w0 = w_lo, x0 = x_lo, p0 = parity;
          for (int i = 0; i < lag; ++i, next()) {
            arrived();
            half(0, i > 0);
          }
          mbar_wait_issuer(&bars.acc_empty[1], free_par, dead);
          w_fence_after();
          if (lag > 0) s = s0, w_lo = w0, x_lo = x0, parity = p0;
          for (int i = 0; i < lag; ++i, next()) {
            half(1, i > 0);
            wp_commit(dead ? &bars.dropped : &bars.empty[s]);
          }
          for (int i = lag; i < nk - lag; ++i, next()) {
            arrived();
            half(0, i > 0);
            half(1, i > 0);
            wp_commit(dead ? &bars.dropped : &bars.empty[s]);
          }
          // the last ones: the first half is whole before the second's products begin
          s0 = s, w0 = w_lo, x0 = x_lo, p0 = parity;
          for (int i = 0; i < lag; ++i, next()) {
            arrived();
            half(0, 1u);
          }
          wp_commit(dead ? &bars.dropped : &bars.acc_full[0]);
          if (lag > 0) s = s0, w_lo = w0, x_lo = x0, parity = p0;
          for (int i = 0; i < lag; ++i, next()) {
            half(1, 1u);
            wp_commit(dead ? &bars.dropped : &bars.empty[s]);
          }
          wp_commit(dead ? &bars.dropped : &bars.acc_full[1]);
        }
      } else {
        for (int tile = pair; tile < n_tiles; tile += n_pairs, ++j) {
          tile_at(tile, n0, t0, split, kb0, kb1);
          const uint32_t d = tmem + (uint32_t)(j & 1) * 256u;
          mbar_wait_issuer(&bars.acc_empty[j & 1], ((j >> 1) & 1) ^ 1, dead);
          w_fence_after();
          uint32_t acc = 0;
          for (int kb = kb0; kb < kb1; ++kb) {
            mbar_wait_issuer(&bars.full[s], parity, dead);
            w_fence_after();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              wp_umma(d, w_lo + k * 2, x_lo + k * 2, idesc, acc);
              acc = 1;
            }
            wp_commit(dead ? &bars.dropped : &bars.empty[s]);
            w_lo += step;
            x_lo += step;
            if (++s == NS) s = 0, w_lo = w_first, x_lo = x_first, parity ^= 1;
          }
          wp_commit(dead ? &bars.dropped : &bars.acc_full[j & 1]);   // (an accumulator that is not whole is not handed over)
        }
      }
      if (dead) *static_cast<volatile int*>(&failed) = 1;
    }
  } else if (warp >= 4) {  // ===== epilogue =====
    w_pdl_wait();
    int j = 0, n0, t0, split, kb0, kb1;
    bool ok = true;   // (the same in a warp)
    const int half = HALVES == 2 ? (warp - 4) >> 3 : 0;   // eight warps to a half
    for (int tile = pair; tile < n_tiles; tile += n_pairs, ++j) {
      tile_at(tile, n0, t0, split, kb0, kb1);
      const int a = HALVES == 2 ? half : j & 1;   // accumulator
      const int row0 = n0 + half * 2 * unit, tid = (int)(threadIdx.x - 128) & 255;
      const float bias = wt_bias<TOWER>(p, row0, tid);
      ok = ok && __all_sync(0xffffffffu, mbar_wait(&bars.acc_full[a], (HALVES == 2 ? j : j >> 1) & 1, &failed));
      w_fence_after();
      wt_store_tile<TOWER>(p, WtTile{tmem + (uint32_t)a * 256u, row0, t0, 0, split, tid, bias, !ok});
      w_fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(wp_leader(&bars.acc_empty[a]))
                     : "memory");
    }
  }
  __syncwarp();
  w_fence_before();
  __syncthreads();
  if (failed && threadIdx.x == 0)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.b32 [a], %2;\n\t}" ::"r"(w_smem_u32(&failed)),
                   "r"(r), "r"(1)
                   : "memory");
  wp_cluster_sync();   // nobody's shared memory or TMEM goes while the peer still uses it
  // (in both CTAs) nothing is left in flight: the last load of every slot that the leader counts, the products; loads that only
  // the other CTA requested have had the time of a wait that ran out
  if (*static_cast<volatile int*>(&failed)) {
    if (rank == 0 && lane == 0) {
      if (warp == 0) {
        g_pair_wait_failed = B200_WAIT_PAIR;
        for (int i = 0; i < NS; ++i) mbar_drain(&bars.full[i], i < s_next ? free_parity ^ 1 : free_parity);   // (never loaded: ends at once)
      } else if (warp == 1) {
        wp_commit(&bars.drained);
        mbar_drain(&bars.drained, 0);
      }
    }
    __syncwarp();
    wp_cluster_sync();
  }
  if (warp == 2) {
    w_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// finish_rows: h[t] = r(resid[t] + r(sum_s P[s][t] + bias)) and, fused, the normalisation that
// the NEXT block applies to h (RMSNorm / LayerNorm with the oracle's rounding points).  One CTA
// per token row; the split-K partials are added in split order (deterministic).
// ---------------------------------------------------------------------------------------------
// <threads, vectors of 4 a thread> as the row's width and the number of rows ask for (finish_rows): a chain of L2 round trips, so a
// thread has one vector where it can, and the loads of a row and of the weights go out together.  (Weights ahead of the wait for the
// product, as a caller who makes them on the device right before may not have it: the same times.)
// Against <256, 8> for all sequences, weights behind the sums: one picture through four vision blocks (2 - 7 partials of 1280 a row)
// 255 -> 251 us, 272 tokens through four 2B layers 227 -> 224; the few rows of a decode step (1024 threads) take the same time.
constexpr int FIN_N_MAX = 8192;  // N <= FIN_THREADS * 4 * FIN_MAXV in the widest shapes

// Sum of a row's vectors (q[u]: vector thread + FIN_THREADS * u).  1024 threads: as they lie.  Fewer: as 256 threads of up to 8 vectors
// each would add them, so that a row's bits do not depend on the shape: the threads from 256 on hand theirs over, ahead of the
// barrier that `red` needs anyway.
template <int FIN_THREADS, int FIN_MAXV>
__device__ __forceinline__ float fin_block_sum(const float (&q)[FIN_MAXV], float* red, float (*ex)[256]) {
  constexpr int SUMS = FIN_THREADS == 1024 ? 1024 : 256;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x >= SUMS)
#pragma unroll
    for (int u = 0; u < FIN_MAXV; ++u) ex[u][threadIdx.x - SUMS] = q[u];
  __syncthreads();
  if (threadIdx.x < SUMS) {
    float v = 0.f;
#pragma unroll
    for (int u = 0; u < FIN_MAXV; ++u) {
      v += q[u];
      if (threadIdx.x + SUMS < FIN_THREADS) v += ex[u][threadIdx.x];
    }
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
  }
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < SUMS / 32; ++w) t += red[w];
  return t;
}

template <int FIN_THREADS, int FIN_MAXV>
__global__ void __launch_bounds__(FIN_THREADS)
finish_rows_kernel(const float* __restrict__ P, int S, const bf16* bias, const bf16* resid, long ldr, bf16* h_out, long ldh,
                   int norm_kind, const bf16* nw, const bf16* nb, float eps, bf16* xn, long ldx, int T, int N) {
  __shared__ float red[FIN_THREADS / 32], ex[FIN_MAXV][256];
  w_pdl_launch();
  const int t = blockIdx.x;
  const int nv = N >> 2;
  w_pdl_wait();
  // residual, bias, norm weight and bias (plain loads of pointers that may alias: the compiler may move neither these nor those of a
  // read-only path ahead of the wait)
  uint2 rv[FIN_MAXV], wb[FIN_MAXV], wn[FIN_MAXV], wnb[FIN_MAXV];
#pragma unroll
  for (int u = 0; u < FIN_MAXV; ++u) {
    const int c = threadIdx.x + FIN_THREADS * u;
    rv[u] = resid && c < nv ? *reinterpret_cast<const uint2*>(resid + (long)t * ldr + c * 4) : make_uint2(0, 0);
    wb[u] = bias && c < nv ? *reinterpret_cast<const uint2*>(bias + c * 4) : make_uint2(0, 0);
    wn[u] = norm_kind != B200_NORM_NONE && nw && c < nv ? *reinterpret_cast<const uint2*>(nw + c * 4) : make_uint2(0, 0);
    wnb[u] = norm_kind != B200_NORM_NONE && norm_kind != B200_NORM_RMS && nb && c < nv ? *reinterpret_cast<const uint2*>(nb + c * 4) : make_uint2(0, 0);
  }
  float4 h[FIN_MAXV];
  float s1[FIN_MAXV], s2[FIN_MAXV];   // of a vector
#pragma unroll
  for (int u = 0; u < FIN_MAXV; ++u) {
    const int c = threadIdx.x + FIN_THREADS * u;
    h[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    s1[u] = s2[u] = 0.f;
    if (c < nv) {
      // the split-K partials of this chunk: up to 8 loads in flight, added in split order
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
      for (int s0 = 0; s0 < S; s0 += 8) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          v[i] = (s0 + i < S) ? __ldcg(reinterpret_cast<const float4*>(P + ((long)(s0 + i) * T + t) * N + c * 4))
                              : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          a.x += v[i].x; a.y += v[i].y; a.z += v[i].z; a.w += v[i].w;
        }
      }
      if (bias) {
        float bb[4];
        unpack4(wb[u], bb);
        a.x += bb[0]; a.y += bb[1]; a.z += bb[2]; a.w += bb[3];
      }
      a.x = rbf(a.x); a.y = rbf(a.y); a.z = rbf(a.z); a.w = rbf(a.w);
      if (resid) {
        float rr[4];
        unpack4(rv[u], rr);
        a.x = rbf(rr[0] + a.x); a.y = rbf(rr[1] + a.y); a.z = rbf(rr[2] + a.z); a.w = rbf(rr[3] + a.w);
      }
      h[u] = a;
      if (h_out)
        *reinterpret_cast<uint2*>(h_out + (long)t * ldh + c * 4) = make_uint2(pack2(a.x, a.y), pack2(a.z, a.w));
      s1[u] = (a.x + a.y) + (a.z + a.w);
      s2[u] = (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
    }
  }
  if (norm_kind == B200_NORM_NONE) return;
  if (norm_kind == B200_NORM_RMS) {
    const float tot = fin_block_sum<FIN_THREADS>(s2, red, ex);
    const float rs = 1.0f / sqrtf(tot / (float)N + eps);
#pragma unroll
    for (int u = 0; u < FIN_MAXV; ++u) {
      const int c = threadIdx.x + FIN_THREADS * u;
      if (c < nv) {
        float w[4];
        unpack4(wn[u], w);
        const float4 a = h[u];
        *reinterpret_cast<uint2*>(xn + (long)t * ldx + c * 4) =
            make_uint2(pack2(rbf(rbf(a.x * rs) * w[0]), rbf(rbf(a.y * rs) * w[1])),
                       pack2(rbf(rbf(a.z * rs) * w[2]), rbf(rbf(a.w * rs) * w[3])));
      }
    }
    return;
  }
  // LayerNorm: fp32 mean / variance (two passes over the registers), cast, * w, + b
  const float mu = fin_block_sum<FIN_THREADS>(s1, red, ex) / (float)N;
  float v[FIN_MAXV];
#pragma unroll
  for (int u = 0; u < FIN_MAXV; ++u) {
    const int c = threadIdx.x + FIN_THREADS * u;
    v[u] = 0.f;
    if (c < nv) {
      const float4 a = h[u];
      const float d0 = a.x - mu, d1 = a.y - mu, d2 = a.z - mu, d3 = a.w - mu;
      v[u] = (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
    }
  }
  const float var = fin_block_sum<FIN_THREADS>(v, red, ex) / (float)N;
  const float rstd = 1.0f / sqrtf(var + eps);
#pragma unroll
  for (int u = 0; u < FIN_MAXV; ++u) {
    const int c = threadIdx.x + FIN_THREADS * u;
    if (c < nv) {
      const float4 a = h[u];
      float o[4] = {rbf((a.x - mu) * rstd), rbf((a.y - mu) * rstd), rbf((a.z - mu) * rstd),
                    rbf((a.w - mu) * rstd)};
      if (nw) {
        float w[4];
        unpack4(wn[u], w);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = rbf(o[e] * w[e]);
      }
      if (nb) {
        float b[4];
        unpack4(wnb[u], b);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = rbf(o[e] + b[e]);
      }
      *reinterpret_cast<uint2*>(xn + (long)t * ldx + c * 4) = make_uint2(pack2(o[0], o[1]), pack2(o[2], o[3]));
    }
  }
}

// ---- host: tensor maps ------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn wt_get_encode() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}
struct WtKey {
  const void* ptr;
  long ld;
  int rows, k, box_rows;
  bool gate_up;
  bool operator==(const WtKey& o) const {
    return ptr == o.ptr && ld == o.ld && rows == o.rows && k == o.k && box_rows == o.box_rows && gate_up == o.gate_up;
  }
};
struct WtHash {
  size_t operator()(const WtKey& k) const {
    size_t h = std::hash<const void*>()(k.ptr);
    h = h * 1000003u ^ std::hash<long>()(k.ld);
    h = h * 1000003u ^ (size_t)k.rows;
    h = h * 1000003u ^ (size_t)k.k;
    h = h * 1000003u ^ (size_t)(2 * k.box_rows + k.gate_up);
    return h;
  }
};
// 2-D K-major bf16 operand (rows x K, row pitch ld elements), box = box_rows x 64; gate_up: [gate rows; up rows], `rows` of each,
// as a 3-D one (rows x 2 x K), so that a box has box_rows / 2 of both in turn
int wt_tmap(const void* ptr, long ld, int rows, int k, int box_rows, CUtensorMap* out, bool gate_up = false) {
  static std::unordered_map<WtKey, CUtensorMap, WtHash> cache;
  static std::mutex mu;
  WtKey key{ptr, ld, rows, k, box_rows, gate_up};
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return B200_OK;
    }
  }
  EncodeTiledFn enc = wt_get_encode();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled unavailable (no CUDA driver?)");
    return B200_ERR_CUDA;
  }
  const int last = gate_up ? 2 : 1;   // the dimension of the rows
  cuuint64_t gdim[3] = {(cuuint64_t)k, 2, 0};
  cuuint64_t gstr[2] = {(cuuint64_t)rows * ld * 2, 0};
  cuuint32_t box[3] = {(cuuint32_t)WT_BK, 2, 0};
  cuuint32_t estr[3] = {1, 1, 1};
  gdim[last] = (cuuint64_t)rows;
  gstr[last - 1] = (cuuint64_t)ld * 2;
  box[last] = (cuuint32_t)(gate_up ? box_rows / 2 : box_rows);
  CUtensorMap tm;
  CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, last + 1, const_cast<void*>(ptr), gdim, gstr,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) ptr=%p ld=%ld rows=%d k=%d box_rows=%d", (int)r, ptr,
              ld, rows, k, box_rows);
    return B200_ERR_CUDA;
  }
  {
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 16384) cache.clear();
    cache[key] = tm;
  }
  *out = tm;
  return B200_OK;
}

static bool g_wt_pdl = true;

}  // namespace

static WaitWord g_pair_wait_word([](int* v) -> int {
  B200_CUDA(cudaMemcpyFromSymbol(v, g_pair_wait_failed, sizeof(int)));
  return B200_OK;
});

void gemm_wt_set_pdl(bool on) { g_wt_pdl = on; }

static int round16(int x) { return (x + 15) & ~15; }

constexpr int WP_PAIRS = 74;   // pairs of SMs
constexpr int WT_KS_WIDE = -1; // WtConfig::KS of a pair with 512 weight rows (0: 256)
static bool wt_swiglu(int mode) { return mode == B200_WT_SWIGLU || mode == B200_WT_SWIGLU_SPLIT; }
constexpr size_t WT_SMEM_MAX = 227 * 1024 - 1024;
static size_t wt_smem(const WtConfig& c) {
  const int stage = c.KS <= 0 ? (c.KS == WT_KS_WIDE ? 2 : 1) * WT_WBLK + c.TN * 64 : c.KS * (WT_WBLK + c.TN * 128);
  return (size_t)c.stages * stage + 1024;
}
// what gemm_wt takes as the choice of a product (whatever its operands are)
static bool wt_takes(const WtConfig& c, int K, int mode, int col_groups) {
  const bool pair = c.KS <= 0;
  const int kb = cdiv(K, WT_BK);
  return K > 0 && c.TN >= 16 && c.TN <= 256 && c.TN % (pair ? 32 : 16) == 0 && c.KS >= (col_groups > 0 ? 1 : WT_KS_WIDE) && c.KS <= WT_MAX_STAGES &&
         c.stages >= 2 && c.stages <= (pair ? WP_MAX_STAGES : WT_MAX_STAGES) && wt_smem(c) <= WT_SMEM_MAX && c.split >= 1 && c.split <= kb &&
         cdiv(kb, cdiv(kb, c.split)) == c.split && (mode == B200_WT_PARTIAL ? c.KS != WT_KS_WIDE : c.split == 1);
}

// Tile / pipeline configuration for (T, row blocks, K): a small cost model calibrated on a
// sweep (profiles/r2_gemm_wt_sweep.txt, B200):
//   * a CTA costs ~4.5 us of fixed latency (launch, barrier/TMEM set-up, first TMA round trip,
//     epilogue) + per k-block max(MMA time, shared-memory fill time at ~130 GB/s per SM);
//   * two CTAs share an SM when a configuration needs <= ~110 KB of shared memory: the fixed part of
//     one overlaps the main loop of the other, which wins whenever more than one wave exists;
//   * split-K buys parallelism for the GEMMs with few weight rows at the price of fp32 partial
//     traffic (written here, read by finish_rows);
//   * the weights are streamed from HBM once: nothing is faster than bytes / ~6 TB/s.
void gemm_wt_auto(int T, int row_blocks, int K, bool allow_split, WtConfig* best, int sm_count) {
  const int kb_total = cdiv(K, WT_BK);
  const int t16 = round16(T);
  int tn_c[12];
  int n_tn = 0;
  auto add_tn = [&](int tn) {
    if (tn < 16) tn = 16;
    if (tn > 256) tn = 256;
    if (tn > t16) tn = t16;
    for (int i = 0; i < n_tn; ++i)
      if (tn_c[i] == tn) return;
    tn_c[n_tn++] = tn;
  };
  for (int k = 1; k <= 3; ++k) add_tn(round16(cdiv(T, k)));
  if (T > 256) {
    const int nt = cdiv(T, 256);
    for (int k = 0; k < 3; ++k) add_tn(round16(cdiv(T, nt + k)));
  }
  add_tn(96); add_tn(128); add_tn(144); add_tn(192);
  double best_t = 1e30;
  best->TN = tn_c[0]; best->KS = 1; best->stages = 2; best->split = 1;
  for (int it = 0; it < n_tn; ++it) {
    const int TN = tn_c[it];
    const int tt = cdiv(T, TN);
    const long base = (long)row_blocks * tt;
    for (int KS = 1; KS <= 4; KS *= 2) {
      const int stage = KS * (WT_WBLK + TN * 128);
      for (int occ = 2; occ >= 1; --occ) {
        const int budget = occ == 2 ? 110 * 1024 : 208 * 1024;
        int st = budget / stage;
        if (st > 8) st = 8;
        if (st < 2 || st * KS < 3) continue;
        if (occ == 1 && (long)st * stage + 2048 <= 110 * 1024) continue;  // same as the occ == 2 case
        int cand[6] = {1, 0, 0, 0, 0, 0};
        int n_sp = 1;
        if (allow_split) {
          for (int target : {sm_count, 2 * sm_count, 3 * sm_count}) {
            int sp = (int)(target / base);
            if (sp > kb_total / 4) sp = kb_total / 4;
            if (sp < 1) sp = 1;
            sp = cdiv(kb_total, cdiv(kb_total, sp));
            bool dup = false;
            for (int i = 0; i < n_sp; ++i) dup |= cand[i] == sp;
            if (!dup) cand[n_sp++] = sp;
          }
        }
        for (int is = 0; is < n_sp; ++is) {
          const int split = cand[is];
          if (split > 1 && (long)split * T * row_blocks * 128 * 4 > (40L << 20)) continue;  // partial-tile budget
          const long ctas = base * split;
          const int kbs = cdiv(kb_total, split);
          const double t_mma = 4.0 * (TN / 2.0) / 1900.0;                          // us per k-block
          const double t_fill = (WT_WBLK + TN * 128) / 130e3 * (KS == 1 ? 1.15 : 1.0);
          const double t_kb = t_mma > t_fill ? t_mma : t_fill;
          const double t_fix = 5.2;                                  // first wave, prologue hidden by PDL
          const long per_sm = (ctas + sm_count - 1) / sm_count;      // CTAs an SM has to run
          double t;
          if (occ == 2) {
            const long waves = (ctas + 2L * sm_count - 1) / (2L * sm_count);
            t = t_fix + per_sm * kbs * t_kb + (waves - 1) * 4.0;
          } else {
            t = t_fix + kbs * t_kb + (per_sm - 1) * (9.5 + kbs * t_kb);  // serialised waves pay the full CTA latency
          }
          if (st * KS < 4) t *= 1.08;
          const double fill_total = (double)ctas * kbs * (WT_WBLK + TN * 128);
          if (t < t_fix + fill_total / 12e6) t = t_fix + fill_total / 12e6;   // chip-wide L2 -> SM fill rate
          const double hbm = (double)row_blocks * 128 * K * 2 / 6e6 + 3.0;   // weights stream from HBM once
          if (t < hbm) t = hbm + 0.01 * kbs * t_kb;
          if (split > 1) t += (double)split * T * row_blocks * 128 * 4 / 6e6 + 0.2 * split;
          if (t < best_t) {
            best_t = t;
            best->TN = TN; best->KS = KS; best->stages = st; best->split = split;
          }
        }
      }
    }
  }
}

int gemm_wt(const void* X, long ldx, const void* W, const void* bias, const void* residual, long ldr,
            void* C, long ldc, float* partial, int T, int N, int K, int epilogue, int mode, int inter,
            const WtConfig& cfg, unsigned flags, cudaStream_t st, const WtExt* ext) {
  B200_REQUIRE(T > 0 && N > 0 && K > 0, "gemm_wt: empty problem T=%d N=%d K=%d", T, N, K);
  B200_REQUIRE((ldx % 8) == 0 && (K % 8) == 0, "gemm_wt: ldx (%ld) and K (%d) must be multiples of 8", ldx, K);
  B200_REQUIRE(((uintptr_t)X & 15) == 0 && ((uintptr_t)W & 15) == 0, "gemm_wt: X and W must be 16-byte aligned");
  const bool pair = cfg.KS <= 0, wide = cfg.KS == WT_KS_WIDE;   // CTA pairs
  B200_REQUIRE(cfg.TN >= 16 && cfg.TN <= 256 && (cfg.TN % (pair ? 32 : 16)) == 0, "gemm_wt: TN=%d", cfg.TN);
  B200_REQUIRE(cfg.KS >= WT_KS_WIDE && cfg.stages >= 2 && cfg.stages <= (pair ? WP_MAX_STAGES : WT_MAX_STAGES) && cfg.split >= 1,
               "gemm_wt: bad config KS=%d stages=%d split=%d", cfg.KS, cfg.stages, cfg.split);
  B200_REQUIRE(mode >= B200_WT_BF16 && mode <= B200_WT_SWIGLU_SPLIT, "gemm_wt: mode %d", mode);
  const bool tower = mode == B200_WT_F32 || mode == B200_WT_SPLIT || mode == B200_WT_SWIGLU_SPLIT, swiglu = wt_swiglu(mode);
  B200_REQUIRE(!tower || ext, "gemm_wt: fp32 / split output needs WtExt");
  B200_REQUIRE(mode != B200_WT_F32 || (ext->C32 && ((uintptr_t)ext->C32 & 15) == 0), "gemm_wt: fp32 output missing / misaligned");
  B200_REQUIRE((mode != B200_WT_SPLIT && mode != B200_WT_SWIGLU_SPLIT) || (ext->Csplit && (ext->n_pad % 8) == 0 && (ext->ld_split % 8) == 0 &&
                                         ((uintptr_t)ext->Csplit & 15) == 0),
               "gemm_wt: split output missing / misaligned");
  B200_REQUIRE(mode != B200_WT_PARTIAL || partial, "gemm_wt: partial buffer missing");
  B200_REQUIRE(mode == B200_WT_PARTIAL || cfg.split == 1, "gemm_wt: split-K needs the partial mode");
  B200_REQUIRE(!wide || mode != B200_WT_PARTIAL, "gemm_wt: wide pairs write no partial tiles");
  B200_REQUIRE(!swiglu || (inter > 0 && inter % (tower ? 4 : 8) == 0 && N == 2 * inter),
               "gemm_wt: SwiGLU needs N == 2 * inter, inter a multiple of 8 (fp32: 4)");
  const int kb_total = cdiv(K, WT_BK);
  WtParams p;
  memset(&p, 0, sizeof(p));
  p.bias = (const bf16*)bias; p.residual = (const bf16*)residual; p.C = (bf16*)C; p.partial = partial;
  p.ldc = ldc; p.ldr = ldr; p.T = T; p.N = N; p.K = K;
  p.TN = cfg.TN; p.KS = cfg.KS; p.n_stages = cfg.stages;
  p.kb_per_split = cdiv(kb_total, cfg.split);
  const int splits = cdiv(kb_total, p.kb_per_split);
  B200_REQUIRE(splits == cfg.split, "gemm_wt: split %d leaves empty splits (%d k-blocks)", cfg.split, kb_total);
  p.epilogue = epilogue; p.mode = mode; p.inter = inter; p.flags = flags & 7u;
  int k_w = K;  // columns of W (the split operand repeats the weight k-blocks)
  if (ext) {
    p.kb_w = ext->kb_w; p.C32 = ext->C32; p.res32 = ext->res32; p.ldc32 = ext->ldc32; p.ldr32 = ext->ldr32;
    p.Csplit = ext->Csplit; p.ld_split = ext->ld_split; p.n_pad = ext->n_pad;
    if (ext->kb_w > 0) k_w = ext->k_w;
    p.tile_group = ext->tile_group;
    p.col_groups = ext->col_groups; p.x_group_cols = ext->x_group_cols; p.c_group_cols = ext->c_group_cols;
    p.w_group_cols = ext->w_group_cols;
  }
  const bool heads = ext && ext->col_groups > 0;
  B200_REQUIRE(!heads || (mode == B200_WT_F32 && cfg.split == 1 && !bias && !ext->res32 && !ext->tile_group &&
                          ext->x_group_cols % 8 == 0 && ext->x_cols >= (ext->col_groups - 1) * ext->x_group_cols + k_w),
               "gemm_wt: column groups are fp32-output, unsplit, without bias / residual, 16-byte column offsets");
  const bool w_cols = heads && ext->w_group_cols > 0;
  B200_REQUIRE(!w_cols || (ext->w_group_cols % 8 == 0 && ext->ldw >= (long)(ext->col_groups - 1) * ext->w_group_cols + k_w),
               "gemm_wt: weight columns of the groups need 16-byte offsets inside the rows");
  const bool grouped = ext && ext->tile_group;
  B200_REQUIRE(!grouped || (mode == B200_WT_F32 && ext->n_groups > 0 && cfg.split == 1 && !bias),
               "gemm_wt: grouped products are fp32-output, unsplit, without bias");
  B200_REQUIRE(!pair || (!grouped && !heads), "gemm_wt: pairs take no groups");
  const size_t smem = wt_smem(cfg);
  B200_REQUIRE(smem <= WT_SMEM_MAX, "gemm_wt: %zu B of shared memory", smem);
  CUtensorMap tw, tx;
  int rc = wt_tmap(W, (long)(ext && ext->ldw > 0 ? ext->ldw : k_w),
                   grouped ? ext->n_groups * N : (heads && !w_cols ? ext->col_groups * N : (swiglu ? inter : N)),
                   w_cols ? (ext->col_groups - 1) * ext->w_group_cols + k_w : k_w,
                   WT_ROWS, &tw, swiglu);
  if (rc) return rc;
  if ((rc = wt_tmap(X, ldx, T, heads ? ext->x_cols : K, pair ? cfg.TN / 2 : cfg.TN, &tx))) return rc;
  static unsigned long long set_mask = 0ull;
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  if (!(set_mask >> (dev & 63) & 1ull)) {
    B200_CUDA(cudaFuncSetAttribute(gemm_wt_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM_MAX));
    B200_CUDA(cudaFuncSetAttribute(gemm_wt_kernel<false>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
    B200_CUDA(cudaFuncSetAttribute(gemm_wt_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM_MAX));
    B200_CUDA(cudaFuncSetAttribute(gemm_wt_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
    for (auto kern : {gemm_wt_pair_kernel<false, 1>, gemm_wt_pair_kernel<true, 1>, gemm_wt_pair_kernel<false, 2>, gemm_wt_pair_kernel<true, 2>})
      B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM_MAX));
    set_mask |= 1ull << (dev & 63);
  }
  const int row_blocks = swiglu ? cdiv(inter, 64) : cdiv(N, WT_ROWS);
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(row_blocks, cdiv(T, cfg.TN) * (heads ? ext->col_groups : 1), splits);
  lc.blockDim = dim3(256);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = (g_wt_pdl && !grouped) ? 1 : 0;
  if (pair) {
    const int tiles = cdiv(swiglu ? 2 * inter : N, (wide ? 4 : 2) * WT_ROWS) * cdiv(T, cfg.TN) * splits;
    lc.gridDim = dim3(2 * (tiles < WP_PAIRS ? tiles : WP_PAIRS));
    lc.blockDim = dim3(wide ? WP_WIDE_THREADS : WP_THREADS);
    cudaLaunchAttribute pa[2];
    pa[0].id = cudaLaunchAttributeClusterDimension;
    pa[0].val.clusterDim.x = 2;
    pa[0].val.clusterDim.y = pa[0].val.clusterDim.z = 1;
    pa[1] = at[0];
    lc.attrs = pa;
    lc.numAttrs = g_wt_pdl ? 2 : 1;
    const auto kern = wide ? (tower ? gemm_wt_pair_kernel<true, 2> : gemm_wt_pair_kernel<false, 2>)
                           : (tower ? gemm_wt_pair_kernel<true, 1> : gemm_wt_pair_kernel<false, 1>);
    B200_CUDA(cudaLaunchKernelEx(&lc, kern, tw, tx, p));
    return B200_OK;
  }
  if (tower) {
    B200_CUDA(cudaLaunchKernelEx(&lc, gemm_wt_kernel<true>, tw, tx, p));
  } else {
    B200_CUDA(cudaLaunchKernelEx(&lc, gemm_wt_kernel<false>, tw, tx, p));
  }
  return B200_OK;
}

// ---------------------------------------------------------------------------------------------
// Measured configuration choice ("measure, don't guess"): the first call for a problem class
// (tokens rounded up to 64, N, K, mode) times a short list of candidate configurations on the
// caller's stream with the call's own operands (CUDA events, a warm-up and one or two timed replays
// each) and caches the winner; later calls cost one hash lookup.  Candidates follow what that
// sweep showed matters: token tile {96,128,144,192,256}, one CTA per SM with 2 k-blocks
// per stage vs two CTAs per SM with 1, split-K to one or two waves, and CTA pairs.  The list is ordered and
// the first candidate within 3 % of the best wins, so the choice is stable run to run.
// B200_WT_TUNE=0 uses the cost model (gemm_wt_auto) instead.
// ---------------------------------------------------------------------------------------------
// groups: column groups of the product (0: a plain Linear).  They multiply the tiles and take no CTA pairs, so the choice
// of a plain product of the same T, N and K is not one for them.
struct TuneKey {
  int tb, N, K, mode, split_ok, groups, dev;
  bool operator==(const TuneKey& o) const {
    return tb == o.tb && N == o.N && K == o.K && mode == o.mode && split_ok == o.split_ok && groups == o.groups && dev == o.dev;
  }
};
struct TuneHash {
  size_t operator()(const TuneKey& k) const {
    size_t h = (size_t)k.tb;
    for (int v : {k.N, k.K, k.mode, k.split_ok, k.groups, k.dev}) h = h * 1000003u ^ (size_t)v;
    return h;
  }
};

// B200_WT_TUNE_FILE=<path>: measured choices are appended to the file and read back at the first call of a
// later process, so a service does not re-measure at every start and a profiler run (whose serialised
// replays distort the measurement) uses exactly the production configurations.  A line: token bucket, N, K, mode, split
// allowed, TN, KS (0: CTA pairs, -1: wide ones), stages, split, column groups (a line without the last is a plain product's).
static const char* tune_file() {
  static const char* f = getenv("B200_WT_TUNE_FILE");
  return (f && *f) ? f : nullptr;
}

static int tune_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("B200_WT_TUNE");
    v = (e && atoi(e) == 0) ? 0 : 1;
  }
  return v;
}

int gemm_wt_tuned(const void* X, long ldx, const void* W, const void* bias, const void* residual, long ldr,
                  void* C, long ldc, float* partial, long partial_bytes, int T, int N, int K, int epilogue,
                  int mode, int inter, bool allow_split, int sm_count, int* split_out, cudaStream_t st,
                  const WtExt* ext) {
  static std::unordered_map<TuneKey, WtConfig, TuneHash> cache;
  static std::mutex mu;
  const int row_blocks = wt_swiglu(mode) ? cdiv(inter, 64) : cdiv(N, WT_ROWS);
  const int kb_total = cdiv(K, WT_BK);
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  const int groups = ext ? ext->col_groups : 0;
  const TuneKey key{(T + 63) / 64, N, K, mode, allow_split ? 1 : 0, groups, dev};
  WtConfig cfg;
  bool have = false;
  {
    std::lock_guard<std::mutex> g(mu);
    static bool file_read = false;
    if (!file_read) {
      file_read = true;
      if (const char* path = tune_file()) {
        if (FILE* fp = fopen(path, "r")) {
          char line[256];
          while (fgets(line, sizeof line, fp)) {
            int tb, n, k, md, so, tn, ks, stg, sp, g = 0;
            if (sscanf(line, "%d %d %d %d %d %d %d %d %d %d", &tb, &n, &k, &md, &so, &tn, &ks, &stg, &sp, &g) < 9) continue;
            const WtConfig c{tn, ks, stg, sp};   // (a line that no call takes is passed over: its product is measured)
            if (wt_takes(c, k, md, g)) cache[TuneKey{tb, n, k, md, so, g, dev}] = c;
          }
          fclose(fp);
        }
      }
    }
    auto it = cache.find(key);
    if (it != cache.end()) {
      cfg = it->second;
      have = true;
    }
  }
  auto fits = [&](const WtConfig& c) {
    return !(mode == B200_WT_PARTIAL && (long)c.split * T * N * 4 > partial_bytes);
  };
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &cap);
  if (!have && (!tune_enabled() || cap != cudaStreamCaptureStatusNone)) {
    gemm_wt_auto(T, row_blocks, K, allow_split, &cfg, sm_count);
    while (cfg.split > 1 && !fits(cfg)) cfg.split = cdiv(kb_total, cdiv(kb_total, cfg.split - 1));
    have = true;  // not cached: a later un-captured call may still tune
  } else if (!have) {
    // ---- candidate list ----
    std::vector<WtConfig> cand;
    auto add = [&](int tn, int ks, int budget, int split) {
      if (tn > round16(T)) tn = round16(T);
      if (tn > 256) tn = 256;
      const int stage = ks * (WT_WBLK + tn * 128);
      int stg = budget / stage;
      if (stg > 6) stg = 6;
      if (stg < 2) return;
      split = cdiv(kb_total, cdiv(kb_total, split < 1 ? 1 : split));
      WtConfig c{tn, ks, stg, split};
      if (!fits(c)) return;
      for (const auto& o : cand)
        if (o.TN == c.TN && o.KS == c.KS && o.stages == c.stages && o.split == c.split) return;
      cand.push_back(c);
    };
    WtConfig model;
    gemm_wt_auto(T, row_blocks, K, allow_split, &model, sm_count);
    if (fits(model)) cand.push_back(model);
    int tns[8], n_tn = 0;
    if (T <= 96) {
      tns[n_tn++] = round16(T);
      if (T > 48) tns[n_tn++] = round16(cdiv(T, 2));
    } else {
      for (int tn : {144, 96, 192, 128}) tns[n_tn++] = tn;
      if (T > 512) tns[n_tn++] = 256;
    }
    for (int i = 0; i < n_tn; ++i) {
      const int tn = tns[i];
      const long base = (long)row_blocks * cdiv(T, tn);
      int sps[3] = {1, 1, 1};
      if (allow_split) {
        int a = (int)(sm_count / base), b = (int)(2L * sm_count / base);
        const int cap_k = kb_total / 4 > 0 ? kb_total / 4 : 1;
        sps[1] = a < 1 ? 1 : (a > cap_k ? cap_k : a);
        sps[2] = b < 1 ? 1 : (b > cap_k ? cap_k : b);
      }
      // (measured and discarded: restricting the list to <= 110 KB configurations so that the NEXT kernel's prologue
      // can always co-reside under PDL made the prefill of 272 tokens 2-5 % slower)
      for (int sp : sps) {
        add(tn, 2, 208 * 1024, sp);  // one CTA per SM, 256-byte weight-row bursts
        add(tn, 1, 110 * 1024, sp);  // two CTAs per SM
      }
    }
    // CTA pairs (KS = 0) from about a wave of them on: the token tile whose last wave is fullest, the next best, and 256
    if (T >= 192 && !(ext && (ext->tile_group || ext->col_groups > 0))) {
      const int w_rows = wt_swiglu(mode) ? 2 * inter : N, pair_rows = cdiv(w_rows, 2 * WT_ROWS), wide_rows = cdiv(w_rows, 4 * WT_ROWS);
      auto add_pair = [&](int tn, int split, bool wide = false) {
        const int stage = (wide ? 2 : 1) * WT_WBLK + tn * 64;
        int stg = (int)((226 * 1024 - 1024) / stage);
        if (stg > WP_MAX_STAGES) stg = WP_MAX_STAGES;
        split = cdiv(kb_total, cdiv(kb_total, split < 1 ? 1 : split));
        const WtConfig c{tn, wide ? WT_KS_WIDE : 0, stg, split};
        if (!fits(c)) return;
        for (const auto& o : cand)
          if (o.TN == c.TN && o.KS == c.KS && o.split == c.split) return;
        cand.push_back(c);
      };
      int order[5] = {256, 224, 192, 160, 128};
      auto waves_cost = [&](int tn) { return cdiv((long)pair_rows * cdiv(T, tn), WP_PAIRS) * (long)(128 + tn / 2); };
      std::stable_sort(order, order + 5, [&](int a, int b) { return waves_cost(a) < waves_cost(b); });
      for (int tn : {order[0], order[1], 256}) {
        const int base = pair_rows * cdiv(T, tn);
        add_pair(tn, 1);
        if (allow_split && base < WP_PAIRS) add_pair(tn, WP_PAIRS / base);
      }
      // 512 weight rows a pair: for long k (gemm_wt_pair_kernel), from half a wave of them on (fewer leave more than half of the
      // chip idle, and halves of them are there among the candidates above)
      if (mode != B200_WT_PARTIAL && K >= 3072) {
        int worder[3] = {256, 224, 192};
        auto wide_cost = [&](int tn) { return cdiv((long)wide_rows * cdiv(T, tn), WP_PAIRS) * (long)(256 + tn / 2); };
        std::stable_sort(worder, worder + 3, [&](int a, int b) { return wide_cost(a) < wide_cost(b); });
        for (int tn : {worder[0], worder[1]})
          if (2 * wide_rows * cdiv(T, tn) >= WP_PAIRS) add_pair(tn, 1, true);
      }
    }
    if (cand.empty()) {
      gemm_wt_auto(T, row_blocks, K, false, &model, sm_count);
      B200_REQUIRE(fits(model), "gemm_wt: the partial-tile buffer (%ld B) is too small for T=%d N=%d", partial_bytes, T, N);
      cand.push_back(model);
    }
    // ---- time them (the tuning launches never add a residual: the output stays idempotent) ----
    // An output that is also its own residual (h += W.x in place) must not be overwritten by the
    // measurement: those launches write a scratch buffer from the stream-ordered allocator instead.
    WtExt ext_copy;
    const WtExt* ext_t = nullptr;
    float* scratch32 = nullptr;
    void *scratch16 = nullptr, *Ct = C;
    if (mode == B200_WT_BF16 && residual && residual == C) {
      B200_CUDA(cudaMallocAsync(&scratch16, (size_t)T * (size_t)ldc * sizeof(bf16), st));
      Ct = scratch16;
    }
    if (ext) {
      ext_copy = *ext;
      if (mode == B200_WT_F32 && ext->res32 && ext->C32) {
        B200_CUDA(cudaMallocAsync((void**)&scratch32, (size_t)T * (size_t)ext->ldc32 * sizeof(float), st));
        ext_copy.C32 = scratch32;
      }
      ext_copy.res32 = nullptr;
      ext_t = &ext_copy;
    }
    // each candidate is replayed from a small captured graph (16 launches): the measurement sees the
    // kernel back to back with its programmatic dependent launch, not the host's launch overhead.  One replay behind the warm-up where
    // the candidate before took a millisecond for it, else two: a caller waits for all this at the first prompt of a new length (three
    // models of a layer, 17 lengths of 300 - 2048 tokens in all, medians: 7.7 s with the candidates before wide pairs, 7.9 with those,
    // 5.9 so; the chosen products take the same time, 13.3 / 13.2 / 13.1 ms for the second passes together)
    cudaEvent_t e0, e1;
    B200_CUDA(cudaEventCreate(&e0));
    B200_CUDA(cudaEventCreate(&e1));
    std::vector<float> ms(cand.size(), 1e30f);
    int rc = B200_OK;
    constexpr int REP = 16;
    for (size_t i = 0; i < cand.size() && rc == B200_OK; ++i) {
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t gx = nullptr;
      if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        rc = B200_ERR_CUDA;
        break;
      }
      for (int r = 0; r < REP && rc == B200_OK; ++r)
        rc = gemm_wt(X, ldx, W, bias, nullptr, 0, Ct, ldc, partial, T, N, K, epilogue, mode, inter, cand[i], 0, st, ext_t);
      cudaError_t ce = cudaStreamEndCapture(st, &graph);
      if (rc != B200_OK || ce != cudaSuccess || !graph) {
        if (graph) cudaGraphDestroy(graph);
        if (rc == B200_OK) rc = B200_ERR_CUDA;
        break;
      }
      ce = cudaGraphInstantiate(&gx, graph, 0);
      cudaGraphDestroy(graph);
      if (ce != cudaSuccess) {
        rc = B200_ERR_CUDA;
        break;
      }
      const int runs = i > 0 && ms[i - 1] * REP >= 1.f ? 1 : 2;
      cudaGraphLaunch(gx, st);  // warm-up
      cudaEventRecord(e0, st);
      for (int r = 0; r < runs; ++r) cudaGraphLaunch(gx, st);
      cudaEventRecord(e1, st);
      if (cudaEventSynchronize(e1) != cudaSuccess) rc = B200_ERR_CUDA;
      float t = 0.f;
      cudaEventElapsedTime(&t, e0, e1);
      ms[i] = t / (float)(runs * REP);
      cudaGraphExecDestroy(gx);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (scratch32) cudaFreeAsync(scratch32, st);
    if (scratch16) cudaFreeAsync(scratch16, st);
    if (rc) {
      set_error("gemm_wt: configuration measurement failed (T=%d N=%d K=%d mode=%d)", T, N, K, mode);
      return rc;
    }
    // Back to back a pair does not show what it costs in a sequence: all of an SM's shared memory, so the next kernel's set-up
    // and weight loads wait for it, and code of its own to fetch.  It has to win by 8 % (a 2048 x 2048 x 2048 product measured 3 %
    // faster alone and was 4 us of 26 slower between row kernels), or by those 4 us: set-up and code do not grow with the product (with 8 % of
    // everything one-CTA tiles took 4096 x 4096 x 28672 in fp32 at 827 us, where wide pairs take 685).
    for (size_t i = 0; i < cand.size(); ++i)
      if (cand[i].KS <= 0) ms[i] += std::min(0.08f * ms[i], 0.004f);
    float best = 1e30f;
    for (float t : ms) best = t < best ? t : best;
    size_t pick = 0;
    for (size_t i = 0; i < cand.size(); ++i)
      if (ms[i] <= best * 1.03f) {
        pick = i;
        break;
      }
    cfg = cand[pick];
    if (getenv("B200_WT_TUNE_LOG"))
      fprintf(stderr, "[gemm_wt tune] T=%d N=%d K=%d mode=%d -> TN=%d KS=%d stages=%d split=%d (%.1f us, %zu candidates)\n",
              T, N, K, mode, cfg.TN, cfg.KS, cfg.stages, cfg.split, ms[pick] * 1000.f, cand.size());
    std::lock_guard<std::mutex> g(mu);
    cache[key] = cfg;
    if (const char* path = tune_file()) {
      if (FILE* fp = fopen(path, "a")) {
        fprintf(fp, "%d %d %d %d %d %d %d %d %d %d\n", key.tb, key.N, key.K, key.mode, key.split_ok, cfg.TN, cfg.KS,
                cfg.stages, cfg.split, key.groups);
        fclose(fp);
      }
    }
  }
  // a cached configuration was tuned for a token count in the same 64-bucket: re-check the bounds
  if (cfg.TN > round16(T) && cfg.KS > 0) cfg.TN = round16(T);
  while (cfg.split > 1 && !fits(cfg)) cfg.split = cdiv(kb_total, cdiv(kb_total, cfg.split - 1));
  B200_REQUIRE(fits(cfg), "gemm_wt: the partial-tile buffer (%ld B) is too small for T=%d N=%d", partial_bytes, T, N);
  if (split_out) *split_out = cfg.split;
  return gemm_wt(X, ldx, W, bias, residual, ldr, C, ldc, partial, T, N, K, epilogue, mode, inter, cfg, 0, st, ext);
}

int finish_rows(const float* P, int S, const void* bias, const void* resid, long ldr, void* h_out,
                long ldh, int norm_kind, const void* nw, const void* nb, float eps, void* xn, long ldx,
                int T, int N, cudaStream_t st) {
  B200_REQUIRE(P && S >= 1 && T > 0 && N > 0 && (N % 4) == 0 && N <= FIN_N_MAX,
               "finish_rows: T=%d N=%d S=%d", T, N, S);
  B200_REQUIRE(norm_kind == B200_NORM_NONE || (xn && (norm_kind != B200_NORM_RMS || nw)),
               "finish_rows: norm output / weight missing");
  B200_REQUIRE((ldr % 4) == 0 && (ldh % 4) == 0 && (ldx % 4) == 0, "finish_rows: strides must be multiples of 4");
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(T);
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = g_wt_pdl ? 1 : 0;
  auto go = [&](auto kern, int threads) {
    lc.blockDim = dim3(threads);
    return cudaLaunchKernelEx(&lc, kern, P, S, (const bf16*)bias, (const bf16*)resid, ldr, (bf16*)h_out, ldh, norm_kind, (const bf16*)nw,
                              (const bf16*)nb, eps, (bf16*)xn, ldx, T, N);
  };
  if (T <= 32) B200_CUDA(N <= 4096 ? go(finish_rows_kernel<1024, 1>, 1024) : go(finish_rows_kernel<1024, 2>, 1024));
  else if (N <= 1536) B200_CUDA(go(finish_rows_kernel<384, 1>, 384));
  else if (N <= 4096) B200_CUDA(go(finish_rows_kernel<512, 2>, 512));
  else B200_CUDA(go(finish_rows_kernel<512, 4>, 512));
  return B200_OK;
}

}  // namespace b200

// ---- C ABI ------------------------------------------------------------------
using namespace b200;
extern "C" {

/* explicit-configuration entry (benchmark sweeps, tests): cfg = {TN, KS, stages, split}; a 0 in
 * cfg[0] asks for the automatic choice.  partial: fp32 [split][T][N] (mode B200_WT_PARTIAL). */
int b200_gemm_wt(const void* X, long ldx, const void* W, const void* bias, const void* residual,
                 long ldr, void* C, long ldc, float* partial, int T, int N, int K, int epilogue,
                 int mode, int inter, const int* cfg4, unsigned flags, void* stream) {
  WtConfig c;
  if (cfg4 && cfg4[0] > 0) {
    c.TN = cfg4[0]; c.KS = cfg4[1]; c.stages = cfg4[2]; c.split = cfg4[3];
    B200_REQUIRE(c.KS >= 1, "gemm_wt: bad config KS=%d", c.KS);
    if (flags & B200_WT_FLAG_PAIR) c.KS = 0;
    if (flags & B200_WT_FLAG_WIDE) c.KS = WT_KS_WIDE;
  } else {
    const int rbs = mode == B200_WT_SWIGLU ? cdiv(inter, 64) : cdiv(N, 128);
    gemm_wt_auto(T, rbs, K, mode == B200_WT_PARTIAL, &c, 148);
  }
  return gemm_wt(X, ldx, W, bias, residual, ldr, C, ldc, partial, T, N, K, epilogue, mode, inter, c,
                 flags, (cudaStream_t)stream);
}

int b200_finish_rows(const float* P, int S, const void* bias, const void* resid, long ldr, void* h_out,
                     long ldh, int norm_kind, const void* nw, const void* nb, float eps, void* xn,
                     long ldx, int T, int N, void* stream) {
  return finish_rows(P, S, bias, resid, ldr, h_out, ldh, norm_kind, nw, nb, eps, xn, ldx, T, N,
                     (cudaStream_t)stream);
}

int b200_gemm_wt_auto_config(int T, int N, int K, int mode, int inter, int* cfg4_out) {
  WtConfig c;
  const int rbs = mode == B200_WT_SWIGLU ? cdiv(inter, 64) : cdiv(N, 128);
  gemm_wt_auto(T, rbs, K, mode == B200_WT_PARTIAL, &c, 148);
  cfg4_out[0] = c.TN; cfg4_out[1] = c.KS; cfg4_out[2] = c.stages; cfg4_out[3] = c.split;
  return B200_OK;
}
}
