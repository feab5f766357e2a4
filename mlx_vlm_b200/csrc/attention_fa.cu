// Prefill / vision attention, pipelined: TMA-fed, warp-specialised, tcgen05 with double-buffered
// score tiles in TMEM.  Same arithmetic and rounding points as attention_tc.cu (the reference's
// mlx-CPU SDPA: oracle/mlx_semantics.py::sdpa; models/base.py:305-373, qwen2_vl/vision.py:154):
//     qs = bf16(q * bf16(scale))       -- done by the rotary kernels that already touch q
//     s  = bf16(qs . k^T);  p = bf16(softmax_fp32(s));  o = bf16(p . v)
// p is rounded AFTER normalisation with the final row max / sum, so the kernel is two-pass over
// the keys and the second pass recomputes the score tile on the tensor cores.
//
// attention_tc.cu stages every tile with the compute threads and runs
// load -> sync -> MMA -> wait -> softmax strictly in sequence (61 us per ViT layer, 2 % of the
// tensor peak).  Here, per CTA = 128 query rows of one head:
//   warp 0      TMA producer: Q once, K tiles for both passes, V tiles for pass 2 (3-D tensor
//               maps over the packed qkv buffer / the KV cache, 128B swizzle, zero-filled tails)
//   warps 1, 18 issue S[i % 2] = Qs . K^T of the even / odd steps (M128 x N128, TMEM cols 0..255)
//   warp 19     issues O += P . V (M128 x N=hd, TMEM cols 256..).  Three threads, because a thread that waits does not issue:
//               the waits of one product (0.2 us of 0.5, ready or not) pass while another thread's keeps the tensor core busy
//   warps 2..17 softmax: two groups of eight warps that take the key tiles in turn, each with a score tile and a P tile
//               of its own; two threads per query row (64 score columns each), TMEM -> registers,
//               pass 1: running max / sum of exp;  pass 2: p -> tensor memory (the A operand)
// V is read as it lies in the qkv buffer or the KV cache ([key][dim]): the B operand of P.V is then MN-major (dims
// contiguous), which tcgen05 takes from the same 128-byte-swizzled 64-dim blocks that K uses.  So nothing transposes V:
// a segment may start at any token (keys are a TMA coordinate without an alignment rule) and a later portion of a prompt
// reads the cached keys and values where they are.  (V^T, [head][dim][key], is still taken by b200_attention_fa.)
// A tile's time, from clock stamps (28 heads of 128): 1280 cycles in pass 1, of which the exponentials' 1024 are one part and
// the two groups' loads and waits, which fall together, the other; 1350 in pass 2, where the thread that issues P.V is the
// chain: 8 products of 64 cycles beside Q.K^T's, a wait for P and one for V.  P in tensor memory instead of shared memory, one
// commit for the value slot and the P tile, half tiles that a warp's rows do not see left out, and waits that ask once before
// they suspend, together (the kernel alone, cold L2): 2048 queries behind 2048 keys, 28 heads, 190.5 -> 186.4 us; 8 prompts of
// 608, 32 heads, 129.0 -> 127.0; four pictures and a clip (6012 patches, 16 heads of 80) 146.2 -> 143.4.
// Measured against the kernel without TMA that such calls fell back to (attention_tc.cu): 2048 queries behind 2048 cached
// keys, 28 heads of 128: 1094 -> 354 us (249 with the pairwise softmax below); four pictures and a clip of four frames (6012
// patches, 16 heads of 80), which start at odd offsets: 773 us in eight launches -> 236 us in one.
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "decode.cuh"

namespace b200 {

namespace {

constexpr int FA_TQ = 128, FA_TK = 128;
constexpr int FA_BLK = 16 * 1024;       // one 128-row x 64-column bf16 operand block
constexpr int FA_THREADS = 640;         // producer warp, 3 MMA warps, 2 groups of 8 softmax warps
constexpr int FA_NK = 2, FA_NV = 2;     // ring slots of key and of value tiles (a value slot and a P tile are free at the same time)
// A key slot belongs to one of the two threads that issue Q.K^T.  With an odd number of slots both would use each in turn, and a
// thread that waits for the round after next would take the parity of a round long past for it: it has to see every round.
static_assert(FA_NK % 2 == 0, "a slot's waiter sees every round of it");
constexpr uint32_t FA_O0 = 256, FA_P0 = 384;   // TMEM columns: scores 2 x 128 | O 128 | P 2 x 64 (two bf16 a column)

struct FaParams {
  bf16* out;
  long o_ts;
  int n_heads, n_kv, hd, hdp, Lq, S, causal;
  int q0, k0;  // token offsets of this segment inside the tensors the maps describe
  const int4* segs;  // optional [gridDim.z]: (q0, Lq, k0, S) of segment blockIdx.z — several independent sequences of one
                     // concatenated batch in ONE launch (the tail wave of a 160-CTA launch per sequence idles half the SMs)
  int flags;
};

struct FaBars {
  uint64_t q_full, k_full[FA_NK], k_empty[FA_NK], v_full[FA_NV], s_full[2], s_empty[2], p_full[2], pv_done[2], o_full, dropped, drained[3];
};

__device__ __forceinline__ uint32_t f_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void f_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(f_u32(bar)), "r"(count));
}
__device__ __forceinline__ void f_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(f_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void f_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(f_u32(bar)) : "memory");
}
__device__ int g_fa_wait_failed;   // a wait of attention_fa_kernel ran out: B200_WAIT_ATTENTION

__device__ __forceinline__ void f_tma_3d(void* dst, const CUtensorMap* tmap, uint64_t* bar, int c0, int c1,
                                         int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(f_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(f_u32(bar))
      : "memory");
}
__device__ __forceinline__ void f_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void f_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void f_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void f_umma(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// A (here P) in tensor memory
__device__ __forceinline__ void f_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void f_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void f_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(f_u32(bar))
               : "memory");
}
__device__ __forceinline__ uint32_t f_desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
// MN-major with the 128-byte swizzle: 64-element blocks along MN are FA_BLK bytes apart (the leading offset), groups of 8
// along K 1024 bytes (the stride offset in F_DESC_HI)
__device__ __forceinline__ uint32_t f_desc_lo_mn(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | ((uint32_t)(FA_BLK >> 4) << 16); }
constexpr uint32_t F_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);

// (its values may be used after f_ld_wait)
__device__ __forceinline__ void f_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void f_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
// 64 scores of a row, rounded to bf16, two to a register; those from column `vis` on are -inf
__device__ __forceinline__ void f_scores(uint32_t taddr, int vis, uint32_t (&pk)[32]) {
  uint32_t v[2][16];
  f_ld16(taddr, v[0]);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t(&x)[16] = v[c & 1];
    f_ld_wait(x);
    if (c < 3) f_ld16(taddr + (uint32_t)(c + 1) * 16, v[(c + 1) & 1]);
    if (__any_sync(0xffffffffu, vis < c * 16 + 16)) {
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] = c * 16 + e < vis ? x[e] : 0xff800000u;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) pk[c * 8 + e] = pack2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1]));
  }
}
__device__ __forceinline__ uint32_t f_max2(uint32_t a, uint32_t b) {   // of bf16 pairs
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint64_t f_pair(uint32_t x) { return f2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
__device__ __forceinline__ void f_tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void f_sbar() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
// 2^x on the SFU (one MUFU instruction, rel. error 2^-22: far below the bf16 rounding of p that follows)
__device__ __forceinline__ float f_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// VT: V arrives transposed (K-major B operand), else as [key][dim] rows (MN-major B operand)
template <bool VT>
__global__ void __launch_bounds__(FA_THREADS, 1)
attention_fa_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const FaParams p_in) {
  FaParams p = p_in;
  if (p_in.segs) {   // static table (written before the producing kernels ran): safe to read ahead of griddepcontrol.wait
    const int4 sg = __ldg(p_in.segs + blockIdx.z);
    p.q0 = sg.x; p.Lq = sg.y; p.k0 = sg.z; p.S = sg.w;
    if ((int)(p.causal ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * FA_TQ >= p.Lq) return;   // sized for the longest segment
  }
  extern __shared__ uint8_t fa_smem_raw[];
  __shared__ FaBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fa_smem_raw) + 1023) &
                                           ~static_cast<uintptr_t>(1023));
  uint8_t* Qs = sm;                          // [128 q][128 d]            2 k-blocks
  uint8_t* Ks = sm + 2 * FA_BLK;             // FA_NK slots x [128 keys][128 d]
  uint8_t* Vs = Ks + 2 * FA_NK * FA_BLK;     // FA_NV slots x (VT: 2 key-blocks x [hdp d][64 keys], else 2 dim-blocks x [128 keys][64 d])
  float2* stat = reinterpret_cast<float2*>(Vs + 2 * FA_NV * FA_BLK);   // [2 groups x 2 halves][128 q], between the passes
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, kvh = h / (p.n_heads / p.n_kv);
  // causal: the query tiles with the most keys start first, of all heads, so that the short ones fill the last wave
  const int row0 = (p.causal ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * FA_TQ;
  const int S = p.S;
  const int q_last = min(row0 + FA_TQ, p.Lq) - 1;
  const int vis_tile = p.causal ? min(S, S - p.Lq + q_last + 1) : S;
  const int n_tiles = (vis_tile + FA_TK - 1) / FA_TK;
  const int kbq = (p.hdp + 63) >> 6;         // 64-column blocks of the head dimension
  const int vblk = p.hdp * 128;              // bytes of one 64-key block of a V^T tile

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmQ)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
    f_init(&bars.q_full, 1);
    for (int i = 0; i < FA_NK; ++i) {
      f_init(&bars.k_full[i], 1);
      f_init(&bars.k_empty[i], 1);
    }
    for (int i = 0; i < FA_NV; ++i) f_init(&bars.v_full[i], 1);
    for (int i = 0; i < 2; ++i) {
      f_init(&bars.s_full[i], 1);
      f_init(&bars.s_empty[i], 256);
      f_init(&bars.p_full[i], 256);
      f_init(&bars.pv_done[i], 1);
    }
    f_init(&bars.o_full, 1);
    f_init(&bars.dropped, 1);
    for (int i = 0; i < 3; ++i) f_init(&bars.drained[i], 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(f_u32(&tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  f_fence_before();
  __syncthreads();
  f_fence_after();
  const uint32_t tmem = tmem_slot;
  // (the next kernel may start from here on, not before: it may ask for tensor memory too, and would hold what this one still needs)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int k_loads = 0, v_loads = 0;   // of the producer

  if (warp == 0) {
    if (lane == 0 && !(p.flags & 1)) {  // ===== TMA producer (flags 1: no loads, every wait for them runs out) =====
      f_expect_tx(&bars.q_full, (uint32_t)kbq * FA_BLK);
      for (int c = 0; c < kbq; ++c) f_tma_3d(Qs + c * FA_BLK, &tmQ, &bars.q_full, c * 64, h, p.q0 + row0);
      auto load_v = [&](int j) {
        const int sv = j & 1;
        if (!mbar_wait(&bars.pv_done[sv], ((j >> 1) & 1) ^ 1, &failed)) return false;
        ++v_loads;
        if constexpr (VT) {
          f_expect_tx(&bars.v_full[sv], 2u * (uint32_t)vblk);
          for (int c = 0; c < 2; ++c)
            f_tma_3d(Vs + sv * 2 * FA_BLK + c * vblk, &tmV, &bars.v_full[sv], p.k0 + j * FA_TK + c * 64, 0, kvh);
        } else {
          f_expect_tx(&bars.v_full[sv], (uint32_t)kbq * FA_BLK);
          for (int c = 0; c < kbq; ++c)
            f_tma_3d(Vs + sv * 2 * FA_BLK + c * FA_BLK, &tmV, &bars.v_full[sv], c * 64, kvh, p.k0 + j * FA_TK);
        }
        return true;
      };
      int jk = 0;   // key tile of step i
      bool ok = true;
      int s = 0;
      uint32_t free_par = 1;
      for (int i = 0; i < 2 * n_tiles && ok; ++i) {
        if (!(ok = mbar_wait(&bars.k_empty[s], free_par, &failed))) break;
        ++k_loads;
        f_expect_tx(&bars.k_full[s], (uint32_t)kbq * FA_BLK);
        for (int c = 0; c < kbq; ++c)
          f_tma_3d(Ks + s * 2 * FA_BLK + c * FA_BLK, &tmK, &bars.k_full[s], c * 64, kvh, p.k0 + jk * FA_TK);
        if (++jk == n_tiles) jk = 0;
        if (++s == FA_NK) s = 0, free_par ^= 1;
        if (i >= n_tiles + 2) ok = load_v(i - n_tiles - 2);   // (in the order of the products: a wait for V holds up no K before it)
      }
      for (int j = max(0, n_tiles - 2); j < n_tiles && ok; ++j) ok = load_v(j);
    }
  } else if (warp == 1 || warp == 18) {
    if (lane == 0) {  // ===== issuer of Q.K^T, of every other step =====
      const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FA_TK >> 3) << 17) | (8u << 24);
      const int ksteps = p.hdp >> 4, s = warp == 1 ? 0 : 1;
      const uint32_t q_lo = f_desc_lo(f_u32(Qs)), k_first = f_desc_lo(f_u32(Ks)), d = tmem + (uint32_t)s * 128u;
      bool dead = false;
      int sk = s;           // ring slot of step i and the parity of its round
      uint32_t k_par = 0;
      mbar_wait_issuer(&bars.q_full, 0, dead);
      for (int i = s; i < 2 * n_tiles; i += 2) {
        const uint32_t k_lo = k_first + (uint32_t)(sk * 2 * (FA_BLK >> 4));
        mbar_wait_issuer(&bars.k_full[sk], k_par, dead);
        mbar_wait_issuer(&bars.s_empty[s], ((i >> 1) & 1) ^ 1, dead);
        f_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          if (ks >= ksteps) break;
          const uint32_t off = (uint32_t)((ks >> 2) * (FA_BLK >> 4) + (ks & 3) * 2);
          f_umma(d, q_lo + off, k_lo + off, F_DESC_HI, idesc_s, ks > 0 ? 1u : 0u);
        }
        f_commit(dead ? &bars.dropped : &bars.k_empty[sk]);
        f_commit(dead ? &bars.dropped : &bars.s_full[s]);
        if ((sk += 2) >= FA_NK) sk -= FA_NK, k_par ^= 1;
      }
      if (dead) *static_cast<volatile int*>(&failed) = 1;
    }
  } else if (warp == 19) {
    if (lane == 0) {  // ===== issuer of P.V =====
      // (bit 16: the B operand is MN-major)
      const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (VT ? 0u : 1u << 16) | ((uint32_t)(p.hdp >> 3) << 17) |
                               (8u << 24);
      bool dead = false;
      for (int j = 0; j < n_tiles; ++j) {
        const int sv = j & 1, sp = (n_tiles + j) & 1;
        const uint32_t p_at = tmem + FA_P0 + (uint32_t)sp * 64u;
        const uint32_t v_lo = VT ? f_desc_lo(f_u32(Vs + sv * 2 * FA_BLK)) : f_desc_lo_mn(f_u32(Vs + sv * 2 * FA_BLK));
        mbar_wait_issuer(&bars.v_full[sv], (j >> 1) & 1, dead);
        mbar_wait_issuer(&bars.p_full[sp], (j >> 1) & 1, dead);
        f_fence_after();
        // (groups of 16 keys that lie wholly behind the segment's last key are left out)
        const int ks_n = VT ? FA_TK / 16 : min(FA_TK / 16, (S - j * FA_TK + 15) >> 4);
#pragma unroll
        for (int ks = 0; ks < FA_TK / 16; ++ks) {
          if (ks >= ks_n) break;
          // VT: 32 bytes along a 64-key row; else 16 rows of 128 bytes
          const uint32_t b = VT ? v_lo + (uint32_t)((ks >> 2) * (vblk >> 4) + (ks & 3) * 2) : v_lo + (uint32_t)(ks * (2048 >> 4));
          f_umma_ts(tmem + FA_O0, p_at + (uint32_t)(ks * 8), b, F_DESC_HI, idesc_o, (j > 0 || ks > 0) ? 1u : 0u);
        }
        f_commit(dead ? &bars.dropped : &bars.pv_done[sv]);   // frees the value slot and the P tile
      }
      f_commit(dead ? &bars.dropped : &bars.o_full);   // (an output that is not whole is not handed over)
      if (dead) *static_cast<volatile int*>(&failed) = 1;
    }
  } else {
    // ===== softmax warps: thread = (group, query row, score-column half) =====
    const int q4 = warp & 3, half = ((warp - 2) >> 2) & 1, grp = (warp - 2) >> 3;
    const int row = q4 * 32 + lane;
    const int qi = row0 + row;
    const int vis = p.causal ? min(S, S - p.Lq + min(qi, p.Lq - 1) + 1) : S;   // (rows behind the last query repeat it)
    const int vis_most = __shfl_sync(0xffffffffu, vis, 31);                     // of the warp's rows
    const uint32_t t_row = tmem + ((uint32_t)(q4 * 32) << 16);
    constexpr float LOG2E = 1.4426950408889634f;
    // The softmax warps bound the kernel (two warps per scheduler, 64 scores per thread and pass), so they work on pairs: one
    // cvt rounds two scores, the maximum is taken of bf16 pairs, exponents and sums are f32x2 operations, 4 instructions per
    // score; the tensor-memory loads of the next 16 columns are in flight meanwhile, and the score tile is free for the next
    // product as soon as it is in registers.  What is left is the SFU: 128 x 128 exponentials at 16 a cycle per pass.
    // Measured (element by element -> pairs, with the long query tiles first): 2048 queries behind 2048 keys, 28 heads of
    // 128: 354 -> 249 us; 8 prompts of about 608 tokens, 32 heads of 128: 154 -> 130; 576 patches, 16 heads of 80: 24 -> 19.
    // Two groups of warps, one exponentiating while the other waits, loads and rounds: two layers of the first 2220 -> 2175 us,
    // two vision blocks on 6012 patches (16 heads of 80) 1098 -> 1082; with an issuer for each product 2111 and 1053.
    const uint64_t log2e = f2(LOG2E, LOG2E);
    uint32_t pk[32];
    float m = -INFINITY, l = 0.f;
    bool ok = true;   // (the same in a warp)
    for (int i = grp; i < n_tiles; i += 2) {  // ---- pass 1: row max and sum of exp over bf16 scores ----
      const int s = grp;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.s_full[s], (i >> 1) & 1, &failed));
      if (!ok) break;
      f_fence_after();
      // (half tiles that no row of the warp sees, a third of a diagonal tile: nothing to add)
      const bool any = vis_most > i * FA_TK + half * 64;
      if (any) f_scores(t_row + (uint32_t)(s * 128 + half * 64), vis - (i * FA_TK + half * 64), pk);
      f_fence_before();
      f_arrive(&bars.s_empty[s]);
      if (!any) continue;
      uint32_t mx = pk[0];
#pragma unroll
      for (int e = 1; e < 32; ++e) mx = f_max2(mx, pk[e]);
      const float cm = fmaxf(__uint_as_float(mx << 16), __uint_as_float(mx & 0xffff0000u));
      if (cm > -INFINITY) {
        const float mn = fmaxf(m, cm);
        const uint64_t nb = f2(-mn * LOG2E, -mn * LOG2E);
        uint64_t add[2] = {0ull, 0ull};
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const uint64_t x = fma2(f_pair(pk[e]), log2e, nb);
          add[e & 1] = add2(add[e & 1], f2(f_ex2(f2_lo(x)), f_ex2(f2_hi(x))));
        }
        add[0] = add2(add[0], add[1]);
        l = l * f_ex2((m - mn) * LOG2E) + (f2_lo(add[0]) + f2_hi(add[0]));
        m = mn;
      }
    }
    stat[(2 * grp + half) * FA_TQ + row] = make_float2(m, l);
    f_sbar();
    {
      float2 a[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = stat[e * FA_TQ + row];
      m = fmaxf(fmaxf(a[0].x, a[1].x), fmaxf(a[2].x, a[3].x));
      l = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) l += a[e].y > 0.f ? a[e].y * f_ex2((a[e].x - m) * LOG2E) : 0.f;
    }
    const float inv_l = 1.0f / l;
    const uint64_t nbm = f2(-m * LOG2E, -m * LOG2E), inv2 = f2(inv_l, inv_l);
    for (int j = (n_tiles ^ grp) & 1; j < n_tiles && ok; j += 2) {  // ---- pass 2: p = bf16(exp(s - m) / l) -> tensor memory ----
      const int i = n_tiles + j, s = grp;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.s_full[s], (i >> 1) & 1, &failed));
      if (!ok) break;
      f_fence_after();
      const bool any = vis_most > j * FA_TK + half * 64;
      if (any) f_scores(t_row + (uint32_t)(s * 128 + half * 64), vis - (j * FA_TK + half * 64), pk);
      f_fence_before();
      f_arrive(&bars.s_empty[s]);
      if (any) {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const uint64_t x = fma2(f_pair(pk[e]), log2e, nbm);
          const uint64_t w = mul2(f2(f_ex2(f2_lo(x)), f_ex2(f2_hi(x))), inv2);
          pk[e] = pack2(f2_lo(w), f2_hi(w));
        }
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) pk[e] = 0u;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.pv_done[j & 1], ((j >> 1) & 1) ^ 1, &failed));  // the group's previous P.V has consumed the P tile
      if (!ok) break;
      f_fence_after();
      f_st16(t_row + FA_P0 + (uint32_t)(s * 64 + half * 32), pk);
      f_st16(t_row + FA_P0 + (uint32_t)(s * 64 + half * 32 + 16), pk + 16);
      if constexpr (!VT) {
        // V rows behind the segment's last key (another segment's, or a cache's unused rows) meet p = 0, but 0 times a NaN
        // or an infinity would still reach O: those of the last group of 16 keys that is multiplied are cleared
        const int first = S - j * FA_TK, end = (first + 15) & ~15;
        if (first < FA_TK && first != end) {
          ok = __all_sync(0xffffffffu, mbar_wait(&bars.v_full[j & 1], (j >> 1) & 1, &failed));
          if (!ok) break;
          const int per = kbq * 8;
          for (int idx = (threadIdx.x - 64) & 255; idx < (end - first) * per; idx += 256) {
            const int r = first + idx / per, ch = idx % per;
            *reinterpret_cast<uint4*>(Vs + (j & 1) * 2 * FA_BLK + (ch >> 3) * FA_BLK + r * 128 + (ch & 7) * 16) =
                make_uint4(0, 0, 0, 0);
          }
          f_fence_async();  // generic-proxy writes -> visible to the tensor core (async proxy)
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      f_fence_before();
      f_arrive(&bars.p_full[s]);
    }
    // ---- epilogue: O row -> bf16 -> global (16-column chunks go round the row's four threads) ----
    ok = ok && __all_sync(0xffffffffu, mbar_wait(&bars.o_full, 0, &failed));
    f_fence_after();
    bf16* orow = p.out + (long)(p.q0 + qi) * p.o_ts + (long)h * p.hd;
    for (int c0 = 16 * (2 * grp + half); c0 < p.hd; c0 += 64) {
      uint32_t r[16];
      f_tmem_ld16(t_row + FA_O0 + (uint32_t)c0, r);
      if (!ok)
        for (int e = 0; e < 16; ++e) r[e] = 0x7FC00000u;
      if (qi < p.Lq) {
        if (c0 + 16 <= p.hd) {
          uint4 o0, o1;
          o0.x = pack2(__uint_as_float(r[0]), __uint_as_float(r[1]));
          o0.y = pack2(__uint_as_float(r[2]), __uint_as_float(r[3]));
          o0.z = pack2(__uint_as_float(r[4]), __uint_as_float(r[5]));
          o0.w = pack2(__uint_as_float(r[6]), __uint_as_float(r[7]));
          o1.x = pack2(__uint_as_float(r[8]), __uint_as_float(r[9]));
          o1.y = pack2(__uint_as_float(r[10]), __uint_as_float(r[11]));
          o1.z = pack2(__uint_as_float(r[12]), __uint_as_float(r[13]));
          o1.w = pack2(__uint_as_float(r[14]), __uint_as_float(r[15]));
          *reinterpret_cast<uint4*>(orow + c0) = o0;
          *reinterpret_cast<uint4*>(orow + c0 + 8) = o1;
        } else {
          for (int e = 0; e < 16 && c0 + e < p.hd; ++e) orow[c0 + e] = f2bf(__uint_as_float(r[e]));
        }
      }
    }
  }
  f_fence_before();
  __syncthreads();
  if (failed) {   // nothing is left in flight: the last loads of every slot, the products of each issuer
    if (lane == 0 && (warp < 2 || warp >= 18)) {
      if (warp == 0) {
        g_fa_wait_failed = B200_WAIT_ATTENTION;
        if (!(p.flags & 1)) mbar_drain(&bars.q_full, 0);
        for (int i = max(0, k_loads - FA_NK); i < k_loads; ++i) mbar_drain(&bars.k_full[i % FA_NK], (i / FA_NK) & 1);
        for (int i = max(0, v_loads - FA_NV); i < v_loads; ++i) mbar_drain(&bars.v_full[i % FA_NV], (i / FA_NV) & 1);
      } else {
        uint64_t* mine = &bars.drained[warp == 1 ? 0 : warp - 17];
        f_commit(mine);
        mbar_drain(mine, 0);
      }
    }
    __syncthreads();
  }
  if (warp == 1) {
    f_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- host: 3-D tensor maps ----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn fa_get_encode() {
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
struct FaKey {
  const void* ptr;
  long s1, s2;
  int d0, d1, d2, b0, b1, b2;
  bool operator==(const FaKey& o) const {
    return ptr == o.ptr && s1 == o.s1 && s2 == o.s2 && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && b0 == o.b0 &&
           b1 == o.b1 && b2 == o.b2;
  }
};
struct FaHash {
  size_t operator()(const FaKey& k) const {
    size_t h = std::hash<const void*>()(k.ptr);
    for (long v : {k.s1, k.s2, (long)k.d0, (long)k.d1, (long)k.d2, (long)k.b0, (long)k.b1, (long)k.b2})
      h = h * 1000003u ^ std::hash<long>()(v);
    return h;
  }
};
// bf16 tensor: dims (d0 contiguous, d1 with stride s1 elements, d2 with stride s2), box (b0, b1, b2)
int fa_tmap3(const void* ptr, int d0, int d1, long s1, int d2, long s2, int b0, int b1, int b2, CUtensorMap* out) {
  static std::unordered_map<FaKey, CUtensorMap, FaHash> cache;
  static std::mutex mu;
  FaKey key{ptr, s1, s2, d0, d1, d2, b0, b1, b2};
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return B200_OK;
    }
  }
  EncodeTiledFn enc = fa_get_encode();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled unavailable");
    return B200_ERR_CUDA;
  }
  cuuint64_t gdim[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
  cuuint64_t gstr[2] = {(cuuint64_t)s1 * 2, (cuuint64_t)s2 * 2};
  cuuint32_t box[3] = {(cuuint32_t)b0, (cuuint32_t)b1, (cuuint32_t)b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap tm;
  CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), gdim, gstr, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled(3d) failed (%d) ptr=%p dims=(%d,%d,%d) strides=(%ld,%ld) box=(%d,%d,%d)", (int)r,
              ptr, d0, d1, d2, s1, s2, b0, b1, b2);
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

}  // namespace

static WaitWord g_fa_wait_word([](int* v) -> int {
  B200_CUDA(cudaMemcpyFromSymbol(v, g_fa_wait_failed, sizeof(int)));
  return B200_OK;
});

// v: V^T (strides head, dim) or V rows (strides token, head): the same alignment rules
bool attention_fa_supported(const void* q, long q_ts, long q_hs, const void* k, long k_ts, long k_hs,
                            const void* vt, long vt_hs, long vt_ds, const void* out, long o_ts, int hd) {
  auto al = [](const void* p) { return ((uintptr_t)p & 15) == 0; };
  return hd % 8 == 0 && hd >= 16 && hd <= 128 && al(q) && al(k) && al(vt) && al(out) && (q_ts % 8) == 0 &&
         (q_hs % 8) == 0 && (k_ts % 8) == 0 && (k_hs % 8) == 0 && (vt_hs % 8) == 0 && (vt_ds % 8) == 0 &&
         (o_ts % 8) == 0;
}

// q: PRE-SCALED queries (bf16(q * bf16(scale))), element (t, h, d) at q + t*q_ts + h*q_hs + d
// k: keys, element (s, kvh, d) at k + s*k_ts + kvh*k_hs + d
// v: values like the keys, element (s, kvh, d) at v + s*v_s0 + kvh*v_s1 + d; v_transposed: element (kvh, d, s) at
//    v + kvh*v_s0 + d*v_s1 + s (keys contiguous; k0 a multiple of 8: TMA starts on 16-byte boundaries)
// The tensors hold q_tot query tokens / k_tot keys; this call attends queries [q0, q0+Lq) to keys
// [k0, k0+S) (or, segs: a device table of (q0, Lq, k0, S) per segment, Lq / S then the longest of them); out row t is
// written at out + t*o_ts.
int attention_fa(const void* q, long q_ts, long q_hs, const void* k, long k_ts, long k_hs, const void* v,
                 long v_s0, long v_s1, void* out, long o_ts, int n_heads, int n_kv, int hd, int Lq, int S,
                 int causal, cudaStream_t st, int q0, int q_tot, int k0, int k_tot, const void* segs, int n_seg,
                 bool v_transposed, int flags) {
  if (q_tot <= 0) q_tot = q0 + Lq;
  if (k_tot <= 0) k_tot = k0 + S;
  B200_REQUIRE(!segs || n_seg > 0, "attention_fa: segment table without segments");
  B200_REQUIRE(attention_fa_supported(q, q_ts, q_hs, k, k_ts, k_hs, v, v_s0, v_s1, out, o_ts, hd),
               "attention_fa: unsupported layout (hd=%d)", hd);
  B200_REQUIRE(Lq > 0 && S > 0 && n_heads % n_kv == 0, "attention_fa: bad shape");
  const int hdp = (hd + 15) & ~15;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = fa_tmap3(q, hd, n_heads, q_hs, q_tot, q_ts, 64, 1, FA_TQ, &tq))) return rc;
  if ((rc = fa_tmap3(k, hd, n_kv, k_hs, k_tot, k_ts, 64, 1, FA_TK, &tk))) return rc;
  if (v_transposed) rc = fa_tmap3(v, k_tot, hd, v_s1, n_kv, v_s0, 64, hdp, 1, &tv);
  else rc = fa_tmap3(v, hd, n_kv, v_s1, k_tot, v_s0, 64, 1, FA_TK, &tv);
  if (rc) return rc;
  const auto kern = v_transposed ? attention_fa_kernel<true> : attention_fa_kernel<false>;
  static unsigned long long set_mask[2] = {0ull, 0ull};
  const size_t smem = (2 + 2 * FA_NK + 2 * FA_NV) * FA_BLK + 4 * FA_TQ * sizeof(float2) + 1024;
  if (FirstUse first{&set_mask[v_transposed]})
    B200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  FaParams p;
  p.out = (bf16*)out; p.o_ts = o_ts; p.n_heads = n_heads; p.n_kv = n_kv; p.hd = hd; p.hdp = hdp;
  p.Lq = Lq; p.S = S; p.causal = causal; p.q0 = q0; p.k0 = k0;
  p.segs = (const int4*)segs;
  p.flags = flags;
  B200_CUDA(launch_pdl(kern, dim3(n_heads, cdiv(Lq, FA_TQ), segs ? n_seg : 1), dim3(FA_THREADS), smem, st, tq, tk, tv, p));
  return B200_OK;
}

}  // namespace b200

extern "C" int b200_attention_fa(const void* q, long q_ts, long q_hs, const void* k, long k_ts, long k_hs,
                                 const void* vt, long vt_hs, long vt_ds, void* out, long o_ts, int n_heads,
                                 int n_kv, int hd, int Lq, int S, int causal, void* stream) {
  return b200::attention_fa(q, q_ts, q_hs, k, k_ts, k_hs, vt, vt_hs, vt_ds, out, o_ts, n_heads, n_kv, hd, Lq, S,
                            causal, (cudaStream_t)stream, 0, Lq, 0, S, nullptr, 0, true);
}
extern "C" int b200_attention_fa_rows(const void* q, long q_ts, long q_hs, const void* k, long k_ts, long k_hs, const void* v,
                                      long v_ts, long v_hs, void* out, long o_ts, int n_heads, int n_kv, int hd, int Lq, int S,
                                      int causal, int q_tot, int k_tot, const int* segs, int n_seg, int flags, void* stream) {
  return b200::attention_fa(q, q_ts, q_hs, k, k_ts, k_hs, v, v_ts, v_hs, out, o_ts, n_heads, n_kv, hd, Lq, S, causal,
                            (cudaStream_t)stream, 0, q_tot, 0, k_tot, segs, n_seg, false, flags);
}
