// fp32 attention of the towers (CLIP, SigLIP and its resampler, Qwen2.5-VL) on the tensor cores.
//
// Every fp32 operand is carried as THREE bf16 parts, x = h + m + l (h = bf16(x), m = bf16(x - h), l = bf16(x - h - m): 24
// mantissa bits, the exponent range of fp32), and a product of two operands as the six products of parts that are not below
// fp32's own rounding: l.h + h.l + m.m + m.h + h.m + h.h, added smallest first so that the small ones meet an accumulator
// of their size.  Rows with a result that is not finite are computed again without parts (plain_row).  tcgen05 truncates its fp32 accumulator at every step, so no sum runs over more than one tile: the scores of
// a tile (one head dimension) and its P.V (64 keys) each start from zero in tensor memory, and the softmax threads add the
// tile's P.V to their fp32 registers with rounding.  Error against 64 bits, relative: 2.2e-7 at 577 keys of 64 dims, 2.5e-7 at
// 1024 of 72 (a register-tiled FMA kernel: 5.2e-7, 6.5e-7).
//
// One CTA = 128 query rows of one head of one segment, tiles of 64 keys:
//   warps 8..14  load the fp32 keys and values of a tile, split them, store the parts as no-swizzle K-major core matrices (8
//                rows x 16 bytes).  A block of 8 columns is 16 bytes longer than its rows need, so that the eight lanes of a
//                store that share a row (K: a key) or a column (V: 8 keys) hit different banks.  V is transposed on the way
//                (a thread holds 8 keys x 4 dims): as an MN-major operand it took the tensor core 138 cycles per
//                128 x 64 x 16 product instead of about 40.
//   warp 15      issues S[g] = Q.K^T and O[g] = P[g].V; P is an operand in tensor memory, no shared memory is touched by it
//   warps 0..7   two groups of 128 threads, thread = query row: group g takes the tiles j = g mod 2 with its own score, P and
//                O buffers in tensor memory and its own running maximum, sum and output, so the tensor core works on one
//                group's tile while the other group is at its exponentials.  At the end the groups merge through shared memory.
// With three loading warps they were what bounds it (without their splitting 319 -> 260 us for two blocks of the first of these, with
// a sixth of the products 264): seven of them, the registers shared out between the roles (setmaxnreg), took CLIP-L, 8 pictures (16
// heads of 64, 577 tokens) from 159 to 136 us a block, SigLIP, 4 of 1024 tokens (16 of 72) from 235 to 183, 64 latents on 1088 keys
// of 96 from 73 to 54.  What is left: products (S at 52 cycles each, which is what its two operands take to leave shared memory, P.V
// at 56) and the softmax between them.  Per block, fp32 FMA kernel -> the form with three loading warps: CLIP-L 417 -> 148 us, SigLIP 790 -> 240,
// 64 latents on 1088 keys of 96 160 -> 75, one frame of 1564 (16 of 80) 583 -> 170, 25 windows of 64 41 -> 33; windows of 32
// tokens cost the same (56, 58).
#include <type_traits>

#include "common.cuh"
#include "decode.cuh"

namespace b200 {

namespace {

constexpr int TC_ROWS = 128, TC_KEYS = 64;
constexpr int TC_LOADERS = 224;
constexpr int TC_THREADS = 256 + TC_LOADERS + 32;   // 8 softmax, 7 loading and 1 MMA warp
constexpr int TC_MMA = TC_THREADS / 32 - 1;         // the last warp
// registers of a softmax thread and of the others: together what the block is launched with, 512 x 128
constexpr int TC_REGS_SOFTMAX = 152, TC_REGS_OTHER = 104;
// (a larger share would be waited for without end: tc_launch asks what the kernel was compiled with, the launch bounds only limit it)
constexpr bool tc_shares_fit(int regs) { return 256 * TC_REGS_SOFTMAX + (TC_THREADS - 256) * TC_REGS_OTHER <= TC_THREADS * regs; }
static_assert(tc_shares_fit(128) && !tc_shares_fit(127), "the shares are those of 128 registers a thread");
constexpr int TC_QB = TC_ROWS * 16 + 16, TC_KB = TC_KEYS * 16 + 16;   // bytes of a block of 8 dims
constexpr int TC_P0 = 128, TC_O0 = 320, TC_GB = 96;   // TMEM columns: S 2 x 64 | P 2 x (3 x 32) | O 2 x 96

struct TcBars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_full[2], o_full[2], drained, dropped;
};

__device__ __forceinline__ uint32_t t_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void t_init(uint64_t* bar, uint32_t n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(t_u32(bar)), "r"(n));
}
__device__ __forceinline__ void t_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(t_u32(bar)) : "memory");
}
__device__ int g_f32_wait_failed;   // a wait of attention_f32_tc_kernel ran out: B200_WAIT_TOWER
__device__ __forceinline__ void t_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void t_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void t_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(t_u32(bar)) : "memory");
}
// no-swizzle K-major operand descriptor, low word: byte offset `lead` between core matrices along K (the high word has the
// 128 bytes between those along M or N).  Walking an operand is an addition of a constant: one thread issues 48 and more
// products a tile, and with the descriptors made anew for each it issued one per 62 (S) and 127 (P.V) cycles, whatever N was.
__device__ __forceinline__ uint32_t t_desc(uint32_t addr, uint32_t lead) { return ((addr & 0x3FFFFu) >> 4) | ((lead >> 4) << 16); }
constexpr uint32_t T_DESC_HI = (128u >> 4) | (1u << 14);
template <bool ACC>
__device__ __forceinline__ void t_mma_ss(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
               "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d),
               "r"(a), "r"(b), "r"(T_DESC_HI), "r"(idesc), "n"((int)ACC)
               : "memory");
}
template <bool ACC>
__device__ __forceinline__ void t_mma_ts(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tmov.b64 db, {%2, %3};\n\t"
               "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d),
               "r"(a), "r"(b), "r"(T_DESC_HI), "r"(idesc), "n"((int)ACC)
               : "memory");
}
// (its values may be used after t_ld_wait)
__device__ __forceinline__ void t_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void t_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
__device__ __forceinline__ void t_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}

// 2^x on the SFU; results below 2^-126 are 0, beside a row's largest weight of 1
__device__ __forceinline__ float t_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float T_LOG2E = 1.4426950408889634f;

// two floats -> their three bf16 parts, packed
__device__ __forceinline__ void split3(uint64_t x, uint32_t& h, uint32_t& m, uint32_t& l) {
  const uint64_t neg = f2(-1.f, -1.f);   // x - part, exactly: part * -1 + x
  h = pack2(f2_lo(x), f2_hi(x));
  x = fma2(f2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), neg, x);
  m = pack2(f2_lo(x), f2_hi(x));
  x = fma2(f2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), neg, x);
  l = pack2(f2_lo(x), f2_hi(x));
}

// Rows [0, ROWS) x HDP dims of a fp32 operand in items of 8 dims: U items per thread from item i0 on, N threads apart.  Rows
// behind the last (rows - 1) and pieces behind the last of the row (4 dims at hd - 4) repeat it, so that no load is
// conditional: such scores are masked, such dims meet zeros of Q or are not stored.  ZERO (Q): those dims are zeros ...
template <int HDP, int ROWS, int U, int N, bool ZERO>
__device__ __forceinline__ void load_items(float4 (&a)[U], float4 (&b)[U], int i0, const float* src, long row_stride, int rows,
                                           int hd) {
  constexpr int NC = HDP / 8;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int i = i0 + N * u, r = min(i / NC, rows - 1), c = i % NC;
    const float* p = src + (long)r * row_stride;
    a[u] = *reinterpret_cast<const float4*>(p + min(c * 8, hd - 4));
    b[u] = *reinterpret_cast<const float4*>(p + min(c * 8 + 4, hd - 4));
    if (ZERO) {
      if (c * 8 >= hd) a[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c * 8 + 4 >= hd) b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}
// ... and their three parts' images at dst (part_bytes apart)
template <int HDP, int ROWS, int U, int N>
__device__ __forceinline__ void store_items(uint8_t* dst, int part_bytes, const float4 (&a)[U], const float4 (&b)[U], int i0,
                                            float scale) {
  constexpr int NC = HDP / 8, BLK = ROWS * 16 + 16;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int i = i0 + N * u, r = i / NC, c = i % NC;
    if (i >= ROWS * NC) continue;
    uint4 h, m, l;
    split3(f2(a[u].x * scale, a[u].y * scale), h.x, m.x, l.x);
    split3(f2(a[u].z * scale, a[u].w * scale), h.y, m.y, l.y);
    split3(f2(b[u].x * scale, b[u].y * scale), h.z, m.z, l.z);
    split3(f2(b[u].z * scale, b[u].w * scale), h.w, m.w, l.w);
    uint8_t* d = dst + c * BLK + r * 16;
    *reinterpret_cast<uint4*>(d) = h;
    *reinterpret_cast<uint4*>(d + part_bytes) = m;
    *reinterpret_cast<uint4*>(d + 2 * part_bytes) = l;
  }
}

// Values: a warp takes 16 dims x 64 keys, a thread 4 dims x 8 keys: lane = (4 dims: lane / 8, 8 keys: lane mod 8) ...
__device__ __forceinline__ void load_values(float4 (&x)[8], const float* src, long row_stride, int rows, int hd, int dim,
                                            int lane) {
  const float* p = src + min(dim + (lane >> 3) * 4, hd - 4);
  const int k = (lane & 7) * 8;
  if (rows == TC_KEYS) {
    p += k * row_stride;
#pragma unroll
    for (int i = 0; i < 8; ++i, p += row_stride) x[i] = *reinterpret_cast<const float4*>(p);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(p + (long)min(k + i, rows - 1) * row_stride);
  }
}
// ... and stores 8 keys of each of its dims as one row of a core matrix
template <int HDP>
__device__ __forceinline__ void store_values(uint8_t* dst, int part_bytes, const float4 (&x)[8], int dim, int lane) {
  uint8_t* d = dst + (lane & 7) * (HDP * 16 + 16) + (dim + (lane >> 3) * 4) * 16;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    auto at = [&](int i) { return u == 0 ? x[i].x : u == 1 ? x[i].y : u == 2 ? x[i].z : x[i].w; };
    uint4 h, m, l;
    split3(f2(at(0), at(1)), h.x, m.x, l.x);
    split3(f2(at(2), at(3)), h.y, m.y, l.y);
    split3(f2(at(4), at(5)), h.z, m.z, l.z);
    split3(f2(at(6), at(7)), h.w, m.w, l.w);
    *reinterpret_cast<uint4*>(d + u * 16) = h;
    *reinterpret_cast<uint4*>(d + u * 16 + part_bytes) = m;
    *reinterpret_cast<uint4*>(d + u * 16 + 2 * part_bytes) = l;
  }
}

// One query row by one warp in plain fp32 arithmetic: p.hd floats to out.  The parts of a number that is no finite bf16 (an
// infinity, a NaN, a magnitude above 3.39e38) are infinities and NaN that the row's other products would spread, so a row
// with such a result is computed again: a key that scores -inf has weight 0, an infinite value stays in its own dimension.
__device__ __noinline__ void plain_row(const AttnF32P& p, const float* q, const float* kb, const float* vb, int S,
                                       const unsigned char* mask, float* out, int lane) {
  auto score = [&](int j) {
    if (j >= S || (mask && !mask[j])) return -INFINITY;
    float s = 0.f;
    for (int d = 0; d < p.hd; d += 4) {
      const float4 a = *reinterpret_cast<const float4*>(q + d), b = *reinterpret_cast<const float4*>(kb + (long)j * p.k_ts + d);
      s = fmaf(a.x * p.scale, b.x, s);
      s = fmaf(a.y * p.scale, b.y, s);
      s = fmaf(a.z * p.scale, b.z, s);
      s = fmaf(a.w * p.scale, b.w, s);
    }
    return s;
  };
  float m = -INFINITY, l = 0.f, o[3] = {0.f, 0.f, 0.f};
  for (int j = lane; j < S; j += 32) m = fmaxf(m, score(j));
  m = warp_max(m);
  for (int j0 = 0; j0 < S; j0 += 32) {
    const int j = j0 + lane;
    const float w = j < S && (!mask || mask[j]) ? expf(score(j) - m) : 0.f;
    l += w;
    for (int i = 0; i < min(32, S - j0); ++i) {
      const float wi = __shfl_sync(0xffffffffu, w, i);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (lane + 32 * e < p.hd) o[e] = fmaf(wi, vb[(long)(j0 + i) * p.v_ts + lane + 32 * e], o[e]);
    }
  }
  const float inv = 1.0f / warp_sum(l);
#pragma unroll
  for (int e = 0; e < 3; ++e)
    if (lane + 32 * e < p.hd) out[lane + 32 * e] = o[e] * inv;
}

template <int HDP>
constexpr int tc_q_part() { return HDP / 8 * TC_QB; }
template <int HDP>
constexpr int tc_k_part() { return HDP / 8 * TC_KB; }
template <int HDP>
constexpr int tc_v_part() { return TC_KEYS / 8 * (HDP * 16 + 16); }
template <int HDP>
constexpr int tc_smem() { return 3 * tc_q_part<HDP>() + 6 * tc_k_part<HDP>() + 6 * tc_v_part<HDP>() + 128; }

template <int HDP>
__global__ void __launch_bounds__(TC_THREADS, 1) attention_f32_tc_kernel(const __grid_constant__ AttnF32P p) {
  extern __shared__ uint8_t tc_raw[];
  __shared__ TcBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ float2 stat[2][TC_ROWS];
  __shared__ int failed;
  __shared__ uint32_t odd[8];   // rows with a result that is not finite, one bit each: [half of the dims][row / 32]
  constexpr int QP = tc_q_part<HDP>(), KP = tc_k_part<HDP>(), VP = tc_v_part<HDP>();
  uint8_t* Qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* Ks = Qs + 3 * QP;      // 2 slots x 3 parts
  uint8_t* Vs = Ks + 6 * KP;      // 2 slots x 3 parts
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, kvh = h / (p.n_heads / p.n_kv), seg = blockIdx.z;
  const int q0 = blockIdx.x * TC_ROWS;
  long q_first = (long)seg * p.q_seg, k_first = (long)seg * p.k_seg;
  int Lq = p.Lq, S = p.S;
  if (p.cu) {
    q_first = k_first = p.cu[seg];
    Lq = S = p.cu[seg + 1] - p.cu[seg];
    if (q0 >= Lq) return;   // uniform per CTA, nothing is allocated yet
  }
  const int n_tiles = (S + TC_KEYS - 1) / TC_KEYS;
  if (tid == 0) {
    failed = 0;
    t_init(&bars.q_full, 256);
    t_init(&bars.drained, 1);
    t_init(&bars.dropped, 1);
    for (int i = 0; i < 2; ++i) {
      t_init(&bars.k_full[i], TC_LOADERS);
      t_init(&bars.v_full[i], TC_LOADERS);
      t_init(&bars.k_empty[i], 1);
      t_init(&bars.v_empty[i], 1);
      t_init(&bars.s_full[i], 1);
      t_init(&bars.p_full[i], 128);
      t_init(&bars.o_full[i], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == TC_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(t_u32(&tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t_fence_before();
  __syncthreads();
  t_fence_after();
  const uint32_t tmem = tmem_slot;
  // (the next kernel may start from here on, not before: it may ask for tensor memory too, and would hold what this one still needs)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REGS_OTHER));   // (one instruction for both roles: a warpgroup executes it together)
    if (warp == TC_MMA) {
      if (lane == 0) {  // ===== MMA issuer =====
        // D = f32, A = B = bf16, both K-major, M = 128; N = keys of the tile / dims
        constexpr uint32_t ID = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);
        constexpr uint32_t ID_O = ID | ((uint32_t)(HDP >> 3) << 17);
        // (part of A, part of B), the smallest product first; 0 = h, 1 = m, 2 = l
        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
        constexpr int KS = HDP / 16, VL = HDP * 16 + 16;
        const uint32_t q_lo = t_desc(t_u32(Qs), TC_QB), k_lo = t_desc(t_u32(Ks), TC_KB), v_lo = t_desc(t_u32(Vs), VL);
        bool dead = false;
        auto keys16 = [&](int j) { return min(TC_KEYS, (S - j * TC_KEYS + 15) & ~15); };
        auto issue_s = [&](int j) {
          const int s = j & 1;
          mbar_wait_issuer(&bars.k_full[s], (j >> 1) & 1, dead);
          t_fence_after();
          const uint32_t idesc = ID | ((uint32_t)(keys16(j) >> 3) << 17), d = tmem + (uint32_t)s * TC_KEYS;
          const uint32_t ka = k_lo + s * (3 * KP >> 4);
          t_mma_ss<false>(d, q_lo + (PA[0] * QP >> 4), ka + (PB[0] * KP >> 4), idesc);
#pragma unroll
          for (int i = 1; i < 6 * KS; ++i) {
            const int t = i / KS, ks = i % KS;
            t_mma_ss<true>(d, q_lo + ((PA[t] * QP + ks * 2 * TC_QB) >> 4), ka + ((PB[t] * KP + ks * 2 * TC_KB) >> 4), idesc);
          }
          t_commit(dead ? &bars.dropped : &bars.k_empty[s]);
          t_commit(dead ? &bars.dropped : &bars.s_full[s]);
        };
        mbar_wait_issuer(&bars.q_full, 0, dead);
        issue_s(0);
        if (n_tiles > 1) issue_s(1);
        for (int j = 0; j < n_tiles; ++j) {
          const int s = j & 1;
          mbar_wait_issuer(&bars.p_full[s], (j >> 1) & 1, dead);
          mbar_wait_issuer(&bars.v_full[s], (j >> 1) & 1, dead);
          t_fence_after();
          const uint32_t d = tmem + TC_O0 + s * TC_GB, pa = tmem + TC_P0 + s * TC_GB, va = v_lo + s * (3 * VP >> 4);
          t_mma_ts<false>(d, pa + PA[0] * 32, va + (PB[0] * VP >> 4), ID_O);
          if (S - j * TC_KEYS > 48) {
#pragma unroll
            for (int i = 1; i < 24; ++i) {
              const int t = i >> 2, ks = i & 3;
              t_mma_ts<true>(d, pa + PA[t] * 32 + ks * 8, va + ((PB[t] * VP + ks * 2 * VL) >> 4), ID_O);
            }
          } else {   // groups of 16 keys that lie wholly behind the last key are left out
            const int steps = keys16(j) >> 4;
#pragma unroll
            for (int t = 0; t < 6; ++t)
              for (int ks = t == 0 ? 1 : 0; ks < steps; ++ks)
                t_mma_ts<true>(d, pa + PA[t] * 32 + ks * 8, va + ((PB[t] * VP) >> 4) + ks * (2 * VL >> 4), ID_O);
          }
          t_commit(dead ? &bars.dropped : &bars.v_empty[s]);
          t_commit(dead ? &bars.dropped : &bars.o_full[s]);
          if (j + 2 < n_tiles) issue_s(j + 2);   // (the group has read S of tile j: it has stored its P)
        }
        if (dead) {   // no product is left in flight; the threads that wait for what was dropped give up as well
          *static_cast<volatile int*>(&failed) = 1;
          t_commit(&bars.drained);
          mbar_drain(&bars.drained, 0);
        }
      }
    } else {  // ===== keys and values of a tile =====
      const int t = tid - 256;
      const float* kb = p.k + k_first * p.k_ts + (long)kvh * p.k_hs;
      const float* vb = p.v + k_first * p.v_ts + (long)kvh * p.v_hs;
      constexpr int U = (TC_KEYS * HDP / 8 + TC_LOADERS - 1) / TC_LOADERS;
      constexpr int VU = (HDP / 16 + TC_LOADERS / 32 - 1) / (TC_LOADERS / 32);   // blocks of 16 dims per warp
      const int wv = warp - 8;
      float4 ka[U], kc[U], x[VU][8];   // the loads of one operand are in flight while the other is split
      load_items<HDP, TC_KEYS, U, TC_LOADERS, false>(ka, kc, t, kb, p.k_ts, min(TC_KEYS, S), p.hd);
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j & 1, rows = min(TC_KEYS, S - j * TC_KEYS);
        const uint32_t free_parity = ((j >> 1) & 1) ^ 1;
#pragma unroll
        for (int u = 0; u < VU; ++u)
          if ((wv + u * (TC_LOADERS / 32)) * 16 < HDP) load_values(x[u], vb + (long)j * TC_KEYS * p.v_ts, p.v_ts, rows, p.hd, (wv + u * (TC_LOADERS / 32)) * 16, lane);
        if (p.flags & 1) break;   // (nothing is loaded: every wait for it runs out)
        if (!mbar_wait(&bars.k_empty[s], free_parity, &failed)) break;
        store_items<HDP, TC_KEYS, U, TC_LOADERS>(Ks + s * 3 * KP, KP, ka, kc, t, 1.f);
        t_fence_async();
        t_arrive(&bars.k_full[s]);
        if (j + 1 < n_tiles)
          load_items<HDP, TC_KEYS, U, TC_LOADERS, false>(ka, kc, t, kb + (long)(j + 1) * TC_KEYS * p.k_ts, p.k_ts,
                                                  min(TC_KEYS, S - (j + 1) * TC_KEYS), p.hd);
        if (!mbar_wait(&bars.v_empty[s], free_parity, &failed)) break;
#pragma unroll
        for (int u = 0; u < VU; ++u) {
          const int dim = (wv + u * (TC_LOADERS / 32)) * 16;
          if (dim < HDP) store_values<HDP>(Vs + s * 3 * VP, VP, x[u], dim, lane);
        }
        t_fence_async();
        t_arrive(&bars.v_full[s]);
      }
    }
  } else {  // ===== softmax: thread = query row; group g = tiles j = g mod 2 =====
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_REGS_SOFTMAX));
    for (int i0 = tid; i0 < TC_ROWS * HDP / 8; i0 += 4 * 256) {
      float4 a[4], b[4];
      load_items<HDP, TC_ROWS, 4, 256, true>(a, b, i0, p.q + (q_first + q0) * p.q_ts + (long)h * p.q_hs, p.q_ts, min(TC_ROWS, Lq - q0),
                                       p.hd);
      store_items<HDP, TC_ROWS, 4, 256>(Qs, QP, a, b, i0, p.scale);
    }
    t_fence_async();
    t_arrive(&bars.q_full);
    const int g = warp >> 2, row = tid & 127;
    const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t t_s = t_row + g * TC_KEYS, t_p = t_row + TC_P0 + g * TC_GB, t_o = t_row + TC_O0 + g * TC_GB;
    uint64_t o[HDP / 2], l2 = 0ull;
    float m = -INFINITY;
#pragma unroll
    for (int e = 0; e < HDP / 2; ++e) o[e] = 0ull;
    auto add_tile = [&](float f) {   // o = (o + P.V of the group's last tile) * f
      const uint64_t ff = f2(f, f);
      uint32_t v[2][16];
      t_ld16(t_o, v[0]);
#pragma unroll
      for (int c = 0; c < HDP / 16; ++c) {
        t_ld_wait(v[c & 1]);
        if (c + 1 < HDP / 16) t_ld16(t_o + (c + 1) * 16, v[(c + 1) & 1]);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          o[c * 8 + e] = mul2(add2(o[c * 8 + e], f2(__uint_as_float(v[c & 1][2 * e]), __uint_as_float(v[c & 1][2 * e + 1]))), ff);
      }
    };
    int t = 0;
    bool ok = true;   // (the same in a warp)
    for (int j = g; j < n_tiles; j += 2, ++t) {
      // keys of this tile that take part, one bit each
      uint32_t on[2];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int key = j * TC_KEYS + w * 32 + lane;
        on[w] = __ballot_sync(0xffffffffu, key < S && (!p.key_mask || p.key_mask[(long)seg * S + key]));
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.s_full[g], t & 1, &failed));
      if (!ok) break;
      t_fence_after();
      uint32_t v[2][16];
      const bool all = (on[0] & on[1]) == 0xffffffffu;
      // a key that takes no part scores -inf: exp 0 (a select around each exponential would be a branch)
      auto masked = [&](uint32_t (&x)[16], int c) {
        if (all) return;
        const uint32_t bits = on[c >> 5] >> (c & 31);
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = (bits >> e) & 1u ? x[e] : 0xff800000u;
      };
      float mx = -INFINITY;
      t_ld16(t_s, v[0]);
#pragma unroll
      for (int c = 0; c < TC_KEYS / 16; ++c) {
        t_ld_wait(v[c & 1]);
        if (c + 1 < TC_KEYS / 16) t_ld16(t_s + (c + 1) * 16, v[(c + 1) & 1]);
        masked(v[c & 1], c * 16);
#pragma unroll
        for (int e = 0; e < 16; ++e) mx = fmaxf(mx, __uint_as_float(v[c & 1][e]));
      }
      const float mn = fmaxf(m, mx);
      const float f = mn == -INFINITY ? 1.f : t_ex2((m - mn) * T_LOG2E);   // nothing seen yet: keep zeros
      const float ref = mn == -INFINITY ? 0.f : -mn;
      m = mn;
      l2 = mul2(l2, f2(f, f));
      if (t > 0) {   // (the last P.V has also read P: it may be written again)
        ok = __all_sync(0xffffffffu, mbar_wait(&bars.o_full[g], (t - 1) & 1, &failed));
        if (!ok) break;
        t_fence_after();
        add_tile(f);
      }
      const uint64_t ref2 = f2(ref, ref), log2e = f2(T_LOG2E, T_LOG2E);
      t_ld16(t_s, v[0]);
#pragma unroll
      for (int c = 0; c < TC_KEYS / 16; ++c) {
        t_ld_wait(v[c & 1]);
        if (c + 1 < TC_KEYS / 16) t_ld16(t_s + (c + 1) * 16, v[(c + 1) & 1]);
        masked(v[c & 1], c * 16);
        uint32_t ph[8], pm[8], pl[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint64_t x = mul2(add2(f2(__uint_as_float(v[c & 1][2 * e]), __uint_as_float(v[c & 1][2 * e + 1])), ref2), log2e);
          const uint64_t w = f2(t_ex2(f2_lo(x)), t_ex2(f2_hi(x)));
          l2 = add2(l2, w);
          split3(w, ph[e], pm[e], pl[e]);
        }
        t_st8(t_p + c * 8, ph);
        t_st8(t_p + 32 + c * 8, pm);
        t_st8(t_p + 64 + c * 8, pl);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      t_fence_before();
      t_arrive(&bars.p_full[g]);
    }
    if (ok && t > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.o_full[g], (t - 1) & 1, &failed));
      if (ok) {
        t_fence_after();
        add_tile(1.f);
      }
    }
    // ---- merge: each group stores half of the dims and gets the other group's share of them through the tiles' memory,
    //      which no MMA reads any more ----
    const int rows = min(TC_ROWS, Lq - q0);
    uint64_t* ox = reinterpret_cast<uint64_t*>(Ks);   // [HDP / 2 pairs][128 rows]
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const bool whole = !*static_cast<volatile int*>(&failed);   // (else all rows of the CTA are NaN)
    const float l = whole ? f2_lo(l2) + f2_hi(l2) : NAN;
    stat[g][row] = make_float2(m, l);
    auto give = [&](auto first) {
#pragma unroll
      for (int e = 0; e < HDP / 4; ++e) ox[(first.value + e) * TC_ROWS + row] = o[first.value + e];
    };
    constexpr std::integral_constant<int, 0> low{};
    constexpr std::integral_constant<int, HDP / 4> high{};
    if (g == 0) give(high);
    else give(low);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    constexpr int PITCH = HDP + 4;
    float* of = reinterpret_cast<float*>(ox + HDP / 2 * TC_ROWS);   // [128 rows][HDP dims] of the result
    auto take = [&](auto first) {
      const float2 b = stat[g ^ 1][row];
      const float mt = fmaxf(m, b.x);
      const float fa = m == mt ? 1.f : t_ex2((m - mt) * T_LOG2E), fb = b.x == mt ? 1.f : t_ex2((b.x - mt) * T_LOG2E);
      const float inv = 1.0f / (l * fa + b.y * fb);
      float zero = 0.f;
#pragma unroll
      for (int e = 0; e < HDP / 4; e += 2) {
        float a[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint64_t x = o[first.value + e + u], y = ox[(first.value + e + u) * TC_ROWS + row];
          a[2 * u] = (f2_lo(x) * fa + f2_lo(y) * fb) * inv;
          a[2 * u + 1] = (f2_hi(x) * fa + f2_hi(y) * fb) * inv;
        }
        *reinterpret_cast<float4*>(of + row * PITCH + (first.value + e) * 2) = make_float4(a[0], a[1], a[2], a[3]);
        zero = fmaf((a[0] + a[1]) + (a[2] + a[3]), 0.f, zero);   // (NaN from the first that is not finite on)
      }
      const uint32_t bits = __ballot_sync(0xffffffffu, !(zero == 0.f) && row < rows && whole);
      if (lane == 0) odd[warp] = bits;
    };
    if (g == 0) take(low);
    else take(high);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) any |= odd[w];
    if (any) {   // (the same in all 256 threads)
      for (uint32_t todo = (odd[warp & 3] | odd[4 + (warp & 3)]) & (g == 0 ? 0xffffu : 0xffff0000u); todo; todo &= todo - 1) {
        const int r = (warp & 3) * 32 + __ffs(todo) - 1;
        plain_row(p, p.q + (q_first + q0 + r) * p.q_ts + (long)h * p.q_hs, p.k + k_first * p.k_ts + (long)kvh * p.k_hs,
                  p.v + k_first * p.v_ts + (long)kvh * p.v_hs, S, p.key_mask ? p.key_mask + (long)seg * S : nullptr, of + r * PITCH,
                  lane);
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    // stored row by row (a thread's own row in pieces would be 32 sectors per store, most of this kernel's tail)
    const int nc = p.hd >> 2;
    for (int i = tid; i < rows * nc; i += 256) {
      const int r = i / nc, d = (i - r * nc) * 4;
      const float4 a = *reinterpret_cast<const float4*>(of + r * PITCH + d);
      const long tok = q_first + q0 + r, col = (long)h * p.hd + d;
      if (p.out32) {
        float* q = p.out32 + tok * p.o_ts + col;
        if (p.out_vec) {
          *reinterpret_cast<float4*>(q) = a;
        } else {
          q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
        }
      }
      if (p.out_split) {
        bf16* q = p.out_split + tok * p.os_ts + col;
        const uint2 hi = make_uint2(pack2(a.x, a.y), pack2(a.z, a.w));
        const uint2 lo = make_uint2(pack2(a.x - __uint_as_float(hi.x << 16), a.y - __uint_as_float(hi.x & 0xffff0000u)),
                                    pack2(a.z - __uint_as_float(hi.y << 16), a.w - __uint_as_float(hi.y & 0xffff0000u)));
        if (p.out_vec) {
          *reinterpret_cast<uint2*>(q) = hi;
          *reinterpret_cast<uint2*>(q + p.n_pad) = lo;
        } else {
          unsigned short* w = reinterpret_cast<unsigned short*>(q);
          w[0] = hi.x; w[1] = hi.x >> 16; w[2] = hi.y; w[3] = hi.y >> 16;
          w += p.n_pad;
          w[0] = lo.x; w[1] = lo.x >> 16; w[2] = lo.y; w[3] = lo.y >> 16;
        }
      }
    }
  }
  t_fence_before();
  __syncthreads();
  if (tid == 0 && failed) g_f32_wait_failed = B200_WAIT_TOWER;
  if (warp == TC_MMA) {
    t_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

template <int HDP>
int tc_launch(const AttnF32P& p, dim3 grid, cudaStream_t st) {
  static unsigned long long attr_mask = 0ull;
  if (FirstUse first{&attr_mask}) {
    cudaFuncAttributes attr;
    B200_CUDA(cudaFuncGetAttributes(&attr, attention_f32_tc_kernel<HDP>));
    if (!tc_shares_fit(attr.numRegs)) first.bit = 0ull;   // (no call gets past this)
    B200_REQUIRE(tc_shares_fit(attr.numRegs), "attention_f32_tc: compiled with %d registers a thread, fewer than its roles share out", attr.numRegs);
    B200_CUDA(cudaFuncSetAttribute(attention_f32_tc_kernel<HDP>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem<HDP>()));
  }
  // Launched plainly, it waits for nothing itself.  As a dependent launch its blocks sat on the SMs that the product before it left
  // and ran longer: the whole SigLIP tower on four pictures 19.0 ms, plainly 18.5; three CLIP blocks on one picture 434 us, 423;
  // on three 641, 650; on eight the same.
  attention_f32_tc_kernel<HDP><<<grid, TC_THREADS, tc_smem<HDP>(), st>>>(p);
  B200_CHECK_LAUNCH();
  return B200_OK;
}

}  // namespace

static WaitWord g_f32_wait_word([](int* v) -> int {
  B200_CUDA(cudaMemcpyFromSymbol(v, g_f32_wait_failed, sizeof(int)));
  return B200_OK;
});

int attention_f32_tc(AttnF32P p, int n_seg, cudaStream_t st) {
  p.out_vec = ((uintptr_t)p.out32 & 15) == 0 && ((uintptr_t)p.out_split & 7) == 0;
  const dim3 grid(cdiv(p.Lq, TC_ROWS), p.n_heads, n_seg);
  if (p.hd <= 32) return tc_launch<32>(p, grid, st);
  if (p.hd <= 64) return tc_launch<64>(p, grid, st);
  if (p.hd <= 80) return tc_launch<80>(p, grid, st);
  return tc_launch<96>(p, grid, st);
}

}  // namespace b200
