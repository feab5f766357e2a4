// Common device/host helpers for the b200vlm kernels (sm_100a only).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/b200vlm.h"

namespace b200 {

// ---- error plumbing (C-ABI: int status + b200_last_error()) ---------------
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define B200_CUDA(call)                                                     \
  do {                                                                      \
    cudaError_t _e = (call);                                                \
    if (_e != cudaSuccess) return ::b200::cuda_fail(_e, #call, __FILE__, __LINE__); \
  } while (0)

#define B200_CHECK_LAUNCH()                                                 \
  do {                                                                      \
    cudaError_t _e = cudaGetLastError();                                    \
    if (_e != cudaSuccess) return ::b200::cuda_fail(_e, "kernel launch", __FILE__, __LINE__); \
  } while (0)

#define B200_REQUIRE(cond, ...)                                             \
  do {                                                                      \
    if (!(cond)) { ::b200::set_error(__VA_ARGS__); return B200_ERR_INVALID; } \
  } while (0)

typedef __nv_bfloat16 bf16;

// ---- bf16 rounding points (the oracle's Rounder.r) ------------------------
__device__ __forceinline__ float rbf(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}
__device__ __forceinline__ float bf2f(bf16 x) { return __bfloat162float(x); }
__device__ __forceinline__ bf16 f2bf(float x) { return __float2bfloat16_rn(x); }

// unpack 8 bf16 (one 16-byte vector) to 8 floats
__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void unpack4(const uint2& v, float* f) {
  f[0] = __uint_as_float(v.x << 16);
  f[1] = __uint_as_float(v.x & 0xffff0000u);
  f[2] = __uint_as_float(v.y << 16);
  f[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}

// pairs of floats: one instruction for two
__device__ __forceinline__ uint64_t f2(float a, float b) {
  return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float f2_lo(uint64_t x) { return __uint_as_float((uint32_t)x); }
__device__ __forceinline__ float f2_hi(uint64_t x) { return __uint_as_float((uint32_t)(x >> 32)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// streaming 16-byte load that does not allocate in L1 (weights are read once)
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// products of bf16 pairs as they are: d0 += lo * lo, d1 += hi * hi, each rounded once like an fp32 FMA of the unpacked values
__device__ __forceinline__ void fma_bf2(float& d0, float& d1, uint32_t a, uint32_t b) {
  asm("{\n\t.reg .b16 al, ah, bl, bh;\n\t"
      "mov.b32 {al, ah}, %2;\n\tmov.b32 {bl, bh}, %3;\n\t"
      "fma.rn.f32.bf16 %0, al, bl, %0;\n\tfma.rn.f32.bf16 %1, ah, bh, %1;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "r"(a), "r"(b));
}
// both onto one sum, lo first
__device__ __forceinline__ void dot_bf2(float& s, uint32_t a, uint32_t b) {
  asm("{\n\t.reg .b16 al, ah, bl, bh;\n\t"
      "mov.b32 {al, ah}, %1;\n\tmov.b32 {bl, bh}, %2;\n\t"
      "fma.rn.f32.bf16 %0, al, bl, %0;\n\tfma.rn.f32.bf16 %0, ah, bh, %0;\n\t}"
      : "+f"(s)
      : "r"(a), "r"(b));
}
// a pair times one number: p is a bf16 value in fp32
__device__ __forceinline__ void axpy_bf2(float& d0, float& d1, float p, uint32_t v) {
  asm("{\n\t.reg .b16 pl, ph, vl, vh;\n\t"
      "mov.b32 {pl, ph}, %2;\n\tmov.b32 {vl, vh}, %3;\n\t"
      "fma.rn.f32.bf16 %0, ph, vl, %0;\n\tfma.rn.f32.bf16 %1, ph, vh, %1;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "r"(__float_as_uint(p)), "r"(v));
}
// warp_sum of 8 values at once, by the same tree: lane L gets the sum of value L / 4
__device__ __forceinline__ float warp_sum8(const float (&x)[8], int lane) {
  float a[4], b[2];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool up = lane & 16;
    a[k] = (up ? x[k + 4] : x[k]) + __shfl_xor_sync(0xffffffffu, up ? x[k] : x[k + 4], 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const bool up = lane & 8;
    b[k] = (up ? a[k + 2] : a[k]) + __shfl_xor_sync(0xffffffffu, up ? a[k] : a[k + 2], 8);
  }
  const bool up = lane & 4;
  float s = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// ---- activation restatements (oracle/mlx_semantics.py) --------------------
// 1 / (1 + e^-x) with the SFU exponential and reciprocal (branch-free, ~3 ulp): far below the bf16 rounding every
// bf16 caller applies next and below the 2^-17 of the split-operand GEMMs on the fp32 paths (the libm expf + IEEE
// division version has a slow-path branch per element and cost ~9 us per GEMM epilogue)
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
// The same of a pair: one packed multiplication and addition, an exponential and a reciprocal each (results below 2^-126 are 0)
__device__ __forceinline__ uint64_t sigmoid2(uint64_t x) {
  const uint64_t t = mul2(x, f2(-1.4426950408889634f, -1.4426950408889634f));
  float a, b;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(f2_lo(t)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(f2_hi(t)));
  const uint64_t d = add2(f2(a, b), f2(1.f, 1.f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(f2_lo(d)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(f2_hi(d)));
  return f2(a, b);
}
// of bf16 pairs: a product of two bf16 is exact in fp32, so the packed multiplication rounds where rbf(a * b) does
__device__ __forceinline__ uint32_t mul_bf2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint64_t unpack_bf2(uint32_t x) { return f2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
__device__ __forceinline__ uint32_t pack_bf2(uint64_t x) { return pack2(f2_lo(x), f2_hi(x)); }
// swiglu_bf and gelu_fast_bf of bf16 pairs, the same roundings
__device__ __forceinline__ uint32_t swiglu_bf2(uint32_t g, uint32_t u) {
  return mul_bf2(mul_bf2(g, pack_bf2(sigmoid2(unpack_bf2(g)))), u);
}
__device__ __forceinline__ uint32_t gelu_fast_bf2(uint32_t x) {
  return mul_bf2(x, pack_bf2(sigmoid2(unpack_bf2(mul_bf2(x, 0x3FDA3FDAu)))));   // 1.703125
}
// nn.silu(g) * u : three roundings
__device__ __forceinline__ float swiglu_bf(float g, float u) {
  float s = rbf(g * rbf(sigmoid_f(g)));
  return rbf(s * u);
}
// nn.GELU(approx="fast"): x * sigmoid(1.702 x); 1.702 weak-typed to bf16 = 1.703125
__device__ __forceinline__ float gelu_fast_bf(float x) {
  return rbf(x * rbf(sigmoid_f(rbf(1.703125f * x))));
}
// nn.GELU(): x * (1 + erf(x / sqrt2)) / 2; sqrt2 weak-typed to bf16 = 1.4140625 (for every bf16 x the product with its reciprocal
// rounds to the same bf16 as the quotient)
__device__ __forceinline__ float gelu_exact_bf(float x) {
  float a = rbf(x * (1.0f / 1.4140625f));
  float b = rbf(erff(a));
  float c = rbf(1.0f + b);
  float d = rbf(x * c);
  return rbf(d * 0.5f);
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

// A unit's device word that its kernels raise when a wait ran out (0: never did); wait_error: the first one raised on the
// current device.  A word stays raised: the results of that launch were NaN, and something that should not happen did.
struct WaitWord {
  explicit WaitWord(int (*read)(int*));
};
int wait_error(int* out);

// per-DEVICE one-time setup (cudaFuncSetAttribute is per device): `if (FirstUse first{&mask}) B200_CUDA(...)` runs until it has
// succeeded once on the current device.  The device is marked when the setup is done, not before: a second thread that comes
// meanwhile does it again instead of launching without it.
struct FirstUse {
  unsigned long long *mask, bit = 0ull;
  explicit FirstUse(unsigned long long* m) : mask(m) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    if (!(__atomic_load_n(mask, __ATOMIC_ACQUIRE) >> (dev & 63) & 1ull)) bit = 1ull << (dev & 63);
  }
  ~FirstUse() {
    if (bit && cudaPeekAtLastError() == cudaSuccess) __atomic_fetch_or(mask, bit, __ATOMIC_RELEASE);
  }
  FirstUse(const FirstUse&) = delete;
  explicit operator bool() const { return bit != 0ull; }
};

// ---- waits that end ----------------------------------------------------------------
// Waits for a phase of an mbarrier of this CTA; false, and *failed (shared memory, zeroed before the first wait) set, after
// WAIT_TRIES tries.  Whoever gets a false multiplies, signals and requests nothing more, and waits for no later phase (a
// barrier of which a phase was passed over answers for another one); so the waits of others for it run out too, its own copies
// and products end (mbar_drain), and NaN is stored.  The kernel raises its unit's word (WaitWord), which b200_wait_error reads.
constexpr int WAIT_TRIES = 1 << 18;   // 4 us each: a second
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(addr), "r"(parity)
      : "memory");
  return done;
}
// (a try_wait takes some 200 cycles even where the phase is over, a test_wait 80: every wait asks once that way first)
__device__ __forceinline__ bool mbar_test(uint32_t addr, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(addr), "r"(parity)
      : "memory");
  return done;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* failed) {
  const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
  if (mbar_test(addr, parity)) return true;
#pragma unroll 1
  for (int i = 0; i < WAIT_TRIES; ++i)
    if (mbar_try(addr, parity)) return true;
  *static_cast<volatile int*>(failed) = 1;
  return false;
}
// The same for a thread that issues tensor-core products: once a wait ran out it goes on without waiting, with `dead` set, and
// its commits then go to a barrier that nobody waits on (a select instead of a branch).  Leaving the loops instead made the
// tower attention, which is bound by its issuing thread, slower: three CLIP blocks of 8 pictures 1400 -> 1440 us.
__device__ __forceinline__ void mbar_wait_issuer(uint64_t* bar, uint32_t parity, bool& dead) {
  const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
  uint32_t done = mbar_test(addr, parity);
  for (int i = 0; !done && !dead; ++i) {
    done = mbar_try(addr, parity);
    if (i > WAIT_TRIES) dead = true;
  }
}
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {   // the same after a failure
  int mine = 0;
  mbar_wait(bar, parity, &mine);
}

// ---- programmatic dependent launch -------------------------------------------------
// Every kernel of the prefill / vision / batched-decode sequences starts with pdl_prologue():
// it lets the NEXT kernel of the stream begin (its barrier / TMEM set-up and the prefetch of its
// weights overlap this kernel) and then waits until everything the PREVIOUS kernels wrote is visible.
__device__ __forceinline__ void pdl_prologue() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
#ifdef __CUDACC__
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}
#endif

}  // namespace b200
