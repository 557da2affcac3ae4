// Host stand-ins for the wrappers of csrc/ptx.cuh: the attention kernels compiled against this file run one thread at a time
// and print what that thread waits for, arrives on, loads, issues and touches.  Every wait returns at once.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __grid_constant__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) alignas(n)

struct Index3 { unsigned x, y, z; };
extern Index3 threadIdx, blockIdx;
struct CUtensorMap { char name; };
struct __nv_bfloat16 { uint16_t bits; };

namespace dtb {

using std::max;
using std::min;

alignas(1024) uint8_t smem_raw[232448];
inline bool recording = true;
template <class... A>
void record(const char* format, A... a) { if (recording) std::printf(format, a...); }
inline uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(static_cast<const uint8_t*>(p) - smem_raw); }
inline bool in_smem(const void* p) { return p >= smem_raw && p < smem_raw + sizeof(smem_raw); }

// Plain accesses to shared memory go through these two types.
struct uint4 {
  uint32_t x, y, z, w;
  uint4& operator=(const uint4& v) {
    if (in_smem(this)) record("stage %u\n", smem_u32(this));
    std::memcpy(static_cast<void*>(this), &v, sizeof v);
    return *this;
  }
};
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
struct float2 {
  float x, y;
  float2() = default;
  float2(float a, float b) : x(a), y(b) {}
  float2(const float2& v) : x(v.x), y(v.y) { if (in_smem(&v)) record("get\n"); }
  float2& operator=(const float2& v) {
    if (in_smem(this)) record("put\n");
    x = v.x; y = v.y;
    return *this;
  }
};
inline float2 make_float2(float x, float y) { return float2(x, y); }
struct float4 { float x, y, z, w; };
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }

inline float __uint_as_float(uint32_t v) { float f; std::memcpy(&f, &v, 4); return f; }
inline uint32_t __float_as_uint(float f) { uint32_t v; std::memcpy(&v, &f, 4); return v; }
inline bool __all_sync(uint32_t, bool v) { return v; }
inline bool __any_sync(uint32_t, bool v) { return v; }
inline void __syncwarp() {}
inline void __nanosleep(unsigned) {}
inline void __syncthreads() { record("sync\n"); }
inline uint64_t globaltimer_ns() { return 0; }

struct AbortCtx { volatile int* cta_abort; int* status; };
inline void mbar_init(uint32_t bar, uint32_t count) { record("init %u %u\n", bar, count); }
inline void mbar_fence_init() {}
inline void mbar_expect_tx(uint32_t bar, uint32_t bytes) { record("expect %u %u\n", bar, bytes); }
inline void mbar_arrive(uint32_t bar) { record("arrive %u\n", bar); }
inline bool mbar_wait(uint32_t bar, uint32_t parity, const AbortCtx&, int) { record("wait %u %u\n", bar, parity); return true; }
inline void tc_fence_before() { record("before\n"); }
inline void tc_fence_after() { record("after\n"); }
inline void tma_load_4d(uint32_t dst, const CUtensorMap* t, uint32_t bar, int c0, int c1, int, int) {
  record("load %u %c %u %d %d\n", dst, t->name, bar, c0, c1);
}
inline void tma_prefetch_desc(const CUtensorMap*) {}
inline void tmem_alloc(uint32_t dst, uint32_t) { std::memset(smem_raw + dst, 0, 4); }
inline void tmem_relinquish() {}
inline void tmem_dealloc(uint32_t, uint32_t) { record("dealloc\n"); }

// S rows: zeros, or logits that grow from one tile to the next (each time the offset has to move).
inline bool growing = false;
inline int tiles_read = 0;
inline void tmem_ld128_sync(uint32_t col, uint32_t (&r)[128]) {
  record("ld %u 128\n", col & 0xffff);
  for (auto& v : r) v = __float_as_uint(growing ? 100.f * static_cast<float>(tiles_read) : 0.f);
  ++tiles_read;
}
inline void tmem_ld32_sync(uint32_t col, uint32_t (&r)[32]) {
  record("ld %u 32\n", col & 0xffff);
  for (auto& v : r) v = 0;
}
inline void tmem_st32(uint32_t col, const uint32_t (&)[32]) { record("st %u 32\n", col & 0xffff); }
inline void tmem_st16(uint32_t col, const uint32_t*) { record("st %u 16\n", col & 0xffff); }
inline void tmem_wait_st() { record("wait_st\n"); }

// A descriptor is the address of its operand; the kernels add offsets in units of 16 bytes.
inline uint64_t make_smem_desc_sw128(uint32_t addr, uint32_t, uint32_t) { return addr >> 4; }
constexpr uint32_t make_idesc_bf16(int, int, bool, bool) { return 0; }
constexpr uint32_t make_idesc_e4m3(int, int) { return 0; }
inline unsigned address(uint64_t desc) { return static_cast<unsigned>(desc << 4); }
inline void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t, uint32_t acc) {
  record("qk %u %u %u %u\n", d, address(a), address(b), acc);
}
inline void mma_ss_f8(uint32_t d, uint64_t a, uint64_t b, uint32_t i, uint32_t acc) { mma_ss(d, a, b, i, acc); }
inline void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t, uint32_t acc) {
  record("pv %u %u %u %u\n", d, a, address(b), acc);
}
inline bool elect_one() { return true; }
inline void mma_commit(uint32_t bar) { record("commit %u\n", bar); }
template <int kRegs> void setmaxnreg_inc() {}
template <int kRegs> void setmaxnreg_dec() {}

inline void ld_global8(const float* src, uint32_t* r) { std::memcpy(r, src, 32); }
inline float ex2(float x) { return std::exp2(x); }
inline uint64_t pack_f32x2(float lo, float hi) { return static_cast<uint64_t>(__float_as_uint(hi)) << 32 | __float_as_uint(lo); }
inline void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  lo = __uint_as_float(static_cast<uint32_t>(v));
  hi = __uint_as_float(static_cast<uint32_t>(v >> 32));
}
inline uint64_t fma_f32x2(uint64_t, uint64_t, uint64_t) { return 0; }
inline uint64_t add_f32x2(uint64_t, uint64_t) { return 0; }
inline float max3(float a, float b, float c) { return std::max(a, std::max(b, c)); }
inline uint32_t pack_bf16x2(float, float) { return 0; }

}  // namespace dtb
