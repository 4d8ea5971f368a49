// Device and host helpers of the tcgen05 convolutions (nn_tc.cu, nn_tile.cu): mbarrier
// waits, TMA loads, shared-memory matrix descriptors, the MMA itself.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

namespace glnn_tc {

typedef __nv_bfloat16 bf16;

constexpr uint32_t kSpinLimit = 1u << 20;   // mbarrier polls before giving up

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

// The same, for a whole warp in step (one elected lane issues), with the descriptors as
// 32-bit halves: a run of MMAs advances the low halves (start addresses, 16-byte units) by
// constants.  The instruction takes its operands from uniform registers; the warp has to be
// in step, the values warp-uniform and the lane elected for the compiler to keep them
// there.  Issued inside a one-lane branch every operand is moved over for every MMA: one
// then took 90-125 cycles, N = 16 to 64 alike (32 -> 32 channels, 64 images of 128^2: 126
// us that way, 72 with constant steps, 49 with the warp in step, 41 with the election).
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                        uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p, l;\n .reg .b64 da, db;\n mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
        " setp.ne.b32 p, %6, 0;\n elect.sync _|l, 0xffffffff;\n"
        " @l tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}\n" ::"r"(tmem_d),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
        : "memory");
}
// tcgen05.commit of the MMAs issued so far by the elected lane to an mbarrier
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile(
        "{\n .reg .pred l;\n elect.sync _|l, 0xffffffff;\n"
        " @l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
        : "memory");
}
// warp index as a warp-uniform value
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t phase) {
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// the wait by a whole warp in step
__device__ __forceinline__ bool wait_parity_warp(uint32_t bar, uint32_t phase) {
    return __all_sync(0xffffffffu, wait_parity(bar, phase));
}

// SM100 shared-memory matrix descriptor, K-major with the 128-byte swizzle:
// start >> 4 (bits 0-13), leading offset 16 B (unused for this layout), stride
// offset between 8-row groups (32-45), version 1 (46-47), layout type
// 2 = 128-byte swizzle (61-63).  A K step of 16 elements advances the start by 32 B.
constexpr uint32_t desc_hi(uint32_t stride) { return (stride >> 4) | (1u << 14) | (2u << 29); }
__device__ __forceinline__ uint32_t desc_lo(uint32_t start) { return (start >> 4) | (1u << 16); }

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
            dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// MN-major with the 128-byte swizzle: leading byte offset = distance between 64-element
// atoms along M or N, stride byte offset = distance between 8-row groups along K.
__device__ __forceinline__ uint32_t desc_lo_mn(uint32_t start, uint32_t lbo) { return (start >> 4) | ((lbo >> 4) << 16); }

// Sixteen accumulator columns of one output pixel: + bias and ReLU (BIAS), to bfloat16,
// as two 16-byte stores.  (A pixel's channels are contiguous, so a warp's store covers 32
// rows whatever its width; with 4-byte stores the epilogue's 32 per thread took longer
// than the tile's MMAs.)
template <int BIAS, int RELU>
__device__ __forceinline__ void store_cols16(const uint32_t (&r)[16], const float* bias, bf16* out) {
    uint4 v[2];
    __nv_bfloat162* h = (__nv_bfloat162*)v;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float v0 = __uint_as_float(r[2 * q]), v1 = __uint_as_float(r[2 * q + 1]);
        if (BIAS) {
            v0 += bias[2 * q];
            v1 += bias[2 * q + 1];
        }
        if (RELU) {
            v0 = fmaxf(v0, 0.f);
            v1 = fmaxf(v1, 0.f);
        }
        h[q] = __floats2bfloat162_rn(v0, v1);
    }
    ((uint4*)out)[0] = v[0];
    ((uint4*)out)[1] = v[1];
}

static PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

}  // namespace glnn_tc
