// Pieces shared by the resident PCG kernels (pcg_resident.cu,
// pcg_resident_factor.cu): the cluster exchange, the sums' shuffle trees and
// the block products.  Header-only: each kernel file instantiates its own copy.
#pragma once

#include <cuda_fp16.h>

#include "block_loads.cuh"
#include "grid_sync.cuh"
#include "internal.h"

namespace mfem {
namespace {

constexpr long long kWaitCycles = 8000000000ll;  // ~4 s at 2 GHz per wait
constexpr int kTripFloats4 = 80;                 // 32 x 40 bytes

enum Scope { kOne, kCluster, kGrid };

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint32_t remote_addr(const void *p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
    return r;
}

// 16 bytes into CTA `rank`'s shared memory, counted by its mbarrier.
__device__ __forceinline__ void push16(const void *dst, const void *mbar, int rank, float a, float b, float c) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     remote_addr(dst, rank)),
                 "f"(a), "f"(b), "f"(c), "f"(0.0f), "r"(remote_addr(mbar, rank))
                 : "memory");
}

__device__ __forceinline__ bool wait_phase(uint64_t *mbar, uint32_t parity) {
    const uint32_t mb = smem_addr(mbar);
    uint32_t done = 0;
    const long long t0 = clock64();
    unsigned spins = 0;
    while (!done) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mb), "r"(parity)
            : "memory");
        if (!done && (++spins & 255u) == 0 && clock64() - t0 > kWaitCycles) return false;
    }
    return true;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void load_minv(const float *Minv, int row, float M[9]) {
#pragma unroll
    for (int i = 0; i < 9; ++i) M[i] = __ldg(Minv + (size_t)9 * row + i);
}

__device__ __forceinline__ void precond(const float M[9], const float r[3], float u[3], int use) {
    if (!use) {
        u[0] = r[0];
        u[1] = r[1];
        u[2] = r[2];
        return;
    }
    u[0] = M[0] * r[0] + M[1] * r[1] + M[2] * r[2];
    u[1] = M[3] * r[0] + M[4] * r[1] + M[5] * r[2];
    u[2] = M[6] * r[0] + M[7] * r[1] + M[8] * r[2];
}

__device__ __forceinline__ void block_mac(const float h[9], const float4 v, float a[3]) {
    a[0] += h[0] * v.x + h[1] * v.y + h[2] * v.z;
    a[1] += h[3] * v.x + h[4] * v.y + h[5] * v.z;
    a[2] += h[6] * v.x + h[7] * v.y + h[8] * v.z;
}

__device__ __forceinline__ void bf16_pair(uint32_t w, float &a, float &b) {
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
}

// Block k of H for the product: fp32, or the widened 16-bit values (five words
// a block; kind 1: bfloat16, else half) times the row's scale, the numbers an
// fp32 copy of the scaled blocks would hold.
__device__ __forceinline__ void load_h(const float *values, const uint32_t *words, int kind, bool full, int k,
                                       float scale, float h[9]) {
    if (full) {
        load_block9(values, k, h);
        return;
    }
    uint32_t u[5];
    load_bf16_words(words, k, u);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        float lo, hi;
        if (kind == 1) {
            bf16_pair(u[i], lo, hi);
        } else {
            __half2 q;
            memcpy(&q, &u[i], 4);
            const float2 t = __half22float2(q);
            lo = t.x;
            hi = t.y;
        }
        h[2 * i] = lo * scale;
        if (2 * i + 1 < 9) h[2 * i + 1] = hi * scale;
    }
}

// The window column of a lane of a trip: a lane without a block (src < 0)
// reads, times zero, with another lane of its quarter warp, which costs no
// bank conflict of its own.
__device__ __forceinline__ int trip_column(int src, int c, int lane) {
    const unsigned with = __ballot_sync(0xffffffffu, src >= 0) & (0xffu << (lane & 24));
    return __shfl_sync(0xffffffffu, c, src >= 0 || with == 0 ? lane : __ffs(with) - 1);
}

// The warp's sums of v[0..2], each added in the order of a shuffle-down tree
// (lane i takes lane i + 16, then + 8, ...): lanes 0, 16 and 8 return the sums
// of v[0], v[1] and v[2].  Each exchange halves what a lane carries, so three
// sums take six shuffles (a block's 16 warps otherwise spend most of a
// reduction issuing shuffles).
__device__ __forceinline__ float warp_sum3(const float v[3], int lane) {
    const bool b0 = lane & 16, b1 = lane & 8;
    float k0 = (b0 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 16);
    float k1 = v[2] + __shfl_xor_sync(0xffffffffu, v[2], 16);
    float k = (b1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 8);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
    return k;
}

__device__ __forceinline__ void spread_sum3(float k, float sum[3]) {
    sum[0] = __shfl_sync(0xffffffffu, k, 0);
    sum[1] = __shfl_sync(0xffffffffu, k, 16);
    sum[2] = __shfl_sync(0xffffffffu, k, 8);
}

// Adds two values a lane over lanes 8g .. 8g + 7 and hands group g's sum to
// every lane as sum[g].
__device__ __forceinline__ void group_sum3(float k, float sum[3]) {
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
#pragma unroll
    for (int i = 0; i < 3; ++i) sum[i] = __shfl_sync(0xffffffffu, k, 8 * i);
}

// What warp 0 decides after a reduction, for the whole CTA.
struct Verdict {
    float alpha, beta;
    int done;  // leave the loop with `status`
    int status;
};


}  // namespace
}  // namespace mfem
