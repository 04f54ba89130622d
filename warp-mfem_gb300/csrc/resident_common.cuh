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
__device__ __forceinline__ void push16(const void *dst, const void *mbar, int rank, float a, float b, float c,
                                       float d = 0.0f) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     remote_addr(dst, rank)),
                 "f"(a), "f"(b), "f"(c), "f"(d), "r"(remote_addr(mbar, rank))
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
template <class Sum>
__device__ __forceinline__ Sum warp_sum3(const Sum v[3], int lane) {
    const bool b0 = lane & 16, b1 = lane & 8;
    Sum k0 = (b0 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 16);
    Sum k1 = v[2] + __shfl_xor_sync(0xffffffffu, v[2], 16);
    Sum k = (b1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 8);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
    return k;
}

template <class Sum>
__device__ __forceinline__ void spread_sum3(Sum k, Sum sum[3]) {
    sum[0] = __shfl_sync(0xffffffffu, k, 0);
    sum[1] = __shfl_sync(0xffffffffu, k, 16);
    sum[2] = __shfl_sync(0xffffffffu, k, 8);
}

// Adds two values a lane over lanes 8g .. 8g + 7 and hands group g's sum to
// every lane as sum[g].
template <class Sum>
__device__ __forceinline__ void group_sum3(Sum k, Sum sum[3]) {
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
#pragma unroll
    for (int i = 0; i < 3; ++i) sum[i] = __shfl_sync(0xffffffffu, k, 8 * i);
}

// A CTA's three partial sums in shared memory, and their way into CTA `rank`'s.
template <class Sum>
struct Part {
    typedef float4 type;
};
template <>
struct Part<double> {
    struct alignas(16) type {
        double v[4];
    };
};
__device__ __forceinline__ void push_sums(const float4 *dst, const void *mbar, int rank, const float s[3]) {
    push16(dst, mbar, rank, s[0], s[1], s[2]);
}
__device__ __forceinline__ void push_sums(const Part<double>::type *part, const void *mbar, int rank,
                                          const double s[3]) {
    const double *dst = part->v;
    push16(dst, mbar, rank, __int_as_float(__double2loint(s[0])), __int_as_float(__double2hiint(s[0])),
           __int_as_float(__double2loint(s[1])), __int_as_float(__double2hiint(s[1])));
    push16(dst + 2, mbar, rank, __int_as_float(__double2loint(s[2])), __int_as_float(__double2hiint(s[2])), 0.0f);
}

// CTA c's partial sums in a grid's array of them, four numbers a CTA; add_sums
// adds those of a CTA that is in the grid.
__device__ __forceinline__ void put_sums(float *partials, int c, const float s[3]) {
    reinterpret_cast<float4 *>(partials)[c] = make_float4(s[0], s[1], s[2], 0.0f);
}
__device__ __forceinline__ void put_sums(double *partials, int c, const double s[3]) {
    double2 *d = reinterpret_cast<double2 *>(partials) + 2 * c;
    d[0] = make_double2(s[0], s[1]);
    d[1] = make_double2(s[2], 0.0);
}
__device__ __forceinline__ void add_sums(const float *partials, int c, bool in, float t[3]) {
    const float4 q = in ? __ldcg(reinterpret_cast<const float4 *>(partials) + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    t[0] += q.x;
    t[1] += q.y;
    t[2] += q.z;
}
__device__ __forceinline__ void add_sums(const double *partials, int c, bool in, double t[3]) {
    if (!in) return;
    const double2 *d = reinterpret_cast<const double2 *>(partials) + 2 * c;
    const double2 a = __ldcg(d), b = __ldcg(d + 1);
    t[0] += a.x;
    t[1] += a.y;
    t[2] += b.x;
}

__device__ __forceinline__ void add_product(float a, float b, float &sum) { sum = __fmaf_rn(a, b, sum); }
__device__ __forceinline__ void add_product(float a, float b, double &sum) { sum = fma((double)a, (double)b, sum); }

// A warp's products of r.u, w.u and r.r over the rows its lanes own (`own`),
// added to sum[].  fp32: a lane its own row.  fp64: an SM starts a warp's fp64
// instruction every 16 cycles, full or not, and with up to 128 rows a CTA
// only eight lanes of a warp own one; so for one or two groups of eight the
// components are dealt out, one a lane, and the warp issues 6 or 12 of them
// instead of 18 (7,560 rows: 8.4 -> 7.0 us an iteration).
__device__ __forceinline__ void add_rows(const float r[3], const float u[3], const float w[3], bool own, int,
                                         float sum[3]) {
    if (own) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            add_product(r[c], u[c], sum[0]);
            add_product(w[c], u[c], sum[1]);
            add_product(r[c], r[c], sum[2]);
        }
    }
}
__device__ __forceinline__ void add_rows(const float r[3], const float u[3], const float w[3], bool own, int lane,
                                         double sum[3]) {
    const unsigned owners = __ballot_sync(0xffffffffu, own);
    if (owners & 0xffff0000u) {
        if (!own) return;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            add_product(r[c], u[c], sum[0]);
            add_product(w[c], u[c], sum[1]);
            add_product(r[c], r[c], sum[2]);
        }
        return;
    }
    const int c = lane % 3;
    for (int from = lane / 3; owners >> (from - lane / 3); from += 8) {
        float v[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float *x = i == 0 ? r : i == 1 ? u : w;
            const float x0 = __shfl_sync(0xffffffffu, x[0], from), x1 = __shfl_sync(0xffffffffu, x[1], from),
                        x2 = __shfl_sync(0xffffffffu, x[2], from);
            v[i] = c == 0 ? x0 : c == 1 ? x1 : x2;
        }
        if (lane < 24 && ((owners >> from) & 1u)) {
            add_product(v[0], v[1], sum[0]);
            add_product(v[2], v[1], sum[1]);
            add_product(v[0], v[0], sum[2]);
        }
    }
}

// What warp 0 decides after a reduction, for the whole CTA.
struct Verdict {
    float alpha, beta;
    int done;  // leave the loop with `status`
    int status;
};


}  // namespace
}  // namespace mfem
