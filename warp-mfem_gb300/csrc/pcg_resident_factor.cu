// Resident PCG with a factor preconditioner (M = F^T F or F F^T on H's lower
// block pattern): the single-reduction iteration of pcg_resident.cu with
// u = M r as two products of the factor's BF16 blocks,
//
//   s = w + beta s;  r -= alpha s;  p = u + beta p;  x += alpha p
//   y = F0 r;  u = F1 y;  w = H u;  gamma = (r, u), delta = (w, u), (r, r)
//
// Each CTA holds a compact block of rows (partition.cpp): H's blocks in
// registers and shared memory, the factor's in shared memory while they fit
// (20 bytes and a column each, 640-byte trips), else streamed from L2.
//
//  * kCluster: the CTAs of a cluster compute y and u of their own rows and push
//    both to the neighbours that need them, each counted by an mbarrier of its
//    own, besides w and the partial sums (three exchanges an iteration, about
//    0.3 us each).  y and u need one buffer each: a CTA pushes them only after
//    the round before, which every CTA joins after it has read its own.
//  * kGrid: a grid-wide meeting costs 2 us, so a CTA computes y and u on every
//    row that its own rows' products need (first_rows, second_rows), from r on
//    a halo of three hops that it updates with the owners' instructions: one
//    exchange an iteration.
//  * kOne: a body of one part.
//
// Measured on GB300, us an iteration with a step's other kernels, against the
// two-barrier windowed factor PCG (FSAI): 637 vertices 4.4 (6.8), 2,673 4.6 (7.3),
// 5,412 4.7 (7.4), 18,785 6.5 (10.0), 7,560 shuffled 6.1 (25.0, the global-memory
// PCG).  What bounds it: the exchange (2.1 us on the grid) and the passes'
// shared-memory reads of the factor and, with bank conflicts, of the window.
//
// A breakdown (non-finite values or a denominator <= 0) starts the solve again
// with block-Jacobi, inside the launch.  As an inner solve of the refinement H
// is read from the 16-bit blocks until the refinement has switched to fp32, and
// where it stands in for the global-memory inner PCG (pcg_mixed.cu) its dot
// products, partial sums and scalars are fp64 as that one's are (FSAI at 7,560
// shuffled rows: 10.9 us an iteration, with fp32 sums 7.1, that form 27.9).
#include "resident_common.cuh"

#include <algorithm>

namespace mfem {
namespace {

constexpr int kFTrip = 40;  // uint4 a trip of 32 factor blocks: 32 x 16 bytes, then 32 x 4
constexpr int kMaxFSlices = 64;

struct FactorArgs {
    ResidentViews v;
    const float *values, *Minv, *b;
    float *x;
    int n;
    int *error;
    SolveStats *stats;  // [slot][bodies]
    int slot, bodies;
    float tol;
    int maxiter;
    const uint32_t *fwords[2];  // the passes' BF16 blocks, five words each
    int nown_max, nhalo_max, push_max, fpush_max, smem_trips, stream_trips;
    int f_trips[2], f_shared[2];
    // kGrid: published rows [2][n], partial sums [2][CTAs][4], barrier arrivals
    float4 *pub;
    void *partials;
    unsigned long long *counter;
    // an inner solve of the refinement: its state words, (1 / ||r||, ||r||), and
    // H's 16-bit blocks (kind 1 BF16, 2 FP16; null: fp32) with row scales
    int *ir_state;
    const float *ir_scale;
    const uint32_t *values_w;
    const float *row_scale;
    int lowp_kind;
};

// Sum: what dot products, partial sums and the scalars are held in.
template <Scope SCOPE, int RS, class Sum = float>
__global__ void __launch_bounds__(kPartThreads, 1) pcg_resident_factor_kernel(FactorArgs a) {
    constexpr int KR = kPartRegTrips;
    constexpr bool kWide = sizeof(Sum) > sizeof(float);
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Sum s_red[3][kPartWarps];
    __shared__ __align__(16) typename Part<Sum>::type s_part[2][kPartMaxCluster];
    __shared__ __align__(8) uint64_t s_mbar[4];  // rounds (two), y, u
    __shared__ __align__(16) Verdict s_verdict;
    __shared__ Sum s_norm[2];
    __shared__ int s_err, s_ok[2];
    __shared__ int s_ftrips[2][kMaxFSlices];  // (first trip << 8 | trips) of each slice of a pass
    const int nall = a.nown_max + a.nhalo_max;
    float4 *rwin = reinterpret_cast<float4 *>(smem);
    float4 *ywin = rwin + nall;
    float4 *win = ywin + nall;  // u, and x0 at the start
    float4 *halo_w = win + nall;
    float4 *trips_s = halo_w + (SCOPE == kCluster ? 2 * a.nhalo_max : 0);
    uint4 *f_s = reinterpret_cast<uint4 *>(trips_s + (size_t)kPartWarps * a.smem_trips * kTripFloats4);
    int *push_s = reinterpret_cast<int *>(
        f_s + (size_t)kFTrip * ((a.f_shared[0] ? a.f_trips[0] : 0) + (a.f_shared[1] ? a.f_trips[1] : 0)));

    int *fpush_s = push_s + a.push_max;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool inner = a.ir_state != nullptr;
    bool full = true;
    if (inner) {
        const volatile int *st = a.ir_state;
        if (st[0] != 0 || st[7] != 0) return;
        full = a.values_w == nullptr || st[6] != 0;
    }
    int ncta = 1, rank = 0;
    if (SCOPE == kCluster) {
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    } else if (SCOPE == kGrid) {
        ncta = gridDim.x;
        rank = blockIdx.x;
    }
    const int4 task = a.v.tasks[SCOPE == kGrid ? 0 : blockIdx.x / ncta];
    const ResPart part = a.v.parts[task.x + rank];
    unsigned long long target = 0;  // kGrid, warp 0: arrivals that release the next barrier
    if (tid == 0) {
        s_err = *(const volatile int *)a.error;
        if (SCOPE == kCluster) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_mbar[i])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    if (SCOPE == kGrid && warp == 0) target = grid_count(a.counter) / ncta * ncta;
    if (SCOPE == kCluster && tid < 2 * kPartMaxCluster) s_part[0][tid] = typename Part<Sum>::type{};
    __syncthreads();
    int err = s_err;
    if (SCOPE == kCluster) {
        // every CTA takes the verdict of the first
        cluster_sync();
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(err) : "r"(remote_addr(&s_err, 0)));
    }
    if (err != 0) {
        if (rank == 0 && tid == 0) {
            if (inner) {
                a.ir_state[5] = MFEM_TIMEOUT;
                a.ir_state[0] = 1;
            } else {
                a.stats[(size_t)a.slot * a.bodies + task.z] = SolveStats{0, MFEM_TIMEOUT, 0.0f, 0.0f};
            }
        }
        if (SCOPE == kCluster) cluster_sync();  // no CTA leaves while another reads its flag
        return;
    }
    const int fslices = (part.nown + kFactorSliceRows - 1) / kFactorSliceRows;  // of own rows
    if (SCOPE == kCluster) {
        for (int i = tid; i < part.push_passes * part.nslices * 32; i += kPartThreads)
            push_s[i] = a.v.push[part.push_off + i];
        for (int i = tid; i < part.fpush_passes * fslices * 32; i += kPartThreads)
            fpush_s[i] = a.v.fpush[part.fpush_off + i];
    }

    // ---- this thread's local rows: local0 + 512 j, own rows first.  Halo row h
    // sits at hbase + h of the windows, the same place in every CTA of a cluster.
    const int local0 = (warp + kPartWarps * (lane >> 3)) * kPartSliceRows + (lane & 7);
    const int nlocal = part.nown + part.nhalo;
    const int hbase = SCOPE == kCluster ? a.nown_max : part.nown;
    auto place = [&](int l) { return l < part.nown ? l : l - part.nown + hbase; };
    const bool own = local0 < part.nown;
    int row_id[RS];
    float x[3], p[3], u[3], w[3], r[RS][3], s[RS][3];
#pragma unroll
    for (int j = 0; j < RS; ++j) {
        const int l = local0 + j * kPartThreads;
        row_id[j] = l >= nlocal ? -1 : l < part.nown ? a.v.rows[part.row_off + l] : a.v.halo[part.halo_off + l - part.nown];
    }
    // ---- this warp's blocks of H: the first slice's first trips in registers,
    // then in shared memory and last in a global buffer of the CTA's own
    float hreg[KR][9];
    unsigned creg[KR / 2] = {0};
    int nreg = 0;
    unsigned ntrips = 0;
    float4 *const trips_w = trips_s + (size_t)warp * a.smem_trips * kTripFloats4;
    float4 *const stream_w = a.v.stream + (size_t)((task.x + rank) * kPartWarps + warp) * a.stream_trips * kTripFloats4;
    {
        int done = 0;
        for (int q = 0; q < 4; ++q) {
            const int sl = warp + kPartWarps * q;
            if (sl >= part.nslices) break;
            const int t0 = a.v.trip_ptr[part.slice_off + sl], t1 = a.v.trip_ptr[part.slice_off + sl + 1];
            ntrips |= (unsigned)(t1 - t0) << (8 * q);
            const int i = sl * kPartSliceRows + (lane & 7);
            const float scale = full || i >= part.nown ? 1.0f : __ldg(a.row_scale + a.v.rows[part.row_off + i]);
            auto fetch = [&](int t, float h[9], int &c) {
                const int src = a.v.src[(size_t)32 * t + lane];
                c = place(a.v.col[(size_t)32 * t + lane]);
                if (src >= 0) {
                    load_h(a.values, a.values_w, a.lowp_kind, full, src, scale, h);
                } else {
#pragma unroll
                    for (int e = 0; e < 9; ++e) h[e] = 0.0f;
                }
            };
            int t = t0;
            if (q == 0) {
                nreg = min(KR, t1 - t0);
#pragma unroll
                for (int k = 0; k < KR; ++k)
                    if (k < nreg) {
                        int c;
                        fetch(t0 + k, hreg[k], c);
                        creg[k / 2] |= (unsigned)c << (16 * (k & 1));
                    }
                t += nreg;
            }
            for (; t < t1; ++t, ++done) {
                float h[9];
                int c;
                fetch(t, h, c);
                float4 *dst = done < a.smem_trips ? trips_w + done * kTripFloats4
                                                  : stream_w + (size_t)(done - a.smem_trips) * kTripFloats4;
                dst[lane] = make_float4(h[0], h[1], h[2], h[3]);
                dst[32 + lane] = make_float4(h[4], h[5], h[6], h[7]);
                reinterpret_cast<float2 *>(dst + 64)[lane] = make_float2(h[8], __int_as_float(c));
            }
        }
    }
    // ---- and of the factor's passes, slice after slice, in shared memory or
    // the global buffer
    uint4 *const f_g = a.v.fstream + (size_t)(task.x + rank) * (a.f_trips[0] + a.f_trips[1]) * kFTrip;
    uint4 *const f_base[2] = {a.f_shared[0] ? f_s : f_g,
                              a.f_shared[1] ? f_s + (a.f_shared[0] ? a.f_trips[0] : 0) * kFTrip
                                            : f_g + (size_t)a.f_trips[0] * kFTrip};
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        const int first = a.v.ftrip_ptr[part.fslice_off[f]];
        for (int sl = warp; sl < part.nfslices[f]; sl += kPartWarps) {
            const int t0 = a.v.ftrip_ptr[part.fslice_off[f] + sl], t1 = a.v.ftrip_ptr[part.fslice_off[f] + sl + 1];
            if (lane == 0) s_ftrips[f][sl] = (t0 - first) << 8 | (t1 - t0);
            uint4 *dst = f_base[f] + (size_t)(t0 - first) * kFTrip;
            for (int t = t0; t < t1; ++t, dst += kFTrip) {
                const int src = a.v.fsrc[(size_t)32 * t + lane], c = place(a.v.fcol[(size_t)32 * t + lane]);
                uint32_t q[5] = {0, 0, 0, 0, 0};
                if (src >= 0) load_bf16_words(a.fwords[f], src, q);
                dst[lane] = make_uint4(q[0], q[1], q[2], q[3]);
                reinterpret_cast<uint32_t *>(dst + 32)[lane] = (q[4] & 0xffffu) | (unsigned)c << 16;
            }
        }
    }

    auto push_row = [&](float4 *dst, uint64_t *mbar, int q, const float v[3]) {
        const int *d = push_s + (warp + kPartWarps * q) * 32 + lane;
        for (int e = 0; e < part.push_passes; ++e, d += part.nslices * 32)
            if (*d >= 0) push16(dst + (*d & 0xffff), mbar, *d >> 16, v[0], v[1], v[2]);
    };
    auto expect = [&](uint64_t *mbar, int values) {  // of 16 bytes
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(mbar)),
                     "r"(16u * (uint32_t)values)
                     : "memory");
    };
    auto reduce_row = [&](float acc[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 16);
            acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 8);
        }
    };
    // w of this thread's own row: H times the window (0 times it with `zero`);
    // row_done(slice of the warp, sum) may change a row's sum and pushes it
    auto product = [&](bool zero, auto row_done) {
        int done = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int count = (ntrips >> (8 * q)) & 0xff;
            if (count == 0) break;
            float acc[3] = {0.0f, 0.0f, 0.0f};
            if (!zero) {
                if (q == 0) {
#pragma unroll
                    for (int k = 0; k < KR; ++k)
                        if (k < nreg) block_mac(hreg[k], win[(creg[k / 2] >> (16 * (k & 1))) & 0xffffu], acc);
                    count -= nreg;
                }
                const int ns = min(count, max(0, a.smem_trips - done));
                const float4 *src = trips_w + done * kTripFloats4;
#pragma unroll 2
                for (int t = 0; t < ns; ++t, src += kTripFloats4) {
                    const float4 h0 = src[lane], h1 = src[32 + lane];
                    const float2 h2 = reinterpret_cast<const float2 *>(src + 64)[lane];
                    const float h[9] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w, h2.x};
                    block_mac(h, win[__float_as_int(h2.y)], acc);
                }
                src = stream_w + (size_t)(done + ns - a.smem_trips) * kTripFloats4;
#pragma unroll 4
                for (int t = ns; t < count; ++t, src += kTripFloats4) {
                    const float4 h0 = __ldcg(src + lane), h1 = __ldcg(src + 32 + lane);
                    const float2 h2 = __ldcg(reinterpret_cast<const float2 *>(src + 64) + lane);
                    const float h[9] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w, h2.x};
                    block_mac(h, win[__float_as_int(h2.y)], acc);
                }
                done += count;
                reduce_row(acc);
            }
            row_done(q, acc);
            if ((lane >> 3) == q) {
#pragma unroll
                for (int c = 0; c < 3; ++c) w[c] = acc[c];
            }
        }
    };
    // Pass f of the factor, a lane a row: row_done(row, sum).  A warp takes 32 rows
    // at once: with four lanes a row as in the product, most of a pass was
    // issue slots for shuffles and per-row work.
    auto factor_pass = [&](int f, const float4 *in, int rows, auto row_done) {
        for (int sl = warp; sl < part.nfslices[f]; sl += kPartWarps) {
            const int count = s_ftrips[f][sl] & 0xff, at = (s_ftrips[f][sl] >> 8) * kFTrip;
            float acc[3] = {0.0f, 0.0f, 0.0f};
            auto mac = [&](const uint4 m, const uint32_t e) {
                float h[9];
                bf16_pair(m.x, h[0], h[1]);
                bf16_pair(m.y, h[2], h[3]);
                bf16_pair(m.z, h[4], h[5]);
                bf16_pair(m.w, h[6], h[7]);
                h[8] = __uint_as_float(e << 16);
                const float4 v = in[e >> 16];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    acc[c] = __fmaf_rn(h[3 * c], v.x, acc[c]);
                    acc[c] = __fmaf_rn(h[3 * c + 1], v.y, acc[c]);
                    acc[c] = __fmaf_rn(h[3 * c + 2], v.z, acc[c]);
                }
            };
            if (a.f_shared[f]) {
                const uint4 *q = f_s + (f == 1 && a.f_shared[0] ? a.f_trips[0] * kFTrip : 0) + at;
#pragma unroll 4
                for (int t = 0; t < count; ++t, q += kFTrip)
                    mac(q[lane], reinterpret_cast<const uint32_t *>(q + 32)[lane]);
            } else {
                const uint4 *q = f_base[f] + at;
#pragma unroll 4
                for (int t = 0; t < count; ++t, q += kFTrip)
                    mac(__ldcg(q + lane), __ldcg(reinterpret_cast<const uint32_t *>(q + 32) + lane));
            }
            const int row = sl * kFactorSliceRows + lane;
            if (row < rows) row_done(row, acc);
        }
    };
    // own row's value to the parts that need it, a lane a row
    auto push_own = [&](float4 *dst, uint64_t *mbar, int row, const float v[3]) {
        const int *d = fpush_s + row;  // slices of 32 rows: the row is the index
        for (int e = 0; e < part.fpush_passes; ++e, d += fslices * 32)
            if (*d >= 0) push16(dst + (*d & 0xffff), mbar, *d >> 16, v[0], v[1], v[2]);
    };
    // The CTA's verdict on warp 0's wait for y (0) or u (1): a word each, so that
    // none is written before every thread has read the last one.
    auto joined = [&](int which, bool ok) {
        if (tid == 0) s_ok[which] = ok;
        __syncthreads();
        return s_ok[which] != 0;
    };

    // Round k: the sums of v[] over the body's own rows, on which warp 0 alone
    // decides, and w of the halo rows (pcg_resident.cu's exchange).
    float halo_v[SCOPE == kGrid ? RS : 1][3];
    auto exchange = [&](unsigned k, const Sum v[3], auto decide) -> Verdict {
        const int buf = k & 1;
        // (fp64: a warp without rows spares the SM's fp64 pipe)
        const Sum k3 = kWide && ntrips == 0 ? (Sum)0.0f : warp_sum3(v, lane);
        if ((lane & 7) == 0 && lane < 24) s_red[lane == 0 ? 0 : lane == 16 ? 1 : 2][warp] = k3;
        __syncthreads();
        Sum sum[3];
        const int g = min(lane >> 3, 2), i = lane & 7;
        bool ok = true;
        if (warp == 0) {
            if (SCOPE == kCluster && lane == 0) expect(&s_mbar[buf], (int)(sizeof(Sum) / 4) * ncta + part.nhalo);
            group_sum3(s_red[g][i] + s_red[g][i + 8], sum);
            if (SCOPE == kCluster) {
                if (lane < ncta) push_sums(&s_part[buf][rank], &s_mbar[buf], lane, sum);
                ok = __all_sync(0xffffffffu, wait_phase(&s_mbar[buf], (k >> 1) & 1u));
                const Sum *t = reinterpret_cast<const Sum *>(s_part[buf]) + g;
                group_sum3(t[4 * i] + t[4 * (i + 8)], sum);
            }
            if (SCOPE == kGrid) {
                target += ncta;
                if (lane == 0) {
                    put_sums(static_cast<Sum *>(a.partials), buf * ncta + rank, sum);
                    grid_arrive(a.counter);
                    const long long t0 = clock64();
                    unsigned spins = 0;
                    while (grid_count(a.counter) < target)
                        if ((++spins & 1023u) == 0 &&
                            (*(const volatile int *)a.error != 0 || clock64() - t0 > kWaitCycles)) {
                            ok = false;
                            break;
                        }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
            }
        }
        if (SCOPE == kGrid) {
            // halo rows and partial sums in one round trip
            __syncthreads();
#pragma unroll
            for (int j = 0; j < RS; ++j) {
                if (row_id[j] < 0 || (j == 0 && own)) continue;
                const float4 t = __ldcg(a.pub + (size_t)buf * a.n + row_id[j]);
                halo_v[j][0] = t.x;
                halo_v[j][1] = t.y;
                halo_v[j][2] = t.z;
            }
            if (warp == 0) {
                Sum t[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int b = 0; b < kPartMaxGrid / 32; ++b) {
                    const int c = lane + 32 * b;
                    add_sums(static_cast<const Sum *>(a.partials), buf * ncta + c, c < ncta, t);
                }
                spread_sum3(warp_sum3(t, lane), sum);
            }
        }
        if (warp == 0 && lane == 0) {
            Verdict d;
            if (ok) d = decide(sum);
            else d = Verdict{0.0f, 0.0f, 1, MFEM_TIMEOUT};
            s_verdict = d;
        }
        __syncthreads();
        return s_verdict;
    };
    auto publish = [&](unsigned k) {
        if (SCOPE == kGrid && own)
            a.pub[(size_t)(k & 1) * a.n + row_id[0]] = make_float4(w[0], w[1], w[2], 0.0f);
    };

    bool factor = true;    // false after a breakdown: block-Jacobi
    unsigned phases = 0;   // exchanges of y and of u so far
    // r over the local rows (with `update` s = w + beta s, r -= alpha s, and p,
    // x of the own row; else r = w), then u = M r over the rows that the
    // product's columns reach.  False: a wait gave up.
    auto precondition = [&](unsigned k, bool update, float alpha, float beta, bool first) {
#pragma unroll
        for (int j = 0; j < RS; ++j) {
            const int l = local0 + j * kPartThreads;
            if (l >= nlocal) continue;
            float v[3];
            if (j == 0 && own) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = w[c];
            } else if (SCOPE == kCluster) {
                const float4 t = halo_w[(k & 1) * a.nhalo_max + l - part.nown];
                v[0] = t.x;
                v[1] = t.y;
                v[2] = t.z;
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = SCOPE == kGrid ? halo_v[SCOPE == kGrid ? j : 0][c] : 0.0f;
            }
            if (update) {
                if (j == 0) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {  // own rows'; a halo row's are not used
                        p[c] = first ? u[c] : __fmaf_rn(beta, p[c], u[c]);
                        x[c] = __fmaf_rn(alpha, p[c], x[c]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    s[j][c] = first ? v[c] : __fmaf_rn(beta, s[j][c], v[c]);
                    r[j][c] = __fmaf_rn(-alpha, s[j][c], r[j][c]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    r[j][c] = v[c];
                    s[j][c] = 0.0f;
                }
            }
            if (factor) {
                rwin[place(l)] = make_float4(r[j][0], r[j][1], r[j][2], 0.0f);
            } else if (l < part.second_rows) {
                float m[9], z[3];
                load_minv(a.Minv, row_id[j], m);
                precond(m, r[j], z, 1);
                win[place(l)] = make_float4(z[0], z[1], z[2], 0.0f);
            }
        }
        bool ok = true;
        const unsigned phase = phases++ & 1u;
        if (factor) {
            __syncthreads();
            factor_pass(0, rwin, part.first_rows, [&](int l, float acc[3]) {
                ywin[place(l)] = make_float4(acc[0], acc[1], acc[2], 0.0f);
                if (SCOPE == kCluster) push_own(ywin + a.nown_max, &s_mbar[2], l, acc);
            });
        }
        if (SCOPE == kCluster) {
            // (y is exchanged only with the factor, but its phase advances
            // with u's)
            if (tid == 0) expect(&s_mbar[2], factor ? part.nhalo : 0);
            if (warp == 0) ok = __all_sync(0xffffffffu, wait_phase(&s_mbar[2], phase));
            if (!joined(0, ok)) return false;
        } else {
            __syncthreads();
        }
        if (factor) {
            factor_pass(1, ywin, part.second_rows, [&](int l, float acc[3]) {
                win[place(l)] = make_float4(acc[0], acc[1], acc[2], 0.0f);
                if (SCOPE == kCluster) push_own(win + a.nown_max, &s_mbar[3], l, acc);
            });
        } else if (SCOPE == kCluster) {
            // the own rows' u to the neighbours
            for (int l = tid; l < part.nown; l += kPartThreads) {
                const float4 z = win[l];
                const float v[3] = {z.x, z.y, z.z};
                push_own(win + a.nown_max, &s_mbar[3], l, v);
            }
        }
        if (SCOPE == kCluster) {
            if (tid == 0) expect(&s_mbar[3], part.nhalo);
            if (warp == 0) ok = __all_sync(0xffffffffu, wait_phase(&s_mbar[3], phase));
            if (!joined(1, ok)) return false;
        } else {
            __syncthreads();
        }
        if (own) {
            const float4 z = win[local0];
            u[0] = z.x;
            u[1] = z.y;
            u[2] = z.z;
        }
        return true;
    };
    auto dots = [&](Sum (&sum)[3]) {
        sum[0] = sum[1] = sum[2] = 0.0f;
        add_rows(r[0], u, w, own, lane, sum);
    };

    const float bscale = inner ? a.ir_scale[0] : 1.0f;
    unsigned round = 0;
    int it = 0, it_done = 0;
    Verdict d;
    for (;;) {  // one attempt
        it = 0;
        __syncthreads();
        // ---- r0 = g - H x0 (x0 = 0 for an inner solve)
#pragma unroll
        for (int j = 0; j < RS; ++j) {
            float v[3] = {0.0f, 0.0f, 0.0f};
            const int l = local0 + j * kPartThreads;
            if (!inner && row_id[j] >= 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = a.x[(size_t)3 * row_id[j] + c];
                win[place(l)] = make_float4(v[0], v[1], v[2], 0.0f);
            }
            if (j == 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    x[c] = v[c];
                    p[c] = u[c] = w[c] = 0.0f;
                }
            }
        }
        __syncthreads();
        product(inner, [&](int q, float acc[3]) {
            const int i = (warp + kPartWarps * q) * kPartSliceRows + (lane & 7);
            if (i < part.nown) {
                const int row = a.v.rows[part.row_off + i];
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[c] = __ldg(a.b + (size_t)3 * row + c) * bscale - acc[c];
            }
            if (SCOPE == kCluster) push_row(halo_w + (round & 1) * a.nhalo_max, &s_mbar[round & 1], q, acc);
        });
        publish(round);
        Sum sum[3] = {0.0f, 0.0f, 0.0f};
        if (own) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float g = __ldg(a.b + (size_t)3 * row_id[0] + c) * bscale;
                add_product(g, g, sum[0]);
            }
        }
        // the recurrence's scalars, kept by thread 0 (||g||^2 and (r, r) in s_norm)
        Sum thr2 = 0.0f, gamma = 0.0f, alpha = 0.0f;  // fp64: alpha holds the last denominator
        d = exchange(round, sum, [&](const Sum t[3]) {
            s_norm[0] = t[0];
            s_norm[1] = 0.0f;
            thr2 = (Sum)a.tol * a.tol * t[0];
            return Verdict{0.0f, 0.0f, 0, MFEM_OK};
        });
        const Verdict lost{0.0f, 0.0f, 1, MFEM_TIMEOUT};
        auto push_w = [&](int q, float acc[3]) {
            if (SCOPE == kCluster)
                push_row(halo_w + ((round + 1) & 1) * a.nhalo_max, &s_mbar[(round + 1) & 1], q, acc);
        };
        if (!d.done && !precondition(round, false, 0.0f, 0.0f, true)) d = lost;
        if (!d.done) {
            product(false, push_w);
            publish(round + 1);
            dots(sum);
            d = exchange(++round, sum, [&](const Sum t[3]) {
                gamma = t[0];
                const Sum rr = t[2];
                s_norm[1] = rr;
                const Sum first = t[1] > 0.0f ? gamma / t[1] : 0.0f;
                alpha = kWide ? t[1] : first;
                int status = MFEM_OK;
                if (!isfinite(gamma) || !isfinite(t[1]) || !isfinite(rr) || !isfinite(s_norm[0])) status = MFEM_NONFINITE;
                else if (!(t[1] > 0.0f) && rr > 0.0f) status = MFEM_STAGNATION;
                // a right-hand side that is met needs no factor
                if (status != MFEM_NONFINITE && rr <= thr2) status = MFEM_OK;
                int done = status != MFEM_OK || rr <= thr2;
                if (!done && a.maxiter <= 0) {
                    done = 1;
                    status = MFEM_MAXITER;
                }
                return Verdict{(float)first, 0.0f, done, status};
            });
        }
        while (!d.done) {
            if (!precondition(round, true, d.alpha, d.beta, it == 0)) {
                d = lost;
                break;
            }
            product(false, push_w);
            publish(round + 1);
            dots(sum);
            ++it;
            d = exchange(++round, sum, [&](const Sum t[3]) {
                const Sum rr = t[2];
                s_norm[1] = rr;
                if (!isfinite(t[0]) || !isfinite(t[1]) || !isfinite(rr)) return Verdict{0.0f, 0.0f, 1, MFEM_NONFINITE};
                if (rr <= thr2) return Verdict{0.0f, 0.0f, 1, MFEM_OK};
                const Sum beta = t[0] / gamma;
                // the ratio in flight with beta, or (a slow fp64 division less) from
                // the last denominator gamma / alpha
                const Sum denom = kWide ? t[1] - beta * beta * alpha : t[1] - beta * (t[0] / alpha);
                if (!(denom > 0.0f)) return Verdict{0.0f, 0.0f, 1, MFEM_STAGNATION};
                const Sum next = t[0] / denom;
                alpha = kWide ? denom : next;
                gamma = t[0];
                return Verdict{(float)next, (float)beta, it >= a.maxiter, it >= a.maxiter ? MFEM_MAXITER : MFEM_OK};
            });
        }
        ++round;  // the next attempt's first
        if (factor && (d.status == MFEM_STAGNATION || d.status == MFEM_NONFINITE)) {
            it_done += it;
            factor = false;
            continue;
        }
        break;
    }
    if (d.status == MFEM_TIMEOUT && tid == 0) atomicExch(a.error, 1);
    const float es = inner ? a.ir_scale[1] : 1.0f;
    if (own) {
        const int row = a.v.rows[part.row_off + local0];
#pragma unroll
        for (int c = 0; c < 3; ++c) a.x[(size_t)3 * row + c] = x[c] * es;
    }
    if (rank == 0 && tid == 0) {
        if (inner) {
            // a solve that stopped at the cap or stagnated still hands over
            // its iterate; a 16-bit H that broke it restarts on the fp32 H
            a.ir_state[2] += it_done + it;
            a.ir_state[3] = 1;
            if (d.status == MFEM_NONFINITE && !full) {
                a.ir_state[3] = 0;
                a.ir_state[6] = 1;
                a.ir_state[7] = 1;
            } else if (d.status == MFEM_TIMEOUT || d.status == MFEM_NONFINITE) {
                a.ir_state[5] = d.status;
                a.ir_state[0] = 1;
            }
        } else {
            const float bb = (float)s_norm[0], rr = (float)s_norm[1];
            const float rel = d.status == MFEM_TIMEOUT ? 0.0f : bb > 0.0f ? sqrtf(rr / bb) : sqrtf(rr);
            a.stats[(size_t)a.slot * a.bodies + task.z] = SolveStats{it_done + it, d.status, rel, 0.0f};
        }
    }
    if (SCOPE == kCluster) cluster_sync();  // no CTA leaves while another may still push to it
}

typedef void (*FacKernel)(FactorArgs);

// With fp64 sums, for the mixed refinement's inner solves (grids only).
FacKernel pick_wide(const ResidentLayout &L) {
    return L.row_slots <= 2 ? pcg_resident_factor_kernel<kGrid, 2, double>
                            : pcg_resident_factor_kernel<kGrid, 3, double>;
}

FacKernel pick(const ResidentLayout &L) {
    if (L.grid) return L.row_slots <= 2 ? pcg_resident_factor_kernel<kGrid, 2> : pcg_resident_factor_kernel<kGrid, 3>;
    if (L.cluster <= 1) return pcg_resident_factor_kernel<kOne, 1>;
    return L.row_slots <= 2 ? pcg_resident_factor_kernel<kCluster, 2> : pcg_resident_factor_kernel<kCluster, 3>;
}

cudaLaunchConfig_t launch_config(const ResidentLayout &L, int n_tasks, cudaLaunchAttribute attr[1], cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_tasks * L.cluster));
    cfg.blockDim = dim3(kPartThreads);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = s;
    if (L.grid) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.numAttrs = 1;
    } else if (L.cluster > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = L.cluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.numAttrs = 1;
    }
    cfg.attrs = attr;
    return cfg;
}

}  // namespace

cudaError_t resident_factor_layout(int device, const ResidentHost &h, int cluster, bool grid, ResidentLayout &L,
                                   bool &fits) {
    fits = false;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    L = ResidentLayout{};
    L.factor = true;
    L.cluster = cluster;
    L.grid = grid;
    L.nown_max = h.nown_max;
    L.nhalo_max = h.nhalo_max;
    L.row_slots = std::max(1, (h.nlocal_max + kPartThreads - 1) / kPartThreads);
    const bool one = !grid && cluster <= 1;
    int slices = 0;
    for (const ResPart &p : h.parts) slices = std::max(slices, std::max(p.nfslices[0], p.nfslices[1]));
    if (h.nown_max > kPartThreads || L.row_slots > (one ? 1 : 3) || h.slice_trips_max > 255 || slices > kMaxFSlices)
        return cudaSuccess;
    const FacKernel k = pick(L);
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, k);
    if (e != cudaSuccess) return e;
    size_t fixed = fa.sharedSizeBytes;
    if (grid) {  // the same layout serves the fp64 sums
        e = cudaFuncGetAttributes(&fa, pick_wide(L));
        if (e != cudaSuccess) return e;
        fixed = std::max(fixed, fa.sharedSizeBytes);
    }
    const size_t most = (size_t)optin - fixed;
    L.push_max = !grid && cluster > 1 ? h.push_max : 0;
    L.fpush_max = !grid && cluster > 1 ? h.fpush_max : 0;
    size_t left = sizeof(float4) * (3 * ((size_t)h.nown_max + h.nhalo_max) + (L.push_max ? 2 * (size_t)h.nhalo_max : 0)) +
                  sizeof(int) * (size_t)(L.push_max + L.fpush_max) + 16;
    if (left > most) return cudaSuccess;
    L.smem = left;
    left = most - left;
    // the factor first (a pass waits on every trip), then H's further trips
    for (int w = 0; w < 2; ++w) {
        L.f_trips[w] = h.f_trips_max[w];
        const size_t bytes = sizeof(uint4) * kFTrip * (size_t)L.f_trips[w];
        L.f_shared[w] = bytes <= left;
        if (!L.f_shared[w]) continue;
        left -= bytes;
        L.smem += bytes;
    }
    const size_t per_trip = sizeof(float4) * kTripFloats4 * kPartWarps;
    L.smem_trips = (int)std::min<size_t>(h.trips_max_reg, left / per_trip);
    L.stream_trips = h.trips_max_reg - L.smem_trips;
    L.smem = (L.smem + per_trip * L.smem_trips + 15) & ~(size_t)15;
    if (L.smem > most) return cudaSuccess;
    // the limit is the kernel's, not the plan's: every plan sets the same one
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess && grid)
        e = cudaFuncSetAttribute(pick_wide(L), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess && !grid && cluster > 8)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    fits = true;
    if (!grid && cluster > 1) {
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = launch_config(L, 1, attr, 0);
        int active = 0;
        e = cudaOccupancyMaxActiveClusters(&active, k, &cfg);
        fits = e == cudaSuccess && active > 0;
    }
    return e;
}

cudaError_t launch_resident_factor(const BsrViews &bv, const VertexViews &vv, const ResidentLayout &L, int n_tasks,
                                   int n_bodies, const PcgWork &w, const BatchViews &bw, SolveStats *stats, int slot,
                                   float tol, int maxiter, int mode, const IrWork *ir, cudaStream_t s) {
    FactorArgs a = {};
    a.v = L.v;
    a.values = bv.values;
    a.Minv = vv.Minv;
    a.b = ir ? ir->res : vv.rhs;
    a.x = ir ? ir->e : vv.dx;
    a.n = bv.n;
    a.error = w.error;
    a.stats = stats;
    a.slot = slot;
    a.bodies = n_bodies;
    a.tol = ir ? ir->inner_tol : tol;
    a.maxiter = maxiter;
    const __nv_bfloat16 *first = mode == 2 ? bw.Lb : bw.Ub, *second = mode == 2 ? bw.Ub : bw.Lb;
    a.fwords[0] = reinterpret_cast<const uint32_t *>(first);
    a.fwords[1] = reinterpret_cast<const uint32_t *>(second);
    a.nown_max = L.nown_max;
    a.nhalo_max = L.nhalo_max;
    a.push_max = L.push_max;
    a.fpush_max = L.fpush_max;
    a.smem_trips = L.smem_trips;
    a.stream_trips = L.stream_trips;
    for (int i = 0; i < 2; ++i) {
        a.f_trips[i] = L.f_trips[i];
        a.f_shared[i] = L.f_shared[i] ? 1 : 0;
    }
    a.pub = reinterpret_cast<float4 *>(w.pub);
    const bool wide = ir && ir->wide && L.grid;
    a.partials = wide ? static_cast<void *>(ir->partials) : w.partials;
    a.counter = w.res_counter;
    if (ir) {
        a.ir_state = ir->state;
        a.ir_scale = ir->scale;
        a.values_w = ir->mode == kIrFp32 ? nullptr : ir->hq_words;
        a.row_scale = ir->row_scale;
        a.lowp_kind = ir->mode == kIrBf16 ? 1 : 2;
    }
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = launch_config(L, n_tasks, attr, s);
    cudaError_t e = cudaLaunchKernelEx(&cfg, wide ? pick_wide(L) : pick(L), a);
    count_launches(1);
    return e;
}

}  // namespace mfem
