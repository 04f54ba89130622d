// Resident block-Jacobi PCG: the single-reduction (Chronopoulos & Gear 1989)
// iteration of pcg.cu on parts of a body that one CTA each holds for the
// whole solve.
//
//   s = w + beta s;  r -= alpha s;  p = u + beta p;  x += alpha p
//   u = M r;  w = H u;  gamma = (r, u), delta = (w, u), (r, r)
//   beta' = gamma' / gamma;  alpha' = gamma' / (delta' - beta' gamma' / alpha)
//
// A part is a compact block of rows (partition.cpp) and its halo, the foreign
// rows its columns reach.  Per row a thread keeps r, s, M (and x, p, u of its
// own rows) in registers: every CTA updates its halo rows with the owner's
// instructions from the same w, so owner and neighbours agree bit for bit and
// w is all that CTAs exchange.  The product runs four lanes a row, eight rows
// a warp; the first slice's blocks sit in registers, further ones in shared
// memory as 1,280-byte trips (32 blocks with their columns: two 16-byte and
// one 8-byte conflict-free load a lane).  The lane that ends up with a row's
// sum owns the row, so w needs no trip through shared memory.
//
// The same iteration with three exchanges (Scope):
//  * kCluster: the parts of a body are one cluster.  Owners push w to the
//    neighbours' halo buffers and each CTA pushes its partial sums to every
//    other with st.async; one mbarrier phase counts all bytes a CTA expects,
//    so an iteration has no barrier besides it.  Buffers alternate by round:
//    a CTA sends round k + 2 only after it has every partial of round k + 1,
//    which each CTA sent after it had read round k.
//  * kGrid: the parts are the CTAs of a cooperative grid.  Owners publish w
//    in global memory (alternating buffers, the same argument), the CTAs meet
//    at the counter barrier of grid_sync.cuh, and halo rows and partial sums
//    are loaded together.
//  * kOne: a body of one part; block reductions only.
//
// What bounds an iteration is its chain: block reduction, exchange, scalars,
// update, product; with streamed blocks (below) the L2 reads of H.  Measured on
// GB300, us an iteration, a step's other kernels included, against the windowed
// kernels of pcg.cu: 99 rows 1.1 (one CTA; 3.6), 425 to 1,225 rows 1.5 (clusters
// of 4 to 16; 3.4), 2,673 rows 1.95 (3.65), 7,560 shuffled rows 3.0 (grid; 9.0),
// 18,785 rows 3.2 (5.0), shuffled 3.5 (12.1), 140,481 rows 9.6 (19.0).
//
// Blocks that fit neither registers nor shared memory (meshes past about
// 55,000 rows) are copied once a solve into trips in global memory, which the
// warps then read in coalesced 16-byte loads, four trips in flight.
//
// As an inner solve of the mixed-precision refinement (fp32 blocks, or the
// 16-bit ones widened and scaled as they are loaded) it starts
// from 0 on the residual scaled to unit norm and updates the refinement's
// state words like the other inner solves (pcg.cu, pcg_factor.cu); where it
// stands in for the global-memory inner PCG (pcg_mixed.cu) its dot products,
// partial sums and scalars are fp64 as that one's are.
//
// Every wait is bounded; after a timeout the kernel sets the sticky error
// flag and every CTA leaves (a cluster's through one more barrier, which all
// its CTAs reach), reporting MFEM_TIMEOUT.
#include "resident_common.cuh"

#include <algorithm>

namespace mfem {
namespace {

struct ResArgs {
    ResidentViews v;
    const float *values, *Minv, *b;
    float *x;
    int n;
    int *error;
    SolveStats *stats;  // [slot][bodies]
    int slot, bodies;
    float tol;
    int maxiter, use_precond;
    int nown_max, nhalo_max, smem_trips, stream_trips, push_max;
    int blocks, block_warps;  // ordered sums: blocks of the body, warps of the longest one
    // kGrid: published rows [2][n], partial sums [2][CTAs][4], barrier arrivals
    float4 *pub;
    void *partials;
    unsigned long long *counter;
    // an inner solve of the refinement: its state words, (1 / ||r||, ||r||)
    int *ir_state;
    const float *ir_scale;
    // its 16-bit blocks, null: the fp32 ones
    const uint32_t *values_w;
    const float *row_scale;
    int lowp_kind;
};

// OS: own rows a thread keeps, RS: rows it keeps in all (the further ones
// halo rows), KR: trips of a warp's first slice kept in registers, STREAM: some
// trips do not fit in shared memory.
//
// LOWP: may load 16-bit blocks.  The large-mesh kernel has an instance without,
// which takes 9.6 us an iteration at 140,481 rows where the other's allocation
// of the same registers takes 10.0.
//
// ORDERED: the sums are added over the same blocks of consecutive rows, in the
// same order, whatever CTAs the rows sit on, and the scalars are formed as in
// the windowed single-reduction kernel (pcg.cu, which sums each CTA's range of
// rows): such a solve has that kernel's iterates bit for bit.  A part is then a
// run of whole blocks.
//
// Sum: what dot products, partial sums and the recurrence's scalars are held
// in; double for the inner solves that the global-memory inner PCG served.  A
// chain of some fifty dependent fp64 operations an iteration: 7.0 us at 7,560
// shuffled rows against 3.1 with fp32 sums (that form: 16.3).
template <Scope SCOPE, int OS, int RS, int KR, bool STREAM, bool ORDERED, bool LOWP = true, class Sum = float>
__global__ void __launch_bounds__(kPartThreads, 1) pcg_resident_kernel(ResArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int kBlocks = ORDERED && SCOPE != kGrid ? kPartMaxBlocks : 1;
    constexpr bool kWide = sizeof(Sum) > sizeof(float);
    constexpr int kSums = SCOPE == kCluster ? kPartMaxCluster * kBlocks : 1;  // partial sums of a round
    __shared__ Sum s_red[kBlocks][3][kPartWarps];
    __shared__ __align__(16) typename Part<Sum>::type s_part[2][kSums];

    __shared__ __align__(8) uint64_t s_mbar[2];
    __shared__ __align__(16) Verdict s_verdict;
    __shared__ Sum s_norm[2];
    __shared__ int s_err;
    float4 *win = reinterpret_cast<float4 *>(smem);                         // u of own rows, then of halo rows
    float4 *halo_w = win + a.nown_max + a.nhalo_max;                        // [2][nhalo_max] pushed by the owners
    float4 *trips_s = halo_w + (SCOPE == kCluster ? 2 * a.nhalo_max : 0);   // [warps][smem_trips][80]
    float *minv_s = reinterpret_cast<float *>(trips_s + (size_t)kPartWarps * a.smem_trips * kTripFloats4);
    int *push_s = reinterpret_cast<int *>(minv_s + (RS > 1 ? 9 * max(0, a.nown_max + a.nhalo_max - kPartThreads) : 0));
    // ORDERED: r, u and w of the own rows, component by component
    float *const own_r = reinterpret_cast<float *>(push_s + a.push_max), *const own_u = own_r + 3 * a.nown_max,
                 *const own_w = own_u + 3 * a.nown_max;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool inner = a.ir_state != nullptr;
    bool full = true;  // the fp32 blocks
    if (inner) {
        // nothing to do once the refinement has finished
        const volatile int *st = a.ir_state;
        if (st[0] != 0 || st[7] != 0) return;
        full = !LOWP || a.values_w == nullptr || st[6] != 0;
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
            for (int i = 0; i < 2; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_mbar[i])) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    if (SCOPE == kGrid && warp == 0) target = grid_count(a.counter) / ncta * ncta;
    for (int i = tid; SCOPE == kCluster && i < 2 * kSums; i += kPartThreads)
        s_part[i / kSums][i % kSums] = typename Part<Sum>::type{};
    if (ORDERED) {
        for (int i = tid; i < kBlocks * 3 * kPartWarps; i += kPartThreads)
            s_red[i / (3 * kPartWarps)][i / kPartWarps % 3][i % kPartWarps] = 0.0f;
    }
    // ORDERED: the part's first row, and per task of this warp (32 consecutive
    // components of a block) the lane's component, the block's end and where
    // the sum goes; -1: no task
    constexpr int kTasks = SCOPE == kCluster ? kPartTasks : 1;
    int row0 = 0, task_i[kTasks], task_end[kTasks], task_dst[kTasks];
    if (ORDERED) {
        auto block_row = [&](int b) { return (int)((long long)a.n * (part.block_lo + b) / a.blocks); };
        row0 = block_row(0);
#pragma unroll
        for (int q = 0; q < kTasks; ++q) {
            const int t = warp + kPartWarps * q, b = t / a.block_warps, wi = t - b * a.block_warps;
            task_dst[q] = b < part.nblocks ? b * 3 * kPartWarps + wi : -1;
            task_i[q] = 3 * (block_row(b) - row0) + 32 * wi + lane;
            task_end[q] = b < part.nblocks ? 3 * (block_row(b + 1) - row0) : 0;
        }
    }
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
    if (SCOPE == kCluster)
        for (int i = tid; i < part.push_passes * part.nslices * 32; i += kPartThreads)
            push_s[i] = a.v.push[part.push_off + i];

    // ---- this thread's local rows: local0 + 512 j, own rows first.  An own
    // row's thread is one of the lanes that will hold its product.
    const int local0 = (warp + kPartWarps * (lane >> 3)) * kPartSliceRows + (lane & 7);
    const int nlocal = part.nown + part.nhalo;
    int row_id[RS];  // vertex of the row, -1: none
    float x[OS][3], p[OS][3], u[OS][3], w[OS][3];
    float r[RS][3], s[RS][3], minv[9] = {0.0f};  // M of the first row; the others' sit in shared memory
#pragma unroll
    for (int j = 0; j < RS; ++j) {
        const int l = local0 + j * kPartThreads;
        row_id[j] = -1;
        float v[3] = {0.0f, 0.0f, 0.0f};
        if (l < nlocal) {
            row_id[j] = l < part.nown ? a.v.rows[part.row_off + l] : a.v.halo[part.halo_off + l - part.nown];
            float m[9];
            load_minv(a.Minv, row_id[j], m);
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                if (j == 0) minv[i] = m[i];
                else minv_s[9 * (l - kPartThreads) + i] = m[i];
            }
            if (!inner) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = a.x[(size_t)3 * row_id[j] + c];
                win[l] = make_float4(v[0], v[1], v[2], 0.0f);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) r[j][c] = s[j][c] = 0.0f;
        if (j < OS) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                x[j][c] = v[c];
                p[j][c] = u[j][c] = w[j][c] = 0.0f;
            }
        }
    }
    bool own[OS];
#pragma unroll
    for (int o = 0; o < OS; ++o) own[o] = local0 + o * kPartThreads < part.nown;

    // ---- this warp's blocks: the first slice's first trips in registers, then
    // in the order the product takes them in shared memory while it lasts and
    // in a global buffer of the CTA's own (a lane reads what it wrote)
    constexpr int kRegs = KR > 0 ? KR : 1;
    float hreg[kRegs][9];
    unsigned creg[(kRegs + 1) / 2] = {0};  // two 16-bit columns a word
    int nreg = 0;
    unsigned ntrips[OS] = {0};  // trips of the warp's slices, one byte each
    float4 *const trips_w = trips_s + (size_t)warp * a.smem_trips * kTripFloats4;
    float4 *const stream_w =
        a.v.stream + (size_t)((task.x + rank) * kPartWarps + warp) * a.stream_trips * kTripFloats4;
    {
        int done = 0;
#pragma unroll
        for (int o = 0; o < OS; ++o)
            for (int qq = 0; qq < 4; ++qq) {
                const int sl = warp + kPartWarps * (4 * o + qq);
                if (sl >= part.nslices) break;
                const int t0 = a.v.trip_ptr[part.slice_off + sl], t1 = a.v.trip_ptr[part.slice_off + sl + 1];
                ntrips[o] |= (unsigned)(t1 - t0) << (8 * qq);
                float scale = 1.0f;
                if (LOWP && !full) {
                    const int i = sl * kPartSliceRows + (lane & 7);
                    if (i < part.nown) scale = __ldg(a.row_scale + a.v.rows[part.row_off + i]);
                }
                auto fetch = [&](int t, float h[9], int &c) {
                    const int src = a.v.src[(size_t)32 * t + lane];
                    c = trip_column(src, a.v.col[(size_t)32 * t + lane], lane);
                    if (src >= 0) {
                        if (LOWP) load_h(a.values, a.values_w, a.lowp_kind, full, src, scale, h);
                        else load_block9(a.values, src, h);
                    } else {
#pragma unroll
                        for (int i = 0; i < 9; ++i) h[i] = 0.0f;
                    }
                };
                int t = t0;
                if (KR > 0 && o == 0 && qq == 0) {
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
                    float4 *dst = !STREAM || done < a.smem_trips ? trips_w + done * kTripFloats4
                                                      : stream_w + (size_t)(done - a.smem_trips) * kTripFloats4;
                    dst[lane] = make_float4(h[0], h[1], h[2], h[3]);
                    dst[32 + lane] = make_float4(h[4], h[5], h[6], h[7]);
                    reinterpret_cast<float2 *>(dst + 64)[lane] = make_float2(h[8], __int_as_float(c));
                }
            }
    }
    const int first_trips = ntrips[0] & 0xff;
    const unsigned more_trips = ntrips[0] >> 8;  // 0: one slice at most
    __syncthreads();  // the window holds x0

    auto push_row = [&](unsigned k, int q, const float v[3]) {
        const int buf = k & 1;
        const int *d = push_s + (warp + kPartWarps * q) * 32 + lane;
        for (int e = 0; e < part.push_passes; ++e, d += part.nslices * 32)
            if (*d >= 0)
                push16(&halo_w[buf * a.nhalo_max + (*d & 0xffff)], &s_mbar[buf], *d >> 16, v[0], v[1], v[2]);
    };

    // w of this thread's own rows: H times the window (0 times it with
    // `zero`).  Each row's four lanes hold its sum: row_done(slice of the
    // warp, sum) may change it and pushes it to the parts that need it.  Lane
    // 8 g + i takes every fourth block of row i: a quarter warp's window reads
    // are then eight rows' same neighbour, mostly consecutive and so free of
    // bank conflicts.
    auto reduce_row = [&](float acc[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 16);
            acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], 8);
        }
    };
    // `count` trips from the warp's `done`-th on
    auto stored_trips = [&](int done, int count, float acc[3]) {
        const int ns = STREAM ? min(count, max(0, a.smem_trips - done)) : count;
        const float4 *src = trips_w + done * kTripFloats4;
#pragma unroll 2
        for (int t = 0; t < ns; ++t, src += kTripFloats4) {
            const float4 h0 = src[lane], h1 = src[32 + lane];
            const float2 h2 = reinterpret_cast<const float2 *>(src + 64)[lane];
            const float h[9] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w, h2.x};
            block_mac(h, win[__float_as_int(h2.y)], acc);
        }
        if (STREAM && count > ns) {
            src = stream_w + (size_t)(done + ns - a.smem_trips) * kTripFloats4;
#pragma unroll 4
            for (int t = ns; t < count; ++t, src += kTripFloats4) {
                const float4 h0 = __ldcg(src + lane), h1 = __ldcg(src + 32 + lane);
                const float2 h2 = __ldcg(reinterpret_cast<const float2 *>(src + 64) + lane);
                const float h[9] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w, h2.x};
                block_mac(h, win[__float_as_int(h2.y)], acc);
            }
        }
    };
    auto product = [&](bool zero, auto row_done) {
        if (first_trips == 0) return;  // a warp without rows
        float acc[3] = {0.0f, 0.0f, 0.0f};
        int done = first_trips - nreg;
        if (!zero) {
#pragma unroll
            for (int k = 0; k < KR; ++k)
                if (k < nreg) block_mac(hreg[k], win[(creg[k / 2] >> (16 * (k & 1))) & 0xffffu], acc);
            if (done > 0) stored_trips(0, done, acc);
            reduce_row(acc);
        }
        row_done(0, acc);
        if (lane < 8) {
#pragma unroll
            for (int c = 0; c < 3; ++c) w[0][c] = acc[c];
            if (ORDERED && own[0]) {
#pragma unroll
                for (int c = 0; c < 3; ++c) own_w[3 * (row_id[0] - row0) + c] = acc[c];
            }
        }
        if (more_trips == 0) return;
#pragma unroll
        for (int o = 0; o < OS; ++o)
#pragma unroll
            for (int qq = o == 0 ? 1 : 0; qq < 4; ++qq) {
                const int count = (ntrips[o] >> (8 * qq)) & 0xff;
                if (count == 0) break;
                acc[0] = acc[1] = acc[2] = 0.0f;
                if (!zero) {
                    stored_trips(done, count, acc);
                    reduce_row(acc);
                }
                done += count;
                row_done(4 * o + qq, acc);
                if ((lane >> 3) == qq) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) w[o][c] = acc[c];
                    if (ORDERED && own[o]) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) own_w[3 * (row_id[o] - row0) + c] = acc[c];
                    }
                }
            }
    };
    auto publish = [&](unsigned k) {
#pragma unroll
        for (int o = 0; o < OS; ++o)
            if (own[o])
                a.pub[(size_t)(k & 1) * a.n + row_id[o]] = make_float4(w[o][0], w[o][1], w[o][2], 0.0f);
    };

    // Round k: the sums of v[] over the body's own rows, on which warp 0 alone
    // decides (decide(sums) fills s_verdict), and the halo rows' values: with
    // a cluster warp 0 acquires the phase that counts the pushed bytes and the
    // barrier hands them on; with the grid they go to halo_v.  CTA-uniform;
    // the verdict of a wait that gave up is a timeout.
    float halo_v[SCOPE == kGrid ? RS : 1][3];
    auto exchange = [&](unsigned k, const Sum v[3], auto term, auto decide) -> Verdict {
        const int buf = k & 1;
        if (ORDERED) {
            __syncthreads();  // own_r, own_u, own_w
#pragma unroll
            for (int q = 0; q < kTasks; ++q) {
                if (task_dst[q] < 0) break;
                Sum acc[3] = {0.0f, 0.0f, 0.0f};
                if (task_i[q] < task_end[q]) term(task_i[q], acc);
                if (SCOPE == kGrid)  // blocks of more than 170 rows
                    for (int i = task_i[q] + kPartThreads; i < task_end[q]; i += kPartThreads) term(i, acc);
                const Sum k3 = warp_sum3(acc, lane);
                if ((lane & 7) == 0 && lane < 24)
                    (&s_red[0][0][0])[task_dst[q] + kPartWarps * (lane == 0 ? 0 : lane == 16 ? 1 : 2)] = k3;
            }
        } else {
            // (fp64: a warp without rows spares the SM's fp64 pipe)
            const Sum k3 = kWide && first_trips == 0 ? (Sum)0.0f : warp_sum3(v, lane);
            if ((lane & 7) == 0 && lane < 24) s_red[0][lane == 0 ? 0 : lane == 16 ? 1 : 2][warp] = k3;
        }
        __syncthreads();
        Sum sum[3];
        const int g = min(lane >> 3, 2), i = lane & 7;
        bool ok = true;
        if (SCOPE == kCluster && tid == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&s_mbar[buf])),
                         "r"(16u * (uint32_t)((kWide ? 2 : 1) * (ORDERED ? a.blocks : ncta) + part.nhalo))
                         : "memory");
        if (warp < (ORDERED ? part.nblocks : 1)) {
            // a block's sum, by a warp of its own
            const int b = ORDERED ? warp : 0;
            group_sum3(s_red[b][g][i] + s_red[b][g][i + 8], sum);
            if (SCOPE == kCluster && lane < ncta)
                push_sums(&s_part[buf][ORDERED ? part.block_lo + b : rank], &s_mbar[buf], lane, sum);
        }
        if (warp == 0) {
            if (SCOPE == kOne && ORDERED && part.nblocks > 1) {
                Sum second[3];
                group_sum3(s_red[kBlocks > 1 ? 1 : 0][g][i] + s_red[kBlocks > 1 ? 1 : 0][g][i + 8], second);
#pragma unroll
                for (int c = 0; c < 3; ++c) sum[c] += second[c];
            }
            if (SCOPE == kCluster) {
                ok = __all_sync(0xffffffffu, wait_phase(&s_mbar[buf], (k >> 1) & 1u));
                if (ORDERED) {
                    Sum t[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int b = 0; b < kSums; b += 32)  // zero past the last block
                        if (b < a.blocks) {
                            const float4 q = *reinterpret_cast<const float4 *>(&s_part[buf][b + lane < kSums ? b + lane : 0]);
                            t[0] += q.x;
                            t[1] += q.y;
                            t[2] += q.z;
                        }
                    spread_sum3(warp_sum3(t, lane), sum);
                } else {
                    const Sum *t = reinterpret_cast<const Sum *>(s_part[buf]) + g;
                    group_sum3(t[4 * i] + t[4 * (i + 8)], sum);
                }
            }
            if (SCOPE == kGrid) {
                target += ncta;
                if (lane == 0) {
                    put_sums(static_cast<Sum *>(a.partials), buf * ncta + rank, sum);
                    // every earlier store of this CTA is released before the
                    // counter moves
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
                if (row_id[j] < 0 || (j < OS && own[j < OS ? j : 0])) continue;
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

    // u = M r of every local row into the window; with `update`, first
    // s = w + beta s, r -= alpha s (and p, x of own rows), else r = w
    auto show_u = [&](unsigned k, bool update, float alpha, float beta, bool first) {
#pragma unroll
        for (int j = 0; j < RS; ++j) {
            const int l = local0 + j * kPartThreads;
            if (l >= nlocal) continue;
            float v[3];
            if (j < OS && own[j < OS ? j : 0]) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = w[j < OS ? j : 0][c];
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
                if (j < OS) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {  // own rows'; a halo row's are not used
                        float &pc = p[j < OS ? j : 0][c], &xc = x[j < OS ? j : 0][c];
                        pc = first ? u[j < OS ? j : 0][c] : __fmaf_rn(beta, pc, u[j < OS ? j : 0][c]);
                        xc = __fmaf_rn(alpha, pc, xc);
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    s[j][c] = first ? v[c] : __fmaf_rn(beta, s[j][c], v[c]);
                    r[j][c] = __fmaf_rn(-alpha, s[j][c], r[j][c]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) r[j][c] = v[c];
            }
            float z[3];
            precond(j > 0 ? minv_s + 9 * (l - kPartThreads) : minv, r[j], z, a.use_precond);
            win[l] = make_float4(z[0], z[1], z[2], 0.0f);
            if (j < OS) {
#pragma unroll
                for (int c = 0; c < 3; ++c) u[j < OS ? j : 0][c] = z[c];
                if (ORDERED && own[j < OS ? j : 0]) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        own_r[3 * (row_id[j] - row0) + c] = r[j][c];
                        own_u[3 * (row_id[j] - row0) + c] = z[c];
                    }
                }
            }
        }
    };
    // partial sums of gamma, delta and (r, r) over the own rows
    auto dots = [&](Sum (&sum)[3]) {
        if (ORDERED) return;
        sum[0] = sum[1] = sum[2] = 0.0f;
#pragma unroll
        for (int o = 0; o < OS; ++o) add_rows(r[o], u[o], w[o], own[o], lane, sum);
    };

    auto term = [&](int i, Sum acc[3]) {  // ORDERED: the same of component i
        const float rc = own_r[i], uc = own_u[i];
        add_product(rc, uc, acc[0]);
        add_product(own_w[i], uc, acc[1]);
        add_product(rc, rc, acc[2]);
    };

    // ---- r0 = g - H x0 (x0 = 0 for an inner solve), exchanged in round 0
    const float bscale = inner ? a.ir_scale[0] : 1.0f;
    Sum sum[3] = {0.0f, 0.0f, 0.0f};
    product(inner, [&](int q, float acc[3]) {
        const int i = (warp + kPartWarps * q) * kPartSliceRows + (lane & 7);
        if (i < part.nown) {
            const int row = a.v.rows[part.row_off + i];
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] = __ldg(a.b + (size_t)3 * row + c) * bscale - acc[c];
        }
        if (SCOPE == kCluster) push_row(0, q, acc);
    });
    if (SCOPE == kGrid) publish(0);
#pragma unroll
    for (int o = 0; o < OS; ++o)
        if (own[o]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float g = __ldg(a.b + (size_t)3 * row_id[o] + c) * bscale;
                add_product(g, g, sum[0]);
                if (ORDERED) own_r[3 * (row_id[o] - row0) + c] = g;
            }
        }
    // the recurrence's scalars, kept by thread 0 (||g||^2 and (r, r) in s_norm)
    Sum thr2 = 0.0f, gamma = 0.0f, alpha = 0.0f;  // fp64: alpha holds the last denominator
    int it = 0;
    unsigned round = 0;
    auto rhs_term = [&](int i, Sum acc[3]) { add_product(own_r[i], own_r[i], acc[0]); };
    Verdict d = exchange(round, sum, rhs_term, [&](const Sum t[3]) {
        s_norm[0] = t[0];
        s_norm[1] = 0.0f;
        thr2 = (Sum)a.tol * a.tol * t[0];
        return Verdict{0.0f, 0.0f, 0, MFEM_OK};
    });
    if (!d.done) {
        show_u(round, false, 0.0f, 0.0f, true);
        __syncthreads();
        // ---- w0 = H u0
        auto push_w = [&](int q, float acc[3]) {
            if (SCOPE == kCluster) push_row(round + 1, q, acc);
        };
        product(false, push_w);
        if (SCOPE == kGrid) publish(round + 1);
        dots(sum);
        d = exchange(++round, sum, term, [&](const Sum t[3]) {
            gamma = t[0];
            const Sum rr = t[2];
            s_norm[1] = rr;
            const Sum first = t[1] > 0.0f ? gamma / t[1] : 0.0f;
            alpha = kWide ? t[1] : first;
            int status = MFEM_OK;
            if (!isfinite(gamma) || !isfinite(t[1]) || !isfinite(rr) || !isfinite(s_norm[0])) status = MFEM_NONFINITE;
            else if (!(t[1] > 0.0f) && rr > 0.0f) status = MFEM_STAGNATION;
            int done = status != MFEM_OK || rr <= thr2;
            if (!done && a.maxiter <= 0) {
                done = 1;
                status = MFEM_MAXITER;
            }
            return Verdict{(float)first, 0.0f, done, status};
        });
        while (!d.done) {
            show_u(round, true, d.alpha, d.beta, it == 0);
            __syncthreads();
            product(false, push_w);
            if (SCOPE == kGrid) publish(round + 1);
            dots(sum);
            ++it;
            d = exchange(++round, sum, term, [&](const Sum t[3]) {
                const Sum rr = t[2];
                s_norm[1] = rr;
                if (!isfinite(t[0]) || !isfinite(t[1]) || !isfinite(rr)) return Verdict{0.0f, 0.0f, 1, MFEM_NONFINITE};
                if (rr <= thr2) return Verdict{0.0f, 0.0f, 1, MFEM_OK};
                const Sum beta = t[0] / gamma;
                // the ratio in flight with beta, or in the windowed kernel's order, or
                // (a slow fp64 division less) from the last denominator gamma / alpha
                const Sum denom = kWide     ? t[1] - beta * beta * alpha
                                  : ORDERED ? t[1] - beta * t[0] / alpha
                                            : t[1] - beta * (t[0] / alpha);
                if (!(denom > 0.0f)) return Verdict{0.0f, 0.0f, 1, MFEM_STAGNATION};
                const Sum next = t[0] / denom;
                alpha = kWide ? denom : next;
                gamma = t[0];
                return Verdict{(float)next, (float)beta, it >= a.maxiter, it >= a.maxiter ? MFEM_MAXITER : MFEM_OK};
            });
        }
    }
    if (d.status == MFEM_TIMEOUT && tid == 0) atomicExch(a.error, 1);
    const float es = inner ? a.ir_scale[1] : 1.0f;
#pragma unroll
    for (int o = 0; o < OS; ++o)
        if (own[o]) {
            const int row = a.v.rows[part.row_off + local0 + o * kPartThreads];
#pragma unroll
            for (int c = 0; c < 3; ++c) a.x[(size_t)3 * row + c] = x[o][c] * es;
        }
    if (rank == 0 && tid == 0) {
        if (inner) {
            // a solve that stopped at the cap or stagnated still hands over
            // its iterate; a 16-bit H that broke it restarts on the fp32 H
            a.ir_state[2] += it;
            a.ir_state[3] = 1;
            if (LOWP && d.status == MFEM_NONFINITE && a.values_w != nullptr && a.ir_state[6] == 0) {
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
            a.stats[(size_t)a.slot * a.bodies + task.z] = SolveStats{it, d.status, rel, 0.0f};
        }
    }
    if (SCOPE == kCluster) cluster_sync();  // no CTA leaves while another may still push to it
}

typedef void (*ResKernel)(ResArgs);

template <bool STREAM>
ResKernel pick_form(const ResidentLayout &L, bool lowp) {
    constexpr int KR = kPartRegTrips;
    if (L.grid) {
        if (L.own_slots == 2)
            return L.row_slots <= 3 ? pcg_resident_kernel<kGrid, 2, 3, 0, STREAM, false>
                   : lowp           ? pcg_resident_kernel<kGrid, 2, 4, 0, STREAM, false>
                                    : pcg_resident_kernel<kGrid, 2, 4, 0, STREAM, false, false>;
        return L.row_slots <= 1   ? pcg_resident_kernel<kGrid, 1, 1, KR, STREAM, false>
               : L.row_slots <= 2 ? pcg_resident_kernel<kGrid, 1, 2, KR, STREAM, false>
                                  : pcg_resident_kernel<kGrid, 1, 4, 0, STREAM, false>;
    }
    if (L.cluster <= 1) return pcg_resident_kernel<kOne, 1, 1, KR, STREAM, false>;
    if (L.own_slots == 2) return pcg_resident_kernel<kCluster, 2, 4, 0, STREAM, false>;
    return L.row_slots <= 1 ? pcg_resident_kernel<kCluster, 1, 1, KR, STREAM, false>
                            : pcg_resident_kernel<kCluster, 1, 2, KR, STREAM, false>;
}

ResKernel pick_ordered(const ResidentLayout &L) {
    constexpr int KR = kPartRegTrips;
    if (L.grid)
        return L.row_slots <= 1 ? pcg_resident_kernel<kGrid, 1, 1, KR, false, true>
                                : pcg_resident_kernel<kGrid, 1, 2, KR, false, true>;
    if (L.cluster <= 1) return pcg_resident_kernel<kOne, 1, 1, KR, false, true>;
    return L.row_slots <= 1 ? pcg_resident_kernel<kCluster, 1, 1, KR, false, true>
                            : pcg_resident_kernel<kCluster, 1, 2, KR, false, true>;
}

// With fp64 sums, for the mixed refinement's inner solves: slots and register
// trips as pick_form's, one instance for meshes with and without streamed trips.
ResKernel pick_wide(const ResidentLayout &L) {
    constexpr int KR = kPartRegTrips;
    if (L.grid) {
        if (L.own_slots == 2) return pcg_resident_kernel<kGrid, 2, 4, 0, true, false, true, double>;
        return L.row_slots <= 1   ? pcg_resident_kernel<kGrid, 1, 1, KR, true, false, true, double>
               : L.row_slots <= 2 ? pcg_resident_kernel<kGrid, 1, 2, KR, true, false, true, double>
                                  : pcg_resident_kernel<kGrid, 1, 4, 0, true, false, true, double>;
    }
    if (L.cluster <= 1) return pcg_resident_kernel<kOne, 1, 1, KR, true, false, true, double>;
    if (L.own_slots == 2) return pcg_resident_kernel<kCluster, 2, 4, 0, true, false, true, double>;
    return L.row_slots <= 1 ? pcg_resident_kernel<kCluster, 1, 1, KR, true, false, true, double>
                            : pcg_resident_kernel<kCluster, 1, 2, KR, true, false, true, double>;
}

ResKernel pick(const ResidentLayout &L, bool lowp, bool wide = false) {
    if (L.blocks > 0) return pick_ordered(L);
    if (wide) return pick_wide(L);
    return L.stream_trips > 0 ? pick_form<true>(L, lowp) : pick_form<false>(L, lowp);
}

// Launch configuration of n_tasks bodies; attr holds its attribute.
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

cudaError_t resident_layout(int device, const ResidentHost &h, int cluster, bool grid, ResidentLayout &L, bool &fits) {
    fits = false;
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    L = ResidentLayout{};
    L.cluster = cluster;
    L.grid = grid;
    L.nown_max = h.nown_max;
    L.nhalo_max = h.nhalo_max;
    L.own_slots = std::max(1, (h.nown_max + kPartThreads - 1) / kPartThreads);
    L.row_slots = std::max(1, (h.nlocal_max + kPartThreads - 1) / kPartThreads);
    if (L.own_slots > 2 || L.row_slots > 4 || h.slice_trips_max > 255) return cudaSuccess;
    if (!grid && cluster <= 1 && (L.own_slots > 1 || L.row_slots > 1)) return cudaSuccess;
    L.blocks = h.blocks;
    if (L.blocks > 0) {
        // ordered sums: one own row and at most two rows a thread, nothing streamed
        if (L.own_slots > 1 || L.row_slots > 2 || !ordered_sums_fit(h, cluster, grid)) return cudaSuccess;
    } else if (!grid && L.row_slots > 2) {
        L.own_slots = 2;  // the cluster form with more than two rows a thread
    }
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, pick(L, false));
    if (e != cudaSuccess) return e;
    const bool regs = !(L.own_slots == 2 || L.row_slots > 2);  // pick()'s kernels with register trips
    const int trips = regs ? h.trips_max_reg : h.trips_max;
    size_t fixed = fa.sharedSizeBytes;
    if (L.blocks == 0) {  // the same layout serves the fp64 sums
        e = cudaFuncGetAttributes(&fa, pick_wide(L));
        if (e != cudaSuccess) return e;
        fixed = std::max(fixed, fa.sharedSizeBytes);
    }
    const size_t most = (size_t)optin - fixed;
    const size_t base = sizeof(float4) * ((size_t)h.nown_max + (!grid && cluster > 1 ? 3 : 1) * (size_t)h.nhalo_max) +
                        (L.row_slots > 1 ? 9 * sizeof(float) * (size_t)std::max(0, h.nown_max + h.nhalo_max - kPartThreads) : 0) +
                        (!grid && cluster > 1 ? sizeof(int) * (size_t)h.push_max : 0) +
                        (L.blocks > 0 ? 9 * sizeof(float) * (size_t)h.nown_max : 0) + 16;
    const size_t per_trip = sizeof(float4) * kTripFloats4 * kPartWarps;
    if (base > most) return cudaSuccess;
    L.smem_trips = (int)std::min<size_t>(trips, (most - base) / per_trip);
    L.stream_trips = trips - L.smem_trips;
    L.smem = (base + per_trip * L.smem_trips + 15) & ~(size_t)15;
    if (L.smem > most || (L.blocks > 0 && L.stream_trips > 0)) return cudaSuccess;
    L.push_max = !grid && cluster > 1 ? h.push_max : 0;
    const ResKernel k = pick(L, false);
    // the limit is the kernel's, not the plan's: every plan sets the same one
    for (const ResKernel f : {k, pick(L, true), pick(L, true, true)}) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e == cudaSuccess && !grid && cluster > 8)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
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

cudaError_t launch_resident(const BsrViews &bv, const VertexViews &vv, const ResidentLayout &L, int n_tasks,
                            int n_bodies, const PcgWork &w, SolveStats *stats, int slot, float tol, int maxiter,
                            int use_precond, const IrWork *ir, cudaStream_t s) {
    ResArgs a = {};
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
    a.use_precond = use_precond;
    a.nown_max = L.nown_max;
    a.nhalo_max = L.nhalo_max;
    a.smem_trips = L.smem_trips;
    a.stream_trips = L.stream_trips;
    a.push_max = L.push_max;
    a.blocks = L.blocks;
    a.block_warps = L.blocks > 0 ? ordered_block_warps(bv.n, L.blocks) : 0;
    a.pub = reinterpret_cast<float4 *>(w.pub);
    const bool wide = ir && ir->wide && L.blocks == 0;
    a.partials = wide ? static_cast<void *>(ir->partials) : w.partials;
    a.counter = w.res_counter;
    a.ir_state = ir ? ir->state : nullptr;
    a.ir_scale = ir ? ir->scale : nullptr;
    if (ir) {
        a.values_w = ir->mode == kIrFp32 ? nullptr : ir->hq_words;
        a.row_scale = ir->row_scale;
        a.lowp_kind = ir->mode == kIrBf16 ? 1 : 2;
    }
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = launch_config(L, n_tasks, attr, s);
    cudaError_t e = cudaLaunchKernelEx(&cfg, pick(L, a.values_w != nullptr, wide), a);
    count_launches(1);
    return e;
}

}  // namespace mfem
