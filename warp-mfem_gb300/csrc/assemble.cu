// Numeric assembly of the global system, without atomics.
//
// The reference builds G^T and H_lambda G as padded BSR matrices and forms
// H with bsr_mm, g with a transposed bsr_mv, then adds (M+Q)/dt^2 with
// bsr_axpy (src/mfem/refinement/solver.py:682-743).  Here the element kernel
// has already formed each tet's 10 upper 3x3 blocks of G^T H_l G and its rhs
// (H_l G)^T g_l; this kernel gathers them into the BSR slots.
//
// The symbolic phase sorted every (tet, k, l) contribution to a diagonal or
// upper slot by destination and packed whole slots into warp-sized chunks.
// A warp takes one chunk at a time, each lane one contribution (lanes stride
// over the single slot of a chunk longer than 32), and a segmented shuffle
// reduction over the lanes of a slot yields its sum in its first lane, in a
// fixed order, so the result is deterministic.  That lane writes the slot and
// its mirror: the lower slot would add the transposes of the same blocks in
// the same order, so its value is the transpose bit for bit.  A diagonal
// slot's first lane also adds the mass/attachment term, inverts the block for
// the block-Jacobi preconditioner, and writes the vertex's rhs
// g = sum fe - g_x and the warm start dx = x~ - x.  With contact, the lists
// also carry the surface tris' barrier blocks, and the diagonal lane adds the
// vertex's barrier and friction block and takes the contact gradients off the
// rhs.
//
// What bounds it: neither bytes nor arithmetic but instructions and the
// latency of chunk -> code -> record -> slot.  So only the upper triangle is
// gathered (10 contributions a tet instead of 16), a contribution is one
// 32-byte and one 4- or 16-byte load (nine and three scalar loads took as
// many L1 passes), the shuffles stop at the chunk's longest slot, a warp reads
// the codes of its next chunk and the descriptor of the one after ahead of
// their use, and the vertex's work, some 250 instructions for one lane, waits
// in shared memory until a lane each can do it.  331,200 tets, 60,528
// vertices: 164 -> 70 us (94 us with the vertex's work in the summing lane);
// 98,304 tets: 49 -> 24 us.
#include <algorithm>

#include "internal.h"

namespace mfem {
namespace {

constexpr int kAssembleThreads = 128;
// resident blocks an SM, and the most blocks of a launch; 4, 5, 6, 7 and 8
// blocks an SM take 86, 78, 71, 70 and 71 us at 331,200 tets
constexpr int kAssembleOccupancy = 7;
constexpr int kAssembleBlocks = 152 * kAssembleOccupancy;
constexpr int kDiagStride = 15;

// One shuffle step of N sums over segments: adds the lane off above, where it
// is in the segment that ends at lane `last`.
template <int N>
__device__ __forceinline__ void seg_step(float (&v)[N], int off, int lane, int last) {
    const bool in = lane + off <= last;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float o = __shfl_down_sync(0xffffffffu, v[i], off);
        if (in) v[i] += o;
    }
}

// 32 bytes of a 32-byte aligned address in one load.
__device__ __forceinline__ void load8(const float *p, float v[8]) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// Contribution `code`: block b, to be transposed if tr, and for a tet's
// diagonal block the vertex's rhs f.
__device__ __forceinline__ void contribution(int code, const float *__restrict__ Ke, const ContactViews &cv, float b[9],
                                             float f[3], bool &tr) {
    if (code >= cv.tri_code_base) {
        // tri contact block w_i w_j k max(b'', 0) n n^T (contact.py:733-741)
        const int tc = code - cv.tri_code_base;
        const int tri = tc / 9;
        const int i = (tc - 9 * tri) / 3, j = tc - 9 * tri - 3 * i;
        const float *td = cv.tri + (size_t)tri * kTriData;
        const float hw = (td[7 + i] * td[7 + j]) * td[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int bb = 0; bb < 3; ++bb) b[a * 3 + bb] = hw * (td[4 + a] * td[4 + bb]);
    } else if (code >= 0) {
        const int k = (code >> 2) & 3;
        const int l = code & 3;
        tr = k > l;
        const float *rec = Ke + (size_t)(code >> 4) * kKeRecord;
        load8(rec + ke_block(min(k, l), max(k, l)) * kKeHead, b);
        if (k == l) {
            const float4 d = *reinterpret_cast<const float4 *>(rec + kKeDiagTail + 4 * k);
            b[8] = d.x;
            f[0] = d.y;
            f[1] = d.z;
            f[2] = d.w;
        } else {
            b[8] = rec[ke_off_tail(min(k, l), max(k, l))];
        }
    }
}

// What a lane holds of a chunk: its contribution's code, and in a slot's
// first lane the slot and its mate.
struct LaneChunk {
    int4 chunk;
    int code;
    int2 pair;
};

__device__ __forceinline__ int4 load_chunk(const AssemblyLists &al, int i) {
    return i < al.n_chunks ? __ldg(al.chunk + i) : make_int4(0, 0, 0, 0);
}

__device__ __forceinline__ void load_lane(const AssemblyLists &al, int lane, const int4 &chunk, LaneChunk &lc) {
    lc.chunk = chunk;
    lc.code = -1;
    lc.pair = make_int2(-1, -1);
    if (chunk.x + lane < chunk.y) {
        lc.code = __ldg(al.code + chunk.x + lane);
        if (((unsigned)chunk.w >> lane) & 1u)
            lc.pair = __ldg(al.pair + chunk.z + __popc((unsigned)chunk.w & ((1u << lane) - 1u)));
    }
}

__device__ __forceinline__ void add_block(float v[9], const float b[9], bool tr) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[a * 3 + c] += tr ? b[c * 3 + a] : b[a * 3 + c];
}

// The vertex's terms of the diagonal block v at `out`: H's block, and the
// row's Minv, rhs and dx.
__device__ __forceinline__ void finish_diagonal(float v[9], const float f[3], int row, float *__restrict__ out,
                                                const float *__restrict__ x, float dt, float alpha_mass,
                                                float singular_threshold, int use_precond, const VertexViews &vv,
                                                const ContactViews &cv) {
    // H += (M + Q) / dt^2 on the diagonal (solver.py:737-743)
    const float hd = alpha_mass * vv.hess_diag[row];
    v[0] += hd;
    v[4] += hd;
    v[8] += hd;
    // + the vertex's barrier and friction blocks (solver.py:745-779)
    float gc[3] = {0.0f, 0.0f, 0.0f};
    if (cv.on) {
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] += cv.vblock[9 * row + i];
#pragma unroll
        for (int a = 0; a < 3; ++a) gc[a] = cv.vgrad[3 * row + a];
        // tri barrier gradients scattered with the barycentric weights
        for (int k = cv.vt_ptr[row]; k < cv.vt_ptr[row + 1]; ++k) {
            const int code3 = cv.vt_code[k];
            const int tri = code3 / 3, corner = code3 - 3 * tri;
            const float *td = cv.tri + (size_t)tri * kTriData;
            const float gw = td[7 + corner] * td[2];
#pragma unroll
            for (int a = 0; a < 3; ++a) gc[a] += gw * td[4 + a];
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) cv.gtot[3 * row + a] = gc[a];
    }
    // block-Jacobi inverse, identity for |det| < threshold (kernels.py:32-53)
    const float c00 = v[4] * v[8] - v[5] * v[7];
    const float c01 = v[5] * v[6] - v[3] * v[8];
    const float c02 = v[3] * v[7] - v[4] * v[6];
    const float det = v[0] * c00 + v[1] * c01 + v[2] * c02;
    float *M = vv.Minv + (size_t)row * 9;
    if (!use_precond || !(fabsf(det) >= singular_threshold)) {
#pragma unroll
        for (int i = 0; i < 9; ++i) M[i] = (i % 4 == 0) ? 1.0f : 0.0f;
    } else {
        const float id = 1.0f / det;
        M[0] = c00 * id;
        M[1] = (v[2] * v[7] - v[1] * v[8]) * id;
        M[2] = (v[1] * v[5] - v[2] * v[4]) * id;
        M[3] = c01 * id;
        M[4] = (v[0] * v[8] - v[2] * v[6]) * id;
        M[5] = (v[2] * v[3] - v[0] * v[5]) * id;
        M[6] = c02 * id;
        M[7] = (v[1] * v[6] - v[0] * v[7]) * id;
        M[8] = (v[0] * v[4] - v[1] * v[3]) * id;
    }
    // g = sum fe - g_x, g_x = m (x - x~)/dt^2 + (k x - k p)/dt^2
    // (kernels.py:172-185; boundary_condition.py:73-80; solver.py:726-733, 946-947)
    const float dt2 = dt * dt;
    const float m = vv.mass[row];
    const float kp = vv.pin_k[row];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float xa = x[3 * row + a];
        const float xt = vv.x_tilde[3 * row + a];
        const float pt = vv.pin_target[3 * row + a];
        const float gx = m * (xa - xt) / dt2 + (kp * xa + (-(kp * pt))) / dt2;
        // - barrier and friction gradients (solver.py:734-735)
        vv.rhs[3 * row + a] = (f[a] - gx) - gc[a];
        vv.dx[3 * row + a] = xt - xa;
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = v[i];
}

__global__ void __launch_bounds__(kAssembleThreads, kAssembleOccupancy)
    assemble_kernel(const float *__restrict__ x, float dt, float alpha_mass, float singular_threshold,
                    int use_precond, TetViews tv, VertexViews vv, BsrViews bv, ContactViews cv) {
    // the warp's summed diagonal blocks and rhs, until a lane each can finish
    // them: [entry][9 block, 3 rhs, row, slot], at an odd stride
    __shared__ float s_diag[kAssembleThreads / 32][32][kDiagStride];
    const AssemblyLists &al = bv.asm_lists;
    const int lane = threadIdx.x & 31;
    float(*const queue)[kDiagStride] = s_diag[threadIdx.x >> 5];
    int queued = 0;  // uniform in the warp
    auto flush = [&] {
        __syncwarp();
        if (lane < queued) {
            const float *q = queue[lane];
            float v[9], f[3];
#pragma unroll
            for (int k = 0; k < 9; ++k) v[k] = q[k];
#pragma unroll
            for (int k = 0; k < 3; ++k) f[k] = q[9 + k];
            finish_diagonal(v, f, __float_as_int(q[12]), bv.values + (size_t)__float_as_int(q[13]) * 9, x, dt, alpha_mass,
                            singular_threshold, use_precond, vv, cv);
        }
        queued = 0;
        __syncwarp();
    };
    const int warps = (gridDim.x * blockDim.x) >> 5;
    int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    LaneChunk nxt;
    load_lane(al, lane, load_chunk(al, i), nxt);
    int4 far = load_chunk(al, i + warps);
    for (; i < al.n_chunks; i += warps) {  // uniform in the warp
        const LaneChunk lc = nxt;
        float v[9], f[3], b[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) b[k] = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) f[k] = 0.0f;
        bool tr = false;
        contribution(lc.code, tv.Ke, cv, b, f, tr);
        load_lane(al, lane, far, nxt);
        far = load_chunk(al, i + 2 * warps);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[a * 3 + c] = tr ? b[c * 3 + a] : b[a * 3 + c];
        // the rest of a slot of more than 32 contributions
        for (int c = lc.chunk.x + 32 + lane; c < lc.chunk.y; c += 32) {
            float fb[3] = {0.0f, 0.0f, 0.0f};
            tr = false;
            contribution(__ldg(al.code + c), tv.Ke, cv, b, fb, tr);
            add_block(v, b, tr);
#pragma unroll
            for (int k = 0; k < 3; ++k) f[k] += fb[k];
        }
        const unsigned heads = (unsigned)lc.chunk.w;
        const int used = min(32, lc.chunk.y - lc.chunk.x);
        const unsigned above = heads & (0xfffffffeu << lane);
        const int last = above ? __ffs(above) - 2 : used - 1;
        const int reach = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(last - lane, 0));
        const bool head = lc.pair.x >= 0;
        const unsigned diags = __ballot_sync(0xffffffffu, head && lc.pair.y < 0);
        for (int off = 1; off <= reach; off <<= 1) {
            seg_step<9>(v, off, lane, last);
            if (diags) seg_step<3>(f, off, lane, last);
        }
        if (head && lc.pair.y >= 0) {
            float *out = bv.values + (size_t)lc.pair.x * 9;
            float *mir = bv.values + (size_t)lc.pair.y * 9;
#pragma unroll
            for (int k = 0; k < 9; ++k) out[k] = v[k];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int c = 0; c < 3; ++c) mir[c * 3 + a] = v[a * 3 + c];
        }
        const int n_diag = __popc(diags);
        if (n_diag) {
            if (queued + n_diag > 32) flush();
            if (head && lc.pair.y < 0) {
                float *q = queue[queued + __popc(diags & ((1u << lane) - 1u))];
#pragma unroll
                for (int k = 0; k < 9; ++k) q[k] = v[k];
#pragma unroll
                for (int k = 0; k < 3; ++k) q[9 + k] = f[k];
                q[12] = __int_as_float(~lc.pair.y);
                q[13] = __int_as_float(lc.pair.x);
            }
            queued += n_diag;
        }
    }
    if (queued) flush();
}

__global__ void true_residual_kernel(BsrViews bv, const float *__restrict__ rhs, const float *__restrict__ dx,
                                     double *out) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0, bb = 0.0;
    if (row < bv.n) {
        double acc[3] = {0.0, 0.0, 0.0};
        for (int k = bv.row_ptr[row]; k < bv.row_ptr[row + 1]; ++k) {
            const int col = bv.col_idx[k];
            const float *h = bv.values + (size_t)k * 9;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) acc[a] += (double)h[a * 3 + b] * (double)dx[3 * col + b];
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double g = rhs[3 * row + a];
            const double r = g - acc[a];
            rr += r * r;
            bb += g * g;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        rr += __shfl_down_sync(0xffffffffu, rr, off);
        bb += __shfl_down_sync(0xffffffffu, bb, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out + 0, rr);
        atomicAdd(out + 1, bb);
    }
}

}  // namespace

cudaError_t launch_assemble(const float *x, float dt, float singular_threshold, int use_precond,
                            const TetViews &tv, const VertexViews &vv, const BsrViews &bv, const ContactViews &cv,
                            cudaStream_t s) {
    if (bv.asm_lists.n_chunks == 0) return cudaSuccess;
    const int warps_per_block = kAssembleThreads / 32;
    const int blocks = std::min((bv.asm_lists.n_chunks + warps_per_block - 1) / warps_per_block, kAssembleBlocks);
    // alpha = 1/(dt*dt) computed in double and rounded once, as the float32
    // bsr_axpy scale of the reference (solver.py:737-743)
    const float alpha_mass = (float)(1.0 / ((double)dt * (double)dt));
    assemble_kernel<<<blocks, kAssembleThreads, 0, s>>>(x, dt, alpha_mass, singular_threshold, use_precond, tv, vv,
                                                        bv, cv);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_true_residual(const BsrViews &bv, const VertexViews &vv, double *out, cudaStream_t s) {
    cudaError_t err = cudaMemsetAsync(out, 0, 2 * sizeof(double), s);
    if (err != cudaSuccess) return err;
    if (bv.n == 0) return cudaSuccess;
    true_residual_kernel<<<(bv.n + 255) / 256, 256, 0, s>>>(bv, vv.rhs, vv.dx, out);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace mfem
