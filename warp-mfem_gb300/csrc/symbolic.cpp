// Host-side symbolic analysis of the global system (run once per mesh).
//
// The reference rebuilds padded BSR topologies every Newton iteration with
// bsr_set_from_triplets and bsr_mm (src/mfem/refinement/solver.py:685-724),
// sized by a row capacity of 1 + 3 * max incident tets (solver.py:203).  The
// topology only changes with the mesh, so here it is computed once, exactly:
//
//  * the vertex-adjacency sparsity of H, diagonal included, ascending columns;
//  * the element -> slot map: the slot of block (tets[e][k], tets[e][l]);
//  * the same map inverted and sorted by slot (then by tet) for the diagonal
//    and upper slots, which the numeric assembly reduces with warp shuffles
//    and mirrors; whole slots are packed into warp-sized chunks so no slot is
//    split between warps.
#include <algorithm>
#include <cstring>

#include "host_parallel.h"
#include "internal.h"

namespace mfem {

constexpr int kThreadRows = 1024;  // 0.1 to 0.5 us of work a row in each pass

static bool check_tets(int n, int T, const int32_t *tets, std::string &err) {
    if (n < 0 || T < 0) {
        err = "negative particle or tet count";
        return false;
    }
    if (T > 0 && tets == nullptr) {
        err = "tet_indices is NULL";
        return false;
    }
    if ((int64_t)T * 16 > (int64_t)INT32_MAX) {
        err = "too many tets for 32-bit contribution codes";
        return false;
    }
    for (int64_t i = 0; i < (int64_t)T * 4; ++i) {
        if (tets[i] < 0 || tets[i] >= n) {
            err = "tet_indices[" + std::to_string(i / 4) + "] references vertex " + std::to_string(tets[i]) +
                  " outside [0, " + std::to_string(n) + ")";
            return false;
        }
    }
    for (int e = 0; e < T; ++e) {
        const int32_t *t = tets + 4 * (int64_t)e;
        for (int a = 0; a < 4; ++a)
            for (int b = a + 1; b < 4; ++b)
                if (t[a] == t[b]) {
                    err = "tet " + std::to_string(e) + " repeats vertex " + std::to_string(t[a]);
                    return false;
                }
    }
    return true;
}

bool vertex_tets(int n, int T, const int32_t *tets, VertexTets &vt, std::string &err) {
    if (!check_tets(n, T, tets, err)) return false;
    vt.ptr.assign((size_t)n + 1, 0);
    for (int64_t i = 0; i < (int64_t)T * 4; ++i) vt.ptr[tets[i] + 1]++;
    for (int v = 0; v < n; ++v) vt.ptr[v + 1] += vt.ptr[v];
    vt.code.resize((size_t)T * 4);
    std::vector<int64_t> fill(vt.ptr.begin(), vt.ptr.end() - 1);
    for (int64_t i = 0; i < (int64_t)T * 4; ++i) vt.code[fill[tets[i]]++] = (int32_t)i;
    return true;
}

bool build_sparsity(int n, const int32_t *tets, const VertexTets &vt, std::vector<int32_t> &row_ptr,
                    std::vector<int32_t> &col_idx, std::string &err) {
    const auto &vptr = vt.ptr;
    const auto &vcode = vt.code;
    // per row: the diagonal and the vertices of the row's tets, made unique
    // with a stamp array and sorted (a few dozen columns a row)
    row_ptr.assign((size_t)n + 1, 0);
    const int threads = thread_count(n, kThreadRows);
    std::vector<std::vector<int32_t>> cols(threads);
    parallel_rows(n, threads, [&](int block, int first, int last) {
        std::vector<int32_t> stamp((size_t)n, -1), row;
        std::vector<int32_t> &out = cols[block];
        out.reserve((size_t)((vptr[last] - vptr[first]) + (last - first)));
        for (int v = first; v < last; ++v) {
            row.clear();
            stamp[v] = v;
            row.push_back(v);
            for (int64_t i = vptr[v]; i < vptr[v + 1]; ++i) {
                const int32_t *t = tets + 4 * (int64_t)(vcode[i] >> 2);
                for (int l = 0; l < 4; ++l)
                    if (stamp[t[l]] != v) {
                        stamp[t[l]] = v;
                        row.push_back(t[l]);
                    }
            }
            std::sort(row.begin(), row.end());
            out.insert(out.end(), row.begin(), row.end());
            row_ptr[v + 1] = (int32_t)row.size();
        }
    });
    size_t total = 0;
    for (const auto &c : cols) total += c.size();
    if (total > (size_t)INT32_MAX) {
        err = "sparsity exceeds 2^31 blocks";
        return false;
    }
    for (int v = 0; v < n; ++v) row_ptr[v + 1] += row_ptr[v];
    col_idx.resize(total);
    parallel_rows(n, threads, [&](int block, int first, int) {
        std::copy(cols[block].begin(), cols[block].end(), col_idx.begin() + row_ptr[first]);
    });
    return true;
}

bool build_slot_map(int n, const int32_t *tets, const VertexTets &vt, const int32_t *row_ptr, const int32_t *col_idx,
                    int32_t *slots, std::string &err) {
    const auto &vptr = vt.ptr;
    const auto &vcode = vt.code;
    // per row: each column's slot through a stamped position array, then
    // the slots of the row's tet corners
    const int threads = thread_count(n, kThreadRows);
    std::vector<std::string> errs(threads);
    parallel_rows(n, threads, [&](int block, int first, int last) {
        std::vector<int32_t> stamp((size_t)n, -1), pos((size_t)n, 0);
        for (int v = first; v < last; ++v) {
            for (int32_t j = row_ptr[v]; j < row_ptr[v + 1]; ++j) {
                const int32_t c = col_idx[j];
                if (c < 0 || c >= n) {
                    errs[block] = "column index out of range in row " + std::to_string(v);
                    return;
                }
                stamp[c] = v;
                pos[c] = j;
            }
            for (int64_t i = vptr[v]; i < vptr[v + 1]; ++i) {
                const int32_t e = vcode[i] >> 2, k = vcode[i] & 3;
                const int32_t *t = tets + 4 * (int64_t)e;
                for (int l = 0; l < 4; ++l) {
                    if (stamp[t[l]] != v) {
                        errs[block] = "sparsity lacks block (" + std::to_string(v) + ", " + std::to_string(t[l]) + ")";
                        return;
                    }
                    slots[(int64_t)e * 16 + k * 4 + l] = pos[t[l]];
                }
            }
        }
    });
    for (const std::string &e : errs)  // the first row's
        if (!e.empty()) {
            err = e;
            return false;
        }
    return true;
}

bool build_tri_slots(int n, int n_tris, const int32_t *tris, const int32_t *row_ptr, const int32_t *col_idx,
                     int32_t *tri_slots, std::vector<int32_t> &vt_ptr, std::vector<int32_t> &vt_code,
                     std::string &err) {
    for (int t = 0; t < n_tris; ++t) {
        const int32_t *v = tris + 3 * (int64_t)t;
        for (int k = 0; k < 3; ++k) {
            if (v[k] < 0 || v[k] >= n) {
                err = "tri " + std::to_string(t) + " has a vertex index out of range";
                return false;
            }
        }
        if (v[0] == v[1] || v[1] == v[2] || v[0] == v[2]) {
            err = "tri " + std::to_string(t) + " repeats a vertex";
            return false;
        }
        for (int i = 0; i < 3; ++i) {
            const int32_t *b = col_idx + row_ptr[v[i]];
            const int32_t *e = col_idx + row_ptr[v[i] + 1];
            for (int j = 0; j < 3; ++j) {
                const int32_t *p = std::lower_bound(b, e, v[j]);
                if (p == e || *p != v[j]) {
                    err = "tri " + std::to_string(t) + " joins vertices that share no tet";
                    return false;
                }
                tri_slots[(int64_t)t * 9 + i * 3 + j] = (int32_t)(p - col_idx);
            }
        }
    }
    // incident tri corners of each vertex, in tri order
    vt_ptr.assign(n + 1, 0);
    for (int64_t i = 0; i < (int64_t)n_tris * 3; ++i) vt_ptr[tris[i] + 1]++;
    for (int v = 0; v < n; ++v) vt_ptr[v + 1] += vt_ptr[v];
    vt_code.assign((size_t)n_tris * 3, 0);
    std::vector<int32_t> fill(vt_ptr.begin(), vt_ptr.end() - 1);
    for (int64_t i = 0; i < (int64_t)n_tris * 3; ++i) vt_code[fill[tris[i]]++] = (int32_t)i;
    return true;
}

bool build_contributions(int n, int T, const VertexTets &vt, const int32_t *row_ptr, const int32_t *slots,
                         Symbolic &sym, std::string &err, int n_tris, const int32_t *tri_slots) {
    const int64_t nnzb = row_ptr[n];
    if ((int64_t)T * 16 + (int64_t)n_tris * 9 > (int64_t)INT32_MAX) {
        err = "too many tets and tris for 32-bit contribution codes";
        return false;
    }
    // Contribution (k, l) of an element with slots S (N x N) is kept where
    // slot (k, l) <= slot (l, k): rows ascend with the slots, so these are the
    // diagonal and the upper triangle of H.  A tet's corners are distinct, so
    // the contributions to a row's slots are those of the row's tets, one
    // corner each: rows are independent.
    const auto &vptr = vt.ptr;
    const auto &vcode = vt.code;
    const int threads = thread_count(n, kThreadRows);
    std::vector<int32_t> start(nnzb + 1, 0), mate(nnzb, 0);
    const auto row_contributions = [&](int v, const auto &keep) {
        for (int64_t i = vptr[v]; i < vptr[v + 1]; ++i) {
            const int64_t e = vcode[i] >> 2;
            const int k = vcode[i] & 3;
            const int32_t *S = slots + 16 * e;
            for (int l = 0; l < 4; ++l)
                if (S[k * 4 + l] <= S[l * 4 + k]) keep(S[k * 4 + l], S[l * 4 + k], (int32_t)(16 * e + 4 * k + l));
        }
    };
    parallel_rows(n, threads, [&](int, int first, int last) {
        for (int v = first; v < last; ++v)
            row_contributions(v, [&](int32_t s, int32_t m, int32_t) {
                start[s + 1]++;
                mate[s] = s == m ? ~v : m;
            });
    });
    for (int64_t t = 0; t < n_tris; ++t) {
        const int32_t *S = tri_slots + 9 * t;
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                const int32_t s = S[i * 3 + j], m = S[j * 3 + i];
                if (s > m) continue;
                start[s + 1]++;
                if (s != m) mate[s] = m;
            }
    }
    // a vertex without tets still owns its diagonal block (mass + attachment):
    // give it one empty contribution so the assembly visits it
    std::vector<int32_t> isolated;  // diagonal slots of vertices in no tet
    for (int v = 0; v < n; ++v) {
        if (vptr[v] < vptr[v + 1]) continue;  // its tets' diagonal blocks are in the slot map
        const int32_t *b = sym.col_idx.data() + row_ptr[v];
        const int32_t *e = sym.col_idx.data() + row_ptr[v + 1];
        const int32_t *p = std::lower_bound(b, e, v);
        if (p == e || *p != v) {
            err = "sparsity lacks diagonal block of vertex " + std::to_string(v);
            return false;
        }
        const int32_t ds = (int32_t)(p - sym.col_idx.data());
        mate[ds] = ~v;
        if (start[ds + 1] == 0) {
            start[ds + 1] = 1;
            isolated.push_back(ds);
        }
    }
    if ((int64_t)T * 16 + (int64_t)n_tris * 9 + (int64_t)isolated.size() > (int64_t)INT32_MAX) {
        err = "too many contributions";
        return false;
    }
    for (int64_t s = 0; s < nnzb; ++s) start[s + 1] += start[s];
    sym.contrib_code.resize(start[nnzb]);
    std::vector<int32_t> fill(start.begin(), start.end() - 1);
    for (int32_t s : isolated) sym.contrib_code[fill[s]++] = mate[s];
    parallel_rows(n, threads, [&](int, int first, int last) {
        for (int v = first; v < last; ++v)
            row_contributions(v, [&](int32_t s, int32_t, int32_t code) { sym.contrib_code[fill[s]++] = code; });
    });
    // surface-tri contact blocks (i, j) after the tets of their slot, coded
    // 16 T + 9 tri + 3 i + j
    for (int64_t t = 0; t < n_tris; ++t) {
        const int32_t *S = tri_slots + 9 * t;
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j)
                if (S[i * 3 + j] <= S[j * 3 + i])
                    sym.contrib_code[fill[S[i * 3 + j]]++] = (int32_t)(16 * (int64_t)T + 9 * t + i * 3 + j);
    }
    // pack whole slots into chunks of <= 32 contributions (a longer slot gets
    // a chunk of its own)
    sym.chunk.clear();
    sym.pair.clear();
    int4 c = {0, 0, 0, 0};
    auto close = [&] {
        if (c.y > c.x) sym.chunk.push_back(c);
        c = {c.y, c.y, (int32_t)sym.pair.size(), 0};
    };
    for (int64_t s = 0; s < nnzb; ++s) {
        const int32_t len = start[s + 1] - start[s];
        if (len == 0) continue;
        if (c.y - c.x + len > 32) close();
        c.w |= (int32_t)(1u << (c.y - c.x));
        c.y += len;
        sym.pair.push_back(int2{(int32_t)s, mate[s]});
        if (c.y - c.x >= 32) close();
    }
    close();
    return true;
}

}  // namespace mfem
