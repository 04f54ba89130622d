// Checks of the resident PCG's host partition (csrc/partition.cpp) on random
// meshes: every row has one part, every block one lane of its row with the
// right local column, every halo row exactly one sender, and the layout's
// maxima bound every part.  Prints "ok" or the first violation.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include <vector>

#include "internal.h"

using namespace mfem;

#define CHECK(cond)                                                     \
    do {                                                                \
        if (!(cond)) {                                                  \
            printf("trial %d, line %d: %s\n", trial, __LINE__, #cond); \
            return 1;                                                   \
        }                                                               \
    } while (0)

int main() {
    std::mt19937 rng(7);
    auto below = [&](int k) { return (int)(rng() % (unsigned)k); };
    for (int trial = 0; trial < 80; ++trial) {
        // a Kuhn grid, shuffled in half of the trials; degenerate positions and
        // extra long-range couplings in some
        const int nx = 1 + below(14), ny = 1 + below(7), nz = 1 + below(7);
        const int n = (nx + 1) * (ny + 1) * (nz + 1), lo = trial % 3 == 0 ? 5 : 0;
        std::vector<int> perm(n);
        for (int i = 0; i < n; ++i) perm[i] = i;
        if (trial & 1) std::shuffle(perm.begin(), perm.end(), rng);
        std::vector<float> q(3 * (size_t)(n + lo), 0.0f);
        std::vector<std::set<int>> adj(n);
        auto id = [&](int i, int j, int k) { return perm[(i * (ny + 1) + j) * (nz + 1) + k]; };
        for (int i = 0; i <= nx; ++i)
            for (int j = 0; j <= ny; ++j)
                for (int k = 0; k <= nz; ++k) {
                    const int v = id(i, j, k);
                    adj[v].insert(v);
                    const float c[3] = {(float)i, (float)j, (float)k};
                    for (int a = 0; a < 3; ++a) q[3 * (size_t)(v + lo) + a] = trial % 7 == 3 ? 0.0f : c[a];
                    for (int d = 1; d < 8; ++d) {
                        const int i2 = i + (d & 1), j2 = j + ((d >> 1) & 1), k2 = k + (d >> 2);
                        if (i2 > nx || j2 > ny || k2 > nz) continue;
                        adj[v].insert(id(i2, j2, k2));
                        adj[id(i2, j2, k2)].insert(v);
                    }
                }
        if (trial % 11 == 4)
            for (int t = 0; t < n / 3; ++t) {
                const int a = below(n), b = below(n);
                adj[a].insert(b);
                adj[b].insert(a);
            }
        if (trial % 13 == 5) q[3 * (size_t)(lo + below(n))] = NAN;
        // the body's rows are [lo, lo + n) of the plan's
        std::vector<int32_t> rp(n + lo + 1, 0), ci;
        for (int i = 0; i < lo; ++i) {
            ci.push_back(i);
            rp[i + 1] = (int32_t)ci.size();
        }
        for (int i = 0; i < n; ++i) {
            for (int c : adj[i]) ci.push_back(c + lo);
            rp[lo + i + 1] = (int32_t)ci.size();
        }
        const int parts = trial % 5 == 0 ? 1 + below(13) : 1 << below(5);
        ResidentHost h;
        // the lower and upper CSR of a factor preconditioner's form
        std::vector<int32_t> lrow(n + lo + 1, 0), urow(n + lo + 1, 0), lcol, ucol;
        for (int r = 0; r < n + lo; ++r) {
            for (int k = rp[r]; k < rp[r + 1]; ++k) {
                if (ci[k] <= r) lcol.push_back(ci[k]);
                if (ci[k] >= r) ucol.push_back(ci[k]);
            }
            lrow[r + 1] = (int32_t)lcol.size();
            urow[r + 1] = (int32_t)ucol.size();
        }
        const ResidentFactor form{2 + trial % 2, lrow.data(), urow.data(), trial % 3 != 1};
        const ResidentFactor *factor = trial % 4 == 3 || trial % 4 == 2 ? &form : nullptr;
        const bool redundant = factor && form.redundant;
        const int32_t off[3] = {0, lo, lo + n};
        if (trial % 4 == 2 && lo > 0) {
            // behind a body of single rows: joined arrays
            ResidentHost both;
            resident_add_bodies(both, rp.data(), ci.data(), q.data(), off, {0, 1}, parts, factor);
            CHECK((int)both.parts.size() == 2 * parts && both.tasks.size() == 2 && both.tasks[1].x == parts);
            both.parts.erase(both.parts.begin(), both.parts.begin() + parts);
            both.tasks.erase(both.tasks.begin());
            h = both;
        } else if (trial % 4 == 1 && lo == 0 && n >= 3 * parts) {
            // runs of whole blocks of consecutive rows
            const int blocks = parts + below(2 * parts);
            resident_add_ranges(h, rp.data(), ci.data(), n, parts, blocks, true);
            for (int p = 0, b = 0; p < parts; ++p) {
                const ResPart &P = h.parts[p];
                CHECK(P.block_lo == b && P.nblocks >= 1 && P.nblocks <= h.block_max);
                b += P.nblocks;
                CHECK(P.row_off == (int)((long long)n * P.block_lo / blocks));
                CHECK(P.row_off + P.nown == (int)((long long)n * b / blocks));
                for (int i = 0; i < P.nown; ++i)
                    CHECK(h.rows[P.row_off + i] >= P.row_off && h.rows[P.row_off + i] < P.row_off + P.nown);
            }
        } else {
            resident_add_body(h, rp.data(), ci.data(), q.data(), lo, lo + n, parts, 0, true, true, factor);
        }
        CHECK((int)h.parts.size() == parts && h.tasks.size() == 1 && h.tasks[0].y == parts);
        std::vector<int> seen(n, 0);
        std::vector<std::vector<int>> sender(parts);
        for (int p = 0; p < parts; ++p) sender[p].assign(h.parts[p].nhalo, -1);
        int most = 0, least = n;
        for (int p = 0; p < parts; ++p) {
            const ResPart &P = h.parts[p];
            most = std::max(most, P.nown);
            least = std::min(least, P.nown);
            CHECK(P.nown <= h.nown_max && P.nhalo <= h.nhalo_max && P.nown + P.nhalo <= h.nlocal_max);
            CHECK(P.push_passes * P.nslices * 32 <= h.push_max);
            for (int s = 0; s < P.nslices; ++s)
                for (int lane = 0; lane < 32; ++lane)
                    for (int e = 0; e < P.push_passes; ++e) {
                        const int d = h.push[P.push_off + (e * P.nslices + s) * 32 + lane];
                        const int r = s * kPartSliceRows + lane % kPartSliceRows;
                        if (d < 0) continue;
                        CHECK(r < P.nown && (d >> 16) < parts && (d >> 16) != p);
                        CHECK((d & 0xffff) < h.parts[d >> 16].nhalo && sender[d >> 16][d & 0xffff] < 0);
                        sender[d >> 16][d & 0xffff] = h.rows[P.row_off + r];
                    }
            std::vector<std::set<int>> blocks(P.nown);
            std::vector<int> warp(kPartWarps, 0), reg(kPartWarps, 0);
            for (int s = 0; s < P.nslices; ++s) {
                const int t0 = h.trip_ptr[P.slice_off + s], t1 = h.trip_ptr[P.slice_off + s + 1];
                CHECK(t1 > t0 && t1 - t0 <= h.slice_trips_max);
                warp[s % kPartWarps] += t1 - t0;
                if (s < kPartWarps) reg[s] = std::min(t1 - t0, kPartRegTrips);
                for (int t = t0; t < t1; ++t)
                    for (int lane = 0; lane < 32; ++lane) {
                        const int k = h.src[32 * t + lane], c = h.col[32 * t + lane];
                        const int r = s * kPartSliceRows + lane % kPartSliceRows;
                        if (k < 0) {
                            CHECK(c == 0);
                            continue;
                        }
                        CHECK(r < P.nown);
                        const int row = h.rows[P.row_off + r];
                        CHECK(k >= rp[row] && k < rp[row + 1]);
                        CHECK(c >= 0 && c < (redundant ? P.second_rows : P.nown + P.nhalo));
                        CHECK((c < P.nown ? h.rows[P.row_off + c] : h.halo[P.halo_off + c - P.nown]) == ci[k]);
                        blocks[r].insert(k);
                    }
            }
            for (int w = 0; w < kPartWarps; ++w)
                CHECK(warp[w] <= h.trips_max && warp[w] - reg[w] <= h.trips_max_reg);
            auto vertex = [&](int i) {
                return i < P.nown ? h.rows[P.row_off + i] : h.halo[P.halo_off + i - P.nown];
            };
            for (int w = 0; factor && w < 2; ++w) {
                // pass w's rows, each block once, its column among the rows
                // that hold the pass's input
                const bool lower = (w == 0) == (form.mode == 2);
                const int rows = w == 0 ? P.first_rows : P.second_rows;
                const int inputs = redundant && w == 1 ? P.first_rows : P.nown + P.nhalo;
                CHECK(rows >= P.nown && rows <= P.nown + P.nhalo && (redundant || rows == P.nown));
                CHECK(P.nfslices[w] == (rows + kFactorSliceRows - 1) / kFactorSliceRows);
                std::vector<int> count(rows, 0);
                for (int s = 0; s < P.nfslices[w]; ++s) {
                    const int t0 = h.ftrip_ptr[P.fslice_off[w] + s], t1 = h.ftrip_ptr[P.fslice_off[w] + s + 1];
                    CHECK(t1 > t0 && t1 - t0 <= h.slice_trips_max);
                    for (int t = t0; t < t1; ++t)
                        for (int lane = 0; lane < 32; ++lane) {
                            const int k = h.fsrc[32 * t + lane], c = h.fcol[32 * t + lane];
                            if (k < 0) continue;
                            const int r = s * kFactorSliceRows + lane;
                            CHECK(r < rows && c < inputs);
                            const int row = vertex(r);
                            const std::vector<int32_t> &ptr = lower ? lrow : urow, &cols = lower ? lcol : ucol;
                            CHECK(k >= ptr[row] && k < ptr[row + 1] && cols[k] == vertex(c));
                            ++count[r];
                        }
                }
                for (int i = 0; i < rows; ++i)
                    CHECK(count[i] == (lower ? lrow : urow)[vertex(i) + 1] - (lower ? lrow : urow)[vertex(i)]);
                CHECK(h.ftrip_ptr[P.fslice_off[w] + P.nfslices[w]] - h.ftrip_ptr[P.fslice_off[w]] <=
                      h.f_trips_max[w]);
            }
            // the passes' push table sends every row where the product's does
            if (factor) {
                const int fs = (P.nown + kFactorSliceRows - 1) / kFactorSliceRows;
                std::vector<std::set<int>> a(P.nown), b(P.nown);
                for (int s = 0; s < P.nslices; ++s)
                    for (int e = 0; e < P.push_passes * 32; ++e) {
                        const int lane = e % 32, d = h.push[P.push_off + (e / 32 * P.nslices + s) * 32 + lane];
                        if (d >= 0) a[s * kPartSliceRows + lane % kPartSliceRows].insert(d);
                    }
                for (int s = 0; s < fs; ++s)
                    for (int e = 0; e < P.fpush_passes * 32; ++e) {
                        const int d = h.fpush[P.fpush_off + (e / 32 * fs + s) * 32 + e % 32];
                        if (d < 0) continue;
                        CHECK(s * kFactorSliceRows + e % 32 < P.nown);
                        b[s * kFactorSliceRows + e % 32].insert(d);
                    }
                CHECK(a == b && P.fpush_passes * fs * 32 <= h.fpush_max);
            }
            for (int i = 0; i < P.nown; ++i) {
                const int row = h.rows[P.row_off + i];
                CHECK(row >= lo && row < lo + n);
                ++seen[row - lo];
                CHECK((int)blocks[i].size() == rp[row + 1] - rp[row]);
            }
        }
        CHECK(h.blocks > 0 || most - least <= 2);
        for (int v : seen) CHECK(v == 1);
        for (int p = 0; p < parts; ++p)
            for (int i = 0; i < h.parts[p].nhalo; ++i) CHECK(sender[p][i] == h.halo[h.parts[p].halo_off + i]);
    }
    puts("ok");
    return 0;
}
