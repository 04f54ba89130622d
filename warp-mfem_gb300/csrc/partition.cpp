// Host side of the resident PCG (pcg_resident.cu): a body's rows split into
// parts by recursive coordinate bisection of the rest positions, each part's
// halo (the other parts' rows its columns reach), the sliced layout of its
// blocks and, per row, the parts that need it.
//
// Bisection by position keeps a part compact whatever the vertex order, so
// the halo stays near the surface of a block of rows: 64x16x16 cells in 152
// parts, 124 rows a part, need 146 to 221 foreign rows against 310 for
// contiguous row ranges of the x-major order (and nearly every row of the
// mesh for a shuffled one).
#include "host_parallel.h"
#include "internal.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>

namespace mfem {
namespace {

constexpr int kThreadRows = 768;  // 0.5 to 1 us of work a row

struct Bisector {
    const float *q;  // [n][3]

    struct Run {
        int first, last, parts, part;  // rows [first, last) become parts [part, part + parts)
    };

    float coord(int v, int axis) const {
        const float c = q[3 * (size_t)v + axis];
        return std::isfinite(c) ? c : 0.0f;
    }

    // Halves a run of at least two parts across its longest extent.
    void halve(int *rows, const Run &r, Run &a, Run &b) const {
        float lo[3], hi[3];
        for (int x = 0; x < 3; ++x) lo[x] = INFINITY, hi[x] = -INFINITY;
        for (int i = r.first; i < r.last; ++i)
            for (int x = 0; x < 3; ++x) {
                const float c = coord(rows[i], x);
                lo[x] = std::min(lo[x], c);
                hi[x] = std::max(hi[x], c);
            }
        int axis = 0;
        for (int x = 1; x < 3; ++x)
            if (hi[x] - lo[x] > hi[axis] - lo[axis]) axis = x;
        const int left = r.parts / 2;
        const int mid = r.first + (int)(((int64_t)(r.last - r.first) * left) / r.parts);
        std::nth_element(rows + r.first, rows + mid, rows + r.last, [&](int u, int v) {
            const float cu = coord(u, axis), cv = coord(v, axis);
            return cu < cv || (cu == cv && u < v);
        });
        a = Run{r.first, mid, left, r.part};
        b = Run{mid, r.last, r.parts - left, r.part + left};
    }

    // Splits the rows into `parts` runs of nearly equal length, level by
    // level; bounds[p], bounds[p + 1] are run p's.
    void split(std::vector<int> &rows, int parts, std::vector<int> &bounds, int threads) const {
        std::vector<Run> runs{Run{0, (int)rows.size(), parts, 0}}, next;
        while (!runs.empty()) {
            next.assign(2 * runs.size(), Run{0, 0, 1, -1});
            parallel_for((int)runs.size(), threads, [&](int i) {
                if (runs[i].parts > 1) halve(rows.data(), runs[i], next[2 * i], next[2 * i + 1]);
            });
            for (const Run &r : runs)
                if (r.parts == 1) bounds[r.part + 1] = r.last;
            runs.clear();
            for (const Run &r : next)
                if (r.part >= 0) runs.push_back(r);
        }
    }
};

// Adds the parts rows[bounds[p] .. bounds[p + 1]) of one body; in_order: the
// blocks of a row stay in their order.
void add_parts(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, int row_lo, int body,
               std::vector<int> &rows, const std::vector<int> &bounds, bool push_lists, int threads,
               const ResidentFactor *factor, bool in_order);

// One part's arrays before they are joined.
struct PartArrays {
    std::vector<int32_t> halo, trip_ptr, src;
    std::vector<uint16_t> col;
    int trips_max = 0, trips_max_reg = 0, slice_trips_max = 0;
    int second_rows = 0, first_rows = 0, f_trips_max[2] = {0, 0};
    std::vector<int32_t> ftrip_ptr[2], fsrc[2];
    std::vector<uint16_t> fcol[2];
};

struct RowBlocks {
    int32_t src;
    const int32_t *cols;
    int len;
};

// Deals the blocks of eight rows, which a quarter warp's lanes multiply side
// by side, to steps: one block a row and step, and as far as possible no two
// blocks of a step in the same bank group of the window (16-byte entries,
// eight groups), so that the eight lanes' reads take one pass of shared
// memory.  This is an edge colouring of the multigraph of rows and bank
// groups; as many steps as the highest degree suffice (Konig 1916), found
// edge by edge with alternating paths.  Blocks of a group with more blocks
// than steps go where their row is free.  A trip's 32 window reads take 5.0
// passes instead of 7.0 (64x16x16 cells in 147 parts, the product; 5.7 for 7.1
// in the FSAI passes; 5.6 for 9.0 and 4.5 for 7.7 in a shuffled mesh), of four
// at least: 1 to 3% of a solve, for 0.1 us a row of one thread here.
class BankDeal {
public:
    static constexpr int kMaxSteps = 64;
    explicit BankDeal(int steps) : steps_(steps) {
        const uint64_t all = steps >= 64 ? ~uint64_t(0) : (uint64_t(1) << steps) - 1;
        for (int i = 0; i < 8; ++i) {
            row_free_[i] = bank_free_[i] = all;
            for (int c = 0; c < steps; ++c) at_row_[i][c] = at_bank_[i][c] = kNone;
        }
    }

    // Block e of row r, whose column is in group `bank`.
    void add(int r, int e, int bank) {
        bank_of_[r][e] = (uint8_t)bank;
        if (!bank_free_[bank]) {
            const int c = first(row_free_[r]);
            bank_of_[r][e] |= kLoose;
            at_row_[r][c] = (uint8_t)e;
            row_free_[r] &= ~bit(c);
            return;
        }
        int c;
        if (const uint64_t both = row_free_[r] & bank_free_[bank]) {
            c = first(both);
        } else {
            c = first(row_free_[r]);
            flip(bank, c, first(bank_free_[bank]));
        }
        at_row_[r][c] = (uint8_t)e;
        at_bank_[bank][c] = (uint8_t)r;
        row_free_[r] &= ~bit(c);
        bank_free_[bank] &= ~bit(c);
    }

    // Row r's block in step c, -1: none.
    int block(int r, int c) const { return at_row_[r][c] == kNone ? -1 : at_row_[r][c]; }

private:
    static constexpr uint8_t kNone = 0xff, kLoose = 0x80;
    static uint64_t bit(int c) { return uint64_t(1) << c; }
    static int first(uint64_t m) { return __builtin_ctzll(m); }

    // Exchanges steps x and y along the path that leaves group b by x, where y
    // is free: x is free there afterwards.
    void flip(int b, int x, int y) {
        bank_free_[b] = (bank_free_[b] | bit(x)) & ~bit(y);
        int r = at_bank_[b][x];
        at_bank_[b][x] = kNone;
        for (;;) {
            const uint8_t e1 = at_row_[r][x], e2 = at_row_[r][y];
            at_bank_[b][y] = (uint8_t)r;
            at_row_[r][y] = e1;
            at_row_[r][x] = e2;
            if (e2 == kNone) {
                row_free_[r] = (row_free_[r] | bit(x)) & ~bit(y);
                return;
            }
            if (bank_of_[r][e2] & kLoose) return;
            b = bank_of_[r][e2];
            const uint8_t next = at_bank_[b][x];
            at_bank_[b][x] = (uint8_t)r;
            if (next == kNone) {
                at_bank_[b][y] = kNone;
                bank_free_[b] = (bank_free_[b] | bit(y)) & ~bit(x);
                return;
            }
            r = next;
        }
    }

    int steps_;
    uint64_t row_free_[8], bank_free_[8];
    uint8_t at_row_[8][kMaxSteps], at_bank_[8][kMaxSteps];  // block of the row, row of the group
    uint8_t bank_of_[8][kMaxSteps];
};

// Slices of ROWS rows, 32 / ROWS lanes a row; a trip is one block a
// lane, padded lanes read no block (src -1).  row_blocks(i) gives local row
// i's blocks: its first src, its columns and their number; local(c) a
// column's local row.  in_order keeps a row's blocks in their order;
// otherwise they are dealt as above.  warp_trips[w] gets the trips of warp w's
// slices.
template <int ROWS, class R, class L>
void slice_rows(int nrows, const R &row_blocks, const L &local, bool in_order, std::vector<int32_t> &trip_ptr,
                std::vector<int32_t> &src, std::vector<uint16_t> &col, std::vector<int> &slice_trips) {
    constexpr int lanes = 32 / ROWS;
    for (int r0 = 0; r0 < nrows; r0 += ROWS) {
        const int nr = std::min(ROWS, nrows - r0);
        RowBlocks rb[ROWS];
        int trips = 0;
        for (int r = 0; r < nr; ++r) {
            rb[r] = row_blocks(r0 + r);
            trips = std::max(trips, (rb[r].len + lanes - 1) / lanes);
        }
        trip_ptr.push_back((int32_t)(src.size() / 32));
        slice_trips.push_back(trips);
        const size_t base = src.size();
        src.resize(base + (size_t)32 * trips, -1);
        col.resize(base + (size_t)32 * trips, 0);
        const int steps = trips * lanes;
        const auto place = [&](int r, int step) {
            return base + (size_t)(step / lanes) * 32 + step % lanes * ROWS + r;
        };
        if (in_order || steps > BankDeal::kMaxSteps) {
            for (int r = 0; r < nr; ++r)
                for (int e = 0; e < rb[r].len; ++e) {
                    const size_t at = place(r, e);
                    src[at] = rb[r].src + e;
                    col[at] = (uint16_t)local(rb[r].cols[e]);
                }
            continue;
        }
        for (int g = 0; g < ROWS; g += 8) {
            BankDeal deal(steps);
            uint16_t cols[8][BankDeal::kMaxSteps];
            for (int r = g; r < std::min(g + 8, nr); ++r)
                for (int e = 0; e < rb[r].len; ++e) {
                    cols[r - g][e] = (uint16_t)local(rb[r].cols[e]);
                    deal.add(r - g, e, cols[r - g][e] & 7);
                }
            for (int c = 0; c < steps; ++c) {
                uint16_t with = 0;
                for (int r = 0; r < 8; ++r) {
                    const int e = deal.block(r, c);
                    if (e < 0) continue;
                    const size_t at = place(g + r, c);
                    src[at] = rb[g + r].src + e;
                    col[at] = with = cols[r][e];
                }
                // a factor pass's lane without a block reads with another one
                // (the product's kernel sees to it itself)
                for (int r = 0; ROWS == kFactorSliceRows && r < 8; ++r)
                    if (deal.block(r, c) < 0) col[place(g + r, c)] = with;
            }
        }
    }
    trip_ptr.push_back((int32_t)(src.size() / 32));
}

}  // namespace

void resident_add_body(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, const float *rest_q,
                       int row_lo, int row_hi, int parts, int body, bool push_lists, bool parallel,
                       const ResidentFactor *factor) {
    const int n = row_hi - row_lo;
    const int threads = parallel ? thread_count(n, kThreadRows) : 1;
    std::vector<int> rows(n), bounds(parts + 1, 0);
    for (int i = 0; i < n; ++i) rows[i] = row_lo + i;
    Bisector{rest_q}.split(rows, parts, bounds, threads);
    add_parts(h, row_ptr, col_idx, row_lo, body, rows, bounds, push_lists, threads, factor, false);
}

bool ordered_sums_fit(const ResidentHost &h, int cluster, bool grid) {
    if (grid) return h.block_max <= 1;
    const int n = h.tasks[0].w, tasks = cluster > 1 ? kPartTasks : 1;
    return h.block_max <= (cluster > 1 ? kPartMaxBlocks : 2) && 3 * ((n + h.blocks - 1) / h.blocks) <= 32 * kPartWarps &&
           h.block_max * ordered_block_warps(n, h.blocks) <= kPartWarps * tasks;
}

void resident_add_ranges(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, int n, int parts, int blocks,
                         bool push_lists) {
    std::vector<int> rows(n), bounds(parts + 1, 0);
    for (int i = 0; i < n; ++i) rows[i] = i;
    const int first_part = (int)h.parts.size();
    for (int p = 1; p <= parts; ++p) bounds[p] = (int)((int64_t)n * ((int64_t)blocks * p / parts) / blocks);
    add_parts(h, row_ptr, col_idx, 0, 0, rows, bounds, push_lists, thread_count(n, kThreadRows), nullptr, true);
    h.blocks = blocks;
    for (int p = 0; p < parts; ++p) {
        ResPart &rp = h.parts[first_part + p];
        rp.block_lo = (int)((int64_t)blocks * p / parts);
        rp.nblocks = (int)((int64_t)blocks * (p + 1) / parts) - rp.block_lo;
        h.block_max = std::max(h.block_max, rp.nblocks);
    }
}

namespace {

void add_parts(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, int row_lo, int body,
               std::vector<int> &rows, const std::vector<int> &bounds, bool push_lists, int threads,
               const ResidentFactor *factor, bool in_order) {
    const int n = (int)rows.size(), parts = (int)bounds.size() - 1;
    const int first_part = (int)h.parts.size();
    std::vector<int> part_of(n), local(n);
    parallel_for(parts, threads, [&](int p) {
        // rows of like length share a slice, so slices carry little padding;
        // else ascending, so that a slice's rows have consecutive neighbours
        const auto trips = [&](int r) { return (row_ptr[r + 1] - row_ptr[r] + kPartLanes - 1) / kPartLanes; };
        std::sort(rows.begin() + bounds[p], rows.begin() + bounds[p + 1], [&](int u, int v) {
            const int tu = trips(u), tv = trips(v);
            return tu > tv || (tu == tv && u < v);
        });
        for (int i = bounds[p]; i < bounds[p + 1]; ++i) {
            part_of[rows[i] - row_lo] = p;
            local[rows[i] - row_lo] = i - bounds[p];
        }
    });
    std::vector<PartArrays> made(parts);
    parallel_for(parts, threads, [&](int p) {
        PartArrays &m = made[p];
        const int lo = bounds[p], nown = bounds[p + 1] - lo;
        std::vector<char> met(n, 0);  // in the halo
        std::unique_ptr<int[]> halo_slot(new int[n]);  // set for the halo rows only
        // the halo: ascending rows of other parts that the columns of `span`
        // reach, appended hop by hop for a redundant factor (the rows that the
        // second pass, the first pass and the residual are needed on)
        const auto hop = [&](int from, int to, int side) {
            // local rows [from, to): every column, or the lower (-1) or upper (1) ones
            const size_t first = m.halo.size();
            for (int i = from; i < to; ++i) {
                const int row = i < nown ? rows[lo + i] : m.halo[i - nown];
                for (int k = row_ptr[row]; k < row_ptr[row + 1]; ++k) {
                    const int c = col_idx[k];
                    if ((side < 0 && c > row) || (side > 0 && c < row)) continue;
                    if (part_of[c - row_lo] == p || met[c - row_lo]) continue;
                    met[c - row_lo] = 1;
                    m.halo.push_back(c);
                }
            }
            std::sort(m.halo.begin() + first, m.halo.end());
            return nown + (int)m.halo.size();
        };
        const int reach = hop(0, nown, 0);
        m.second_rows = m.first_rows = nown;
        // the first pass's columns: lower for F^T F, upper for F F^T
        const int side0 = factor && factor->mode == 2 ? -1 : 1;
        if (factor && factor->redundant) {
            m.second_rows = reach;
            m.first_rows = hop(0, m.second_rows, -side0);
            hop(0, m.first_rows, side0);
        }
        for (size_t i = 0; i < m.halo.size(); ++i) halo_slot[m.halo[i] - row_lo] = (int)i;
        const auto local_row = [&](int c) {
            return part_of[c - row_lo] == p ? local[c - row_lo] : nown + halo_slot[c - row_lo];
        };
        const auto row_of = [&](int i) { return i < nown ? rows[lo + i] : m.halo[i - nown]; };
        std::vector<int> slice_trips;
        slice_rows<kPartSliceRows>(nown,
                   [&](int i) {
                       const int row = rows[lo + i];
                       return RowBlocks{row_ptr[row], col_idx + row_ptr[row], row_ptr[row + 1] - row_ptr[row]};
                   },
                   local_row, in_order, m.trip_ptr, m.src, m.col, slice_trips);
        const auto warp_most = [&](int skip) {
            int warp[kPartWarps] = {0}, most = 0;
            for (size_t s = 0; s < slice_trips.size(); ++s)
                warp[s % kPartWarps] += s < kPartWarps ? std::max(0, slice_trips[s] - skip) : slice_trips[s];
            for (int w : warp) most = std::max(most, w);
            return most;
        };
        m.trips_max = warp_most(0);
        m.trips_max_reg = warp_most(kPartRegTrips);
        for (int t : slice_trips) m.slice_trips_max = std::max(m.slice_trips_max, t);
        for (int w = 0; factor && w < 2; ++w) {
            const bool lower = (w == 0) == (side0 < 0);
            slice_trips.clear();
            slice_rows<kFactorSliceRows>(w == 0 ? m.first_rows : m.second_rows,
                       [&](int i) {
                           // columns ascend: the lower form is a row's head, the
                           // upper its tail, the diagonal in both
                           const int row = row_of(i);
                           const int32_t *c0 = col_idx + row_ptr[row], *c1 = col_idx + row_ptr[row + 1];
                           const int32_t *d = std::lower_bound(c0, c1, row);
                           return lower ? RowBlocks{factor->lrow[row], c0, (int)(d - c0) + 1}
                                        : RowBlocks{factor->urow[row], d, (int)(c1 - d)};
                       },
                       local_row, in_order, m.ftrip_ptr[w], m.fsrc[w], m.fcol[w], slice_trips);
            m.f_trips_max[w] = m.ftrip_ptr[w].back();
            for (int t : slice_trips) m.slice_trips_max = std::max(m.slice_trips_max, t);
        }
    });
    h.rows.insert(h.rows.end(), rows.begin(), rows.end());
    const int row_base = (int)h.rows.size() - n;
    size_t trips = h.src.size() / 32, halos = h.halo.size();
    for (int p = 0; p < parts; ++p) {
        const PartArrays &m = made[p];
        ResPart rp{};
        rp.row_off = row_base + bounds[p];
        rp.nown = bounds[p + 1] - bounds[p];
        rp.halo_off = (int)halos;
        rp.nhalo = (int)m.halo.size();
        rp.slice_off = (int)h.trip_ptr.size();
        rp.nslices = (int)m.trip_ptr.size() - 1;
        for (int32_t t : m.trip_ptr) h.trip_ptr.push_back((int32_t)trips + t);
        trips += m.src.size() / 32;
        halos += m.halo.size();
        h.trips_max = std::max(h.trips_max, m.trips_max);
        h.trips_max_reg = std::max(h.trips_max_reg, m.trips_max_reg);
        h.slice_trips_max = std::max(h.slice_trips_max, m.slice_trips_max);
        h.nown_max = std::max(h.nown_max, rp.nown);
        h.nhalo_max = std::max(h.nhalo_max, rp.nhalo);
        h.nlocal_max = std::max(h.nlocal_max, rp.nown + rp.nhalo);
        rp.second_rows = m.second_rows;
        rp.first_rows = m.first_rows;
        for (int w = 0; factor && w < 2; ++w) {
            const int32_t base = (int32_t)(h.fsrc.size() / 32);
            rp.fslice_off[w] = (int)h.ftrip_ptr.size();
            rp.nfslices[w] = (int)m.ftrip_ptr[w].size() - 1;
            for (int32_t t : m.ftrip_ptr[w]) h.ftrip_ptr.push_back(base + t);
            h.fsrc.insert(h.fsrc.end(), m.fsrc[w].begin(), m.fsrc[w].end());
            h.fcol.insert(h.fcol.end(), m.fcol[w].begin(), m.fcol[w].end());
            h.f_trips_max[w] = std::max(h.f_trips_max[w], m.f_trips_max[w]);
        }
        h.parts.push_back(rp);
    }
    h.halo.resize(halos);
    h.src.resize(32 * trips);
    h.col.resize(32 * trips);
    parallel_for(parts, threads, [&](int p) {
        const ResPart &rp = h.parts[first_part + p];
        const PartArrays &m = made[p];
        std::copy(m.halo.begin(), m.halo.end(), h.halo.begin() + rp.halo_off);
        const size_t at = (size_t)32 * h.trip_ptr[rp.slice_off];
        std::copy(m.src.begin(), m.src.end(), h.src.begin() + at);
        std::copy(m.col.begin(), m.col.end(), h.col.begin() + at);
    });
    h.tasks.push_back(make_int4(first_part, parts, body, n));
    if (!push_lists) return;
    // destinations of a row's product, dealt to the row's lanes: pass e holds
    // entry e * kPartLanes + lane of each row's list
    std::vector<std::vector<int>> push(n);  // per row of the body: (part << 16 | halo index)
    for (int p = 0; p < parts; ++p)
        for (size_t i = 0; i < made[p].halo.size(); ++i) push[made[p].halo[i] - row_lo].push_back(p << 16 | (int)i);
    for (int p = 0; p < parts; ++p) {
        const int lo = bounds[p], hi = bounds[p + 1];
        ResPart &rp = h.parts[first_part + p];
        size_t most = 0;
        for (int i = lo; i < hi; ++i) most = std::max(most, push[rows[i] - row_lo].size());
        rp.push_off = (int)h.push.size();
        rp.push_passes = (int)((most + kPartLanes - 1) / kPartLanes);
        h.push.resize(h.push.size() + (size_t)rp.push_passes * rp.nslices * 32, -1);
        for (int i = lo; i < hi; ++i) {
            const auto &dst = push[rows[i] - row_lo];
            for (size_t e = 0; e < dst.size(); ++e)
                h.push[rp.push_off + (e / kPartLanes * rp.nslices + (i - lo) / kPartSliceRows) * 32 +
                       e % kPartLanes * kPartSliceRows + (i - lo) % kPartSliceRows] = dst[e];
        }
        h.push_max = std::max(h.push_max, rp.push_passes * rp.nslices * 32);
        if (!factor) continue;
        const int slices = (rp.nown + kFactorSliceRows - 1) / kFactorSliceRows;
        rp.fpush_off = (int)h.fpush.size();
        rp.fpush_passes = (int)most;
        h.fpush.resize(h.fpush.size() + most * slices * 32, -1);
        for (int i = lo; i < hi; ++i) {
            const auto &dst = push[rows[i] - row_lo];
            for (size_t e = 0; e < dst.size(); ++e)
                h.fpush[rp.fpush_off + (e * slices + (i - lo) / kFactorSliceRows) * 32 + (i - lo) % kFactorSliceRows] =
                    dst[e];
        }
        h.fpush_max = std::max(h.fpush_max, rp.fpush_passes * slices * 32);
    }
}

}  // namespace

void resident_add_bodies(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, const float *rest_q,
                         const int32_t *row_off, const std::vector<int> &bodies, int parts,
                         const ResidentFactor *factor) {
    std::vector<ResidentHost> made(bodies.size());
    int rows = 0;
    for (int b : bodies) rows += row_off[b + 1] - row_off[b];
    parallel_for((int)bodies.size(), thread_count(rows, kThreadRows), [&](int i) {
        const int b = bodies[i];
        resident_add_body(made[i], row_ptr, col_idx, rest_q, row_off[b], row_off[b + 1], parts, b, parts > 1, false,
                          factor);
    });
    for (const ResidentHost &m : made) {
        const int first = (int)h.parts.size(), trips = (int)(h.src.size() / 32);
        const int ftrips = (int)(h.fsrc.size() / 32);
        for (ResPart rp : m.parts) {
            rp.row_off += (int)h.rows.size();
            rp.halo_off += (int)h.halo.size();
            rp.slice_off += (int)h.trip_ptr.size();
            rp.push_off += (int)h.push.size();
            for (int &off : rp.fslice_off) off += (int)h.ftrip_ptr.size();
            rp.fpush_off += (int)h.fpush.size();
            h.parts.push_back(rp);
        }
        for (int4 t : m.tasks) h.tasks.push_back(make_int4(first + t.x, t.y, t.z, t.w));
        h.rows.insert(h.rows.end(), m.rows.begin(), m.rows.end());
        h.halo.insert(h.halo.end(), m.halo.begin(), m.halo.end());
        for (int32_t t : m.trip_ptr) h.trip_ptr.push_back(trips + t);
        h.src.insert(h.src.end(), m.src.begin(), m.src.end());
        h.col.insert(h.col.end(), m.col.begin(), m.col.end());
        h.push.insert(h.push.end(), m.push.begin(), m.push.end());
        h.fpush.insert(h.fpush.end(), m.fpush.begin(), m.fpush.end());
        h.fpush_max = std::max(h.fpush_max, m.fpush_max);
        for (int32_t t : m.ftrip_ptr) h.ftrip_ptr.push_back(ftrips + t);
        h.fsrc.insert(h.fsrc.end(), m.fsrc.begin(), m.fsrc.end());
        h.fcol.insert(h.fcol.end(), m.fcol.begin(), m.fcol.end());
        for (int w = 0; w < 2; ++w) h.f_trips_max[w] = std::max(h.f_trips_max[w], m.f_trips_max[w]);
        h.nown_max = std::max(h.nown_max, m.nown_max);
        h.nhalo_max = std::max(h.nhalo_max, m.nhalo_max);
        h.nlocal_max = std::max(h.nlocal_max, m.nlocal_max);
        h.push_max = std::max(h.push_max, m.push_max);
        h.trips_max = std::max(h.trips_max, m.trips_max);
        h.trips_max_reg = std::max(h.trips_max_reg, m.trips_max_reg);
        h.slice_trips_max = std::max(h.slice_trips_max, m.slice_trips_max);
    }
}

}  // namespace mfem
