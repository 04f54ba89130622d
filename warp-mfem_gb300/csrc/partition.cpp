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
#include "internal.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <exception>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>

namespace mfem {
namespace {

constexpr int kMaxThreads = 8;
constexpr int kThreadRows = 2048;  // a thread for every so many rows

// Runs fn(i) for i in [0, count) on up to `threads` threads, this one
// included; an exception of fn leaves here, as from a plain loop.
template <class F>
void parallel_for(int count, int threads, const F &fn) {
    std::atomic<int> next{0};
    std::exception_ptr failed;
    std::mutex lock;
    auto work = [&] {
        try {
            for (int i = next++; i < count; i = next++) fn(i);
        } catch (...) {
            std::lock_guard<std::mutex> hold(lock);
            failed = std::current_exception();
            next = count;
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(std::max(0, std::min(threads, count) - 1));
    try {
        for (int t = 1; t < std::min(threads, count); ++t) pool.emplace_back(work);
    } catch (const std::system_error &) {  // no more threads: the ones there are do it
    }
    work();
    for (auto &t : pool) t.join();
    if (failed) std::rethrow_exception(failed);
}

int thread_count(int rows) {
    const int hw = (int)std::thread::hardware_concurrency();
    return std::max(1, std::min(std::min(kMaxThreads, hw), rows / kThreadRows));
}

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

// Adds the parts rows[bounds[p] .. bounds[p + 1]) of one body.
void add_parts(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, int row_lo, int body,
               std::vector<int> &rows, const std::vector<int> &bounds, bool push_lists, int threads);

// One part's arrays before they are joined.
struct PartArrays {
    std::vector<int32_t> halo, trip_ptr, src;
    std::vector<uint16_t> col;
    int trips_max = 0, trips_max_reg = 0, slice_trips_max = 0;
};

}  // namespace

void resident_add_body(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, const float *rest_q,
                       int row_lo, int row_hi, int parts, int body, bool push_lists, bool parallel) {
    const int n = row_hi - row_lo;
    const int threads = parallel ? thread_count(n) : 1;
    std::vector<int> rows(n), bounds(parts + 1, 0);
    for (int i = 0; i < n; ++i) rows[i] = row_lo + i;
    Bisector{rest_q}.split(rows, parts, bounds, threads);
    add_parts(h, row_ptr, col_idx, row_lo, body, rows, bounds, push_lists, threads);
}

void resident_add_ranges(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, int n, int parts, int blocks,
                         bool push_lists) {
    std::vector<int> rows(n), bounds(parts + 1, 0);
    for (int i = 0; i < n; ++i) rows[i] = i;
    const int first_part = (int)h.parts.size();
    for (int p = 1; p <= parts; ++p) bounds[p] = (int)((int64_t)n * ((int64_t)blocks * p / parts) / blocks);
    add_parts(h, row_ptr, col_idx, 0, 0, rows, bounds, push_lists, thread_count(n));
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
               std::vector<int> &rows, const std::vector<int> &bounds, bool push_lists, int threads) {
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
        std::vector<char> met(n, 0);
        std::unique_ptr<int[]> halo_slot(new int[n]);  // set for the halo rows only
        // the halo: ascending rows of other parts
        for (int i = 0; i < nown; ++i)
            for (int k = row_ptr[rows[lo + i]]; k < row_ptr[rows[lo + i] + 1]; ++k)
                if (part_of[col_idx[k] - row_lo] != p && !met[col_idx[k] - row_lo]) {
                    met[col_idx[k] - row_lo] = 1;
                    m.halo.push_back(col_idx[k]);
                }
        std::sort(m.halo.begin(), m.halo.end());
        for (size_t i = 0; i < m.halo.size(); ++i) halo_slot[m.halo[i] - row_lo] = (int)i;
        // slices of kPartSliceRows rows, kPartLanes lanes a row; a trip is one
        // block a lane, padded lanes read no block (src -1)
        const int nslices = (nown + kPartSliceRows - 1) / kPartSliceRows;
        int warp_trips[kPartWarps] = {0}, reg_trips[kPartWarps] = {0};
        for (int s = 0; s < nslices; ++s) {
            const int r0 = s * kPartSliceRows, nr = std::min(kPartSliceRows, nown - r0);
            int trips = 0;
            for (int r = 0; r < nr; ++r) {
                const int row = rows[lo + r0 + r];
                trips = std::max(trips, (row_ptr[row + 1] - row_ptr[row] + kPartLanes - 1) / kPartLanes);
            }
            m.trip_ptr.push_back((int32_t)(m.src.size() / 32));
            warp_trips[s % kPartWarps] += trips;
            if (s < kPartWarps) reg_trips[s] = std::min(trips, kPartRegTrips);
            m.slice_trips_max = std::max(m.slice_trips_max, trips);
            const size_t base = m.src.size();
            m.src.resize(base + (size_t)32 * trips, -1);
            m.col.resize(base + (size_t)32 * trips, 0);
            for (int r = 0; r < nr; ++r) {
                const int row = rows[lo + r0 + r], k0 = row_ptr[row], len = row_ptr[row + 1] - k0;
                for (int e = 0; e < len; ++e) {
                    const int c = col_idx[k0 + e];
                    const size_t at = base + (size_t)(e / kPartLanes) * 32 + e % kPartLanes * kPartSliceRows + r;
                    m.src[at] = k0 + e;
                    m.col[at] = (uint16_t)(part_of[c - row_lo] == p
                                               ? local[c - row_lo]
                                               : nown + halo_slot[c - row_lo]);
                }
            }
        }
        m.trip_ptr.push_back((int32_t)(m.src.size() / 32));
        for (int w = 0; w < kPartWarps; ++w) {
            m.trips_max = std::max(m.trips_max, warp_trips[w]);
            m.trips_max_reg = std::max(m.trips_max_reg, warp_trips[w] - reg_trips[w]);
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
    }
}

}  // namespace

void resident_add_bodies(ResidentHost &h, const int32_t *row_ptr, const int32_t *col_idx, const float *rest_q,
                         const int32_t *row_off, const std::vector<int> &bodies, int parts) {
    std::vector<ResidentHost> made(bodies.size());
    int rows = 0;
    for (int b : bodies) rows += row_off[b + 1] - row_off[b];
    parallel_for((int)bodies.size(), thread_count(rows), [&](int i) {
        const int b = bodies[i];
        resident_add_body(made[i], row_ptr, col_idx, rest_q, row_off[b], row_off[b + 1], parts, b, parts > 1, false);
    });
    for (const ResidentHost &m : made) {
        const int first = (int)h.parts.size(), trips = (int)(h.src.size() / 32);
        for (ResPart rp : m.parts) {
            rp.row_off += (int)h.rows.size();
            rp.halo_off += (int)h.halo.size();
            rp.slice_off += (int)h.trip_ptr.size();
            rp.push_off += (int)h.push.size();
            h.parts.push_back(rp);
        }
        for (int4 t : m.tasks) h.tasks.push_back(make_int4(first + t.x, t.y, t.z, t.w));
        h.rows.insert(h.rows.end(), m.rows.begin(), m.rows.end());
        h.halo.insert(h.halo.end(), m.halo.begin(), m.halo.end());
        for (int32_t t : m.trip_ptr) h.trip_ptr.push_back(trips + t);
        h.src.insert(h.src.end(), m.src.begin(), m.src.end());
        h.col.insert(h.col.end(), m.col.begin(), m.col.end());
        h.push.insert(h.push.end(), m.push.begin(), m.push.end());
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
