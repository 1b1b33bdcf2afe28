// Cell order for compact face tiles (E3D_ORDER_SPATIAL): recursive bisection of the cell graph into
// groups of whole tiles, each cut placed where it crosses few faces.  Host code.
//
// A stage kernel's cost follows its tiles' surfaces: a face between two tiles is evaluated by both,
// its cells are halo records of both, and the largest tile sets every block's shared memory.  A Morton
// order of the cell centres sees coordinates only: on stretched layers (a 256 x 128 x 4 O-grid whose
// wall cells are 800 times longer than high) its 128-cell runs are long strips.  Per cell, faces
// evaluated / halo records / largest tile, Morton against this order:
//   O-grid 256 x 128 x 4   3.73 / 1.75 / 50.9 KB    3.10 / 0.57 / 35.1 KB   (2.75 faces per cell)
//   channel 193 x 97 x 2   4.05 / 0.89 / 38.7 KB    3.82 / 0.49 / 31.3 KB   (3.52)
//   tetrahedra 65x63x61x6  2.65 / 0.97 / 30.4 KB    2.51 / 0.76 / 28.0 KB   (2.02)
// FP64 stage: the O-grid's 35.3 -> 27.1 us, with the growing below an iteration of its 106.5 -> 97.2 us.
#pragma once
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdint>
#include <future>
#include <numeric>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace e3d {

// Bisects parts of k tiles into floor(k / 2) tiles and the rest, down to single tiles.  A cut is a plane
// whose normal comes from a few candidates: the coordinate axes and the normals of some of the part's
// own faces, which follow the grid lines of curved and stretched layers.  With d the vector between the
// centres of a face's two cells, a plane of normal n crosses sum |d . n| / (extent of the part along n)
// of its faces on average; the candidates that promise least are tried and the one that cuts the
// fewest faces is kept.  Parts above kCoarse cells take the estimate's word (a tile's shape is decided
// by the last few cuts).
struct TileBisector {
    static constexpr int kDirs = 16, kCoarse = 1 << 17, kParallel = 1 << 12, kSample = 1 << 10, kGrow = 1 << 17;
    const double *centre;               // 3 per cell
    const int *adj_ptr, *adj, *adj_face;  // interior neighbours of each cell and the faces between
    const double *unit_normal;          // 3 per face
    int tile;
    std::atomic<int> *side;             // per cell: the part it was last put in
    std::atomic<int> *parts;            // parts numbered so far
    std::vector<std::pair<double, int>> key, keep;
    std::vector<int> queue;

    int mark() { return parts->fetch_add(1, std::memory_order_relaxed) + 1; }

    // Faces between the first `left` and the other cells of the order at(0), ..., at(n - 1).
    template <typename AT>
    int cut_faces(int n, int left, AT &&at) {
        const int right_part = mark();
        for (int i = left; i < n; i++) side[at(i)].store(right_part, std::memory_order_relaxed);
        int cut = 0;
        for (int i = 0; i < left; i++) {
            const int c = at(i);
            for (int k = adj_ptr[c]; k < adj_ptr[c + 1]; k++) cut += side[adj[k]].load(std::memory_order_relaxed) == right_part;
        }
        return cut;
    }

    // The part's cells breadth first into `queue`: from the first cell, or where the queue holds an
    // order already, from that order's last one (an end of the part).  Pieces not reached follow.
    void grow(const int *cells, int n) {
        const int inside = mark(), seen = mark();
        const int start = (int)queue.size() == n ? queue[n - 1] : cells[0];
        for (int i = 0; i < n; i++) side[cells[i]].store(inside, std::memory_order_relaxed);
        queue.clear();
        int next = 0;
        auto push = [&](int c) {
            side[c].store(seen, std::memory_order_relaxed);
            queue.push_back(c);
        };
        push(start);
        for (size_t head = 0; (int)queue.size() < n || head < queue.size(); head++) {
            if (head == queue.size()) {  // another piece
                while (side[cells[next]].load(std::memory_order_relaxed) != inside) next++;
                push(cells[next]);
            }
            const int c = queue[head];
            for (int k = adj_ptr[c]; k < adj_ptr[c + 1]; k++)
                if (side[adj[k]].load(std::memory_order_relaxed) == inside) push(adj[k]);
        }
    }

    void split(int *cells, int n, int depth) {
        if (n <= tile) {
            std::sort(cells, cells + n);  // neighbouring ids together: state transfers stay coalesced
            return;
        }
        const int tiles = (n + tile - 1) / tile, left = (tiles / 2) * tile;
        const bool coarse = n > kCoarse;
        double dir[kDirs][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
        int nd = 3;
        for (int s = 0; s < 6; s++) {  // faces of six cells spread over the part
            const int c = cells[(int)((2 * s + 1) * (int64_t)n / 12)];
            for (int k = adj_ptr[c]; k < adj_ptr[c + 1] && nd < kDirs; k++) {
                const double *u = unit_normal + 3 * (size_t)adj_face[k];
                const double len2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
                bool known = !(len2 > 0.25 && len2 < 4.0);  // a degenerate face (its normal may be NaN)
                for (int q = 0; q < nd && !known; q++)
                    known = std::fabs(u[0] * dir[q][0] + u[1] * dir[q][1] + u[2] * dir[q][2]) > 0.97;
                if (known) continue;
                for (int q = 0; q < 3; q++) dir[nd][q] = u[q];
                nd++;
            }
        }
        double lo[kDirs], hi[kDirs], cost[kDirs] = {};
        std::fill(lo, lo + nd, 1e300);
        std::fill(hi, hi + nd, -1e300);
        const int stride = std::max(1, n / kSample);  // a sample of a large part is enough
        for (int i = 0; i < n; i += stride) {
            const int c = cells[i];
            const double *x = centre + 3 * (size_t)c;
            for (int q = 0; q < nd; q++) {
                const double v = x[0] * dir[q][0] + x[1] * dir[q][1] + x[2] * dir[q][2];
                lo[q] = std::min(lo[q], v);
                hi[q] = std::max(hi[q], v);
            }
            for (int k = adj_ptr[c]; k < adj_ptr[c + 1]; k++) {
                const double *y = centre + 3 * (size_t)adj[k];
                const double d[3] = {y[0] - x[0], y[1] - x[1], y[2] - x[2]};
                for (int q = 0; q < nd; q++) cost[q] += std::fabs(d[0] * dir[q][0] + d[1] * dir[q][1] + d[2] * dir[q][2]);
            }
        }
        // no plane cuts across a direction in which the part is flat but for rounding: a mesh one layer thick
        // has one, whose cost of almost nothing over almost nothing would rank anywhere
        double size = 1e-300;
        for (int q = 0; q < nd; q++) size = std::max({size, std::fabs(lo[q]), std::fabs(hi[q]), hi[q] - lo[q]});
        int rank[kDirs];
        for (int q = 0; q < nd; q++) {
            rank[q] = q;
            cost[q] = hi[q] - lo[q] > 1e-13 * size ? cost[q] / (hi[q] - lo[q]) : HUGE_VAL;
        }
        int tries = std::min(nd, coarse ? 1 : n > 16 * tile ? 2 : 4);
        std::partial_sort(rank, rank + tries, rank + nd,
                          [&](int a, int b) { return cost[a] < cost[b] || (cost[a] == cost[b] && a < b); });
        while (tries > 1 && cost[rank[tries - 1]] > 1.6 * cost[rank[0]]) tries--;
        int best = INT_MAX;
        for (int t = 0; t < tries; t++) {
            const double *u = dir[rank[t]];
            key.resize(n);
            for (int i = 0; i < n; i++) {
                const double *x = centre + 3 * (size_t)cells[i];
                key[i] = {x[0] * u[0] + x[1] * u[1] + x[2] * u[2], cells[i]};
            }
            std::nth_element(key.begin(), key.begin() + left, key.end());
            if (tries == 1 && (coarse || n > kGrow)) {
                keep.swap(key);
                break;
            }
            const int cut = cut_faces(n, left, [&](int i) { return key[i].second; });
            if (cut < best) {
                best = cut;
                keep.swap(key);
            }
        }
        // No plane separates layers much thinner than the wall's curvature bends them: a part cut through
        // many more faces than a compact one would be is also grown breadth first, from one of its ends.
        if (!coarse && n <= kGrow && best > std::cbrt((double)n * n)) {
            queue.clear();
            grow(cells, n);
            grow(cells, n);
            const int cut = cut_faces(n, left, [&](int i) { return queue[i]; });
            if (cut < best) {
                for (int i = 0; i < n; i++) cells[i] = queue[i];
            } else {
                for (int i = 0; i < n; i++) cells[i] = keep[i].second;
            }
        } else {
            for (int i = 0; i < n; i++) cells[i] = keep[i].second;
        }
        if (n > kParallel && depth > 0) {  // the halves in two threads, this one with its own buffers
            TileBisector other{centre, adj_ptr, adj, adj_face, unit_normal, tile, side, parts, {}, {}, {}};
            std::future<void> half;  // passes on what the other thread throws; waits on every exit
            try {
                half = std::async(std::launch::async, [&] { other.split(cells, left, depth - 1); });
            } catch (const std::system_error &) {  // no more threads
                other.split(cells, left, 0);
            }
            split(cells + left, n - left, depth - 1);
            if (half.valid()) half.get();
        } else {
            split(cells, left, 0);
            split(cells + left, n - left, 0);
        }
    }
};

// The cells of a mesh in compact tiles: position -> cell.  face2cell: 2 per face, the first n_int
// interior; centre: 3 finite numbers per cell; unit_normal: 3 per face.
inline std::vector<int> compact_tile_order(int n_cells, int n_int, const int32_t *face2cell, const double *unit_normal,
                                           const std::vector<double> &centre, int tile) {
    std::vector<int> ptr(n_cells + 1, 0), adj(2 * (size_t)n_int), face(2 * (size_t)n_int), order(n_cells);
    for (int64_t f = 0; f < 2 * (int64_t)n_int; f++) ptr[face2cell[f] + 1]++;
    for (int c = 0; c < n_cells; c++) ptr[c + 1] += ptr[c];
    std::vector<int> at(ptr.begin(), ptr.end() - 1);
    for (int f = 0; f < n_int; f++) {
        const int l = face2cell[2 * (size_t)f], r = face2cell[2 * (size_t)f + 1];
        adj[at[l]] = r;
        face[at[l]++] = f;
        adj[at[r]] = l;
        face[at[r]++] = f;
    }
    std::iota(order.begin(), order.end(), 0);
    std::vector<std::atomic<int>> side(n_cells);
    std::atomic<int> parts{0};
    int depth = 0;
    for (unsigned t = std::thread::hardware_concurrency(); t > 1; t /= 2) depth++;
    TileBisector{centre.data(), ptr.data(), adj.data(), face.data(), unit_normal, tile, side.data(), &parts, {}, {}, {}}.split(
        order.data(), n_cells, depth);
    return order;
}

}  // namespace e3d
