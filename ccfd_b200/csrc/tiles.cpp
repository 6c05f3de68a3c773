// Orderings of the cells and construction of the flux kernel's tiles (see
// tiles.h).
#include "tiles.h"

#include <algorithm>
#include <cmath>
#include <stdint.h>
#include <thread>

// Hilbert index of (x, y) on a 2^16 x 2^16 grid (the classical iterative
// quadrant-rotation construction).
static uint64_t hilbert_index(uint32_t x, uint32_t y) {
    const uint32_t n = 1u << 16;
    uint64_t d = 0;
    for (uint32_t s = n / 2; s > 0; s /= 2) {
        uint32_t rx = (x & s) ? 1u : 0u;
        uint32_t ry = (y & s) ? 1u : 0u;
        d += (uint64_t)s * s * ((3u * rx) ^ ry);
        if (ry == 0) {
            if (rx == 1) {
                x = n - 1 - x;
                y = n - 1 - y;
            }
            std::swap(x, y);
        }
    }
    return d;
}

void ccfd_hilbert_order(const ccfd_mesh* m, std::vector<int>& cell_order) {
    const long N = m->n_cells;
    double x0 = m->cell_bary[0], x1 = x0, y0 = m->cell_bary[1], y1 = y0;
    for (long c = 0; c < N; ++c) {
        x0 = std::min(x0, m->cell_bary[2 * c]);
        x1 = std::max(x1, m->cell_bary[2 * c]);
        y0 = std::min(y0, m->cell_bary[2 * c + 1]);
        y1 = std::max(y1, m->cell_bary[2 * c + 1]);
    }
    // square bounding box so that tiles stay compact on elongated domains
    double span = std::max(x1 - x0, y1 - y0);
    if (span <= 0) span = 1.0;
    std::vector<uint64_t> key(N);
    auto keys = [&](long a, long b) {
        for (long c = a; c < b; ++c) {
            double fx = (m->cell_bary[2 * c] - x0) / span, fy = (m->cell_bary[2 * c + 1] - y0) / span;
            uint32_t ix = (uint32_t)std::min(65535.0, std::max(0.0, fx * 65535.0));
            uint32_t iy = (uint32_t)std::min(65535.0, std::max(0.0, fy * 65535.0));
            key[c] = hilbert_index(ix, iy);
        }
    };
    {
        unsigned hw = std::thread::hardware_concurrency();
        long nth = std::max(1L, std::min<long>(hw ? hw : 1, std::min(16L, N / 65536)));
        std::vector<std::thread> pool;
        for (long k = 0; k + 1 < nth; ++k) pool.emplace_back(keys, N * k / nth, N * (k + 1) / nth);
        keys(N * (nth - 1) / nth, N);
        for (std::thread& th : pool) th.join();
    }
    // stable sort of the cells by key (the key is below 2^32): LSD radix
    // sort, four passes of 8 bits
    std::vector<int> a(N), b(N);
    for (long c = 0; c < N; ++c) a[c] = (int)c;
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 8 * pass;
        size_t cnt[257] = {0};
        for (long i = 0; i < N; ++i) ++cnt[((key[a[i]] >> shift) & 255u) + 1];
        for (int k = 0; k < 256; ++k) cnt[k + 1] += cnt[k];
        for (long i = 0; i < N; ++i) b[cnt[(key[a[i]] >> shift) & 255u]++] = a[i];
        a.swap(b);
    }
    cell_order.swap(a);
}

// Reverse Cuthill-McKee ordering of the cell graph (face neighbours):
// breadth-first levels from a cell of least degree (per connected
// component), neighbours in order of increasing degree, the whole order
// reversed (Cuthill and McKee 1969, George 1971).
void ccfd_rcm_order(const ccfd_mesh* m, std::vector<int>& cell_order) {
    const long N = m->n_cells;
    std::vector<int> deg(N), order;
    order.reserve(N);
    for (long c = 0; c < N; ++c) {
        int d = 0;
        for (long h = m->hs_offset[c]; h < m->hs_offset[c + 1]; ++h) d += m->hs_nb[h] >= 0;
        deg[c] = d;
    }
    std::vector<char> seen(N, 0);
    std::vector<int> by_deg(N), nb;
    for (long c = 0; c < N; ++c) by_deg[c] = (int)c;
    std::stable_sort(by_deg.begin(), by_deg.end(), [&](int a, int b) { return deg[a] < deg[b]; });
    for (int start : by_deg) {
        if (seen[start]) continue;
        seen[start] = 1;
        size_t head = order.size();
        order.push_back(start);
        while (head < order.size()) {
            const int c = order[head++];
            nb.clear();
            for (long h = m->hs_offset[c]; h < m->hs_offset[c + 1]; ++h) {
                const long e = m->hs_nb[h];
                if (e >= 0 && !seen[e]) {
                    seen[e] = 1;
                    nb.push_back((int)e);
                }
            }
            std::stable_sort(nb.begin(), nb.end(), [&](int a, int b) { return deg[a] < deg[b]; });
            order.insert(order.end(), nb.begin(), nb.end());
        }
    }
    cell_order.assign(order.rbegin(), order.rend());
}

// Host work split into ranges of tiles, one thread each; every range writes
// to its own entries, so the result does not depend on the thread count.
template <typename Fn>
static void tile_ranges(int n_tiles, Fn fn) {
    const unsigned hw = std::thread::hardware_concurrency();
    const int nth = std::max(1, std::min((int)std::min(hw ? hw : 1u, 16u), n_tiles / 64));
    std::vector<std::thread> pool;
    for (int k = 0; k + 1 < nth; ++k)
        pool.emplace_back(fn, (int)((long)n_tiles * k / nth), (int)((long)n_tiles * (k + 1) / nth));
    fn((int)((long)n_tiles * (nth - 1) / nth), n_tiles);
    for (std::thread& th : pool) th.join();
}

void ccfd_build_tiles(const ccfd_mesh* m, const std::vector<int>& cperm, const std::vector<int>& cinv, int T,
                      TileSet& ts) {
    const long N = m->n_cells, F = m->n_faces;
    // (the vectors keep their capacity from an earlier call)
    ts.tile_cells = T;
    ts.n_tiles = (int)((N + T - 1) / T);
    ts.own_off.assign(ts.n_tiles + 1, 0);
    ts.border_off.assign(ts.n_tiles + 1, 0);
    ts.face_of.resize(F);
    ts.id_of.resize(F);
    ts.u_code.resize(4 * (size_t)N);
    // A side's face is new to the tile when this is the face's first side in
    // device order within the tile: the other side's cell is in another tile
    // or later (or the same cell's later side, on a periodic mesh); it is the
    // tile's own when the other side's cell is not in an earlier tile.
    auto classify = [&](long d, long h, long d0, long* f) {
        *f = m->hs_face[h];
        const long nb = m->hs_nb[h];
        if (nb < 0) return 1;
        const long e = cinv[nb];
        if (e < d0) return 2;                          // border: owned by an earlier tile
        if (e >= d0 + T || e > d) return 1;            // own, first seen here
        if (e == d) {                                  // a cell that is its own neighbour: the first of its sides
            const long s0 = m->face_hs[2 * *f], s1 = m->face_hs[2 * *f + 1];
            return h == std::min(s0, s1) ? 1 : 0;
        }
        return 0;                                      // already seen in this tile
    };
    tile_ranges(ts.n_tiles, [&](int ta, int tb) {
        for (int t = ta; t < tb; ++t) {
            const long d0 = (long)t * T, d1 = std::min(N, d0 + T);
            int own = 0, border = 0;
            for (long d = d0; d < d1; ++d)
                for (long h = m->hs_offset[cperm[d]]; h < m->hs_offset[cperm[d] + 1]; ++h) {
                    long f;
                    const int c = classify(d, h, d0, &f);
                    own += c == 1;
                    border += c == 2;
                }
            ts.own_off[t + 1] = own;
            ts.border_off[t + 1] = border;
        }
    });
    ts.max_f = 0;
    for (int t = 0; t < ts.n_tiles; ++t) {
        ts.max_f = std::max(ts.max_f, ts.own_off[t + 1] + ts.border_off[t + 1]);
        ts.own_off[t + 1] += ts.own_off[t];
        ts.border_off[t + 1] += ts.border_off[t];
    }
    ts.border.resize(ts.border_off[ts.n_tiles]);
    tile_ranges(ts.n_tiles, [&](int ta, int tb) {
        for (int t = ta; t < tb; ++t) {
            const long d0 = (long)t * T, d1 = std::min(N, d0 + T);
            int id = ts.own_off[t];
            for (long d = d0; d < d1; ++d)
                for (long h = m->hs_offset[cperm[d]]; h < m->hs_offset[cperm[d] + 1]; ++h) {
                    long f;
                    if (classify(d, h, d0, &f) == 1) {
                        ts.face_of[id] = (int)f;
                        ts.id_of[f] = id++;
                    }
                }
        }
    });
    tile_ranges(ts.n_tiles, [&](int ta, int tb) {
        for (int t = ta; t < tb; ++t) {
            const long d0 = (long)t * T, d1 = std::min(N, d0 + T);
            const int own0 = ts.own_off[t], n_own = ts.own_off[t + 1] - own0;
            int nb = ts.border_off[t];
            for (long d = d0; d < d1; ++d) {
                uint16_t* code = &ts.u_code[4 * (size_t)d];
                int k = 0;
                for (long h = m->hs_offset[cperm[d]]; h < m->hs_offset[cperm[d] + 1]; ++h, ++k) {
                    long f;
                    int local;
                    if (classify(d, h, d0, &f) == 2) {
                        local = n_own + (nb - ts.border_off[t]);
                        ts.border[nb++] = ts.id_of[f];
                    } else {
                        local = ts.id_of[f] - own0;
                    }
                    code[k] = (uint16_t)(2 * local + (m->hs_sign[h] > 0 ? 0 : 1));
                }
                for (; k < 4; ++k) code[k] = 0xffff;
            }
        }
    });
}
