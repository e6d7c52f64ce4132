// Host program of test_cells_host.py: every population that the INSIDE gather of cell_pairs reads lies in its plane.
//
// An INSIDE cell is read without a look at its nodes: a lane whose first node (number `lane` in FP32, 2 lane in the
// 16-bit storages) is in the cell also reads the second one (32 or 1 further), for every direction at the node's index
// minus the direction's offset. So whatever cell cell_gather calls INSIDE, those indices must lie in [0, nodes).
#include <cstdio>
#include <cstdlib>

#include "cells.cuh"

template <int Q>
int check(int nx, int ny, int nz) {
    using L = wk::Lat<Q>;
    wk::Geo g{};
    g.nx = nx, g.ny = ny, g.nz = nz;
    g.by_nx = wk::FastDiv::of(nx);
    g.by_ny = wk::FastDiv::of(ny);
    const long long nodes = static_cast<long long>(nx) * ny * nz;
    long long low = 0, high = 0;  // smallest and largest offset of a direction
    for (int q = 0; q < Q; ++q) {
        const long long d = L::cx(q) + nx * (L::cy(q) + static_cast<long long>(ny) * L::cz(q));
        low = d < low ? d : low;
        high = d > high ? d : high;
    }
    long long inside = 0;
    for (long long i0 = 0; i0 < nodes; ++i0)
        for (int count = 1; count <= wk::CELL && i0 + count <= nodes; ++count) {
            if (wk::cell_gather<Q>(g, static_cast<unsigned>(i0), count) != wk::INSIDE) continue;
            ++inside;
            for (int storage = 0; storage < 2; ++storage) {
                const int lanes = storage ? (count + 1) / 2 : (count < 32 ? count : 32);
                const long long last = i0 + (storage ? 2 * (lanes - 1) + 1 : lanes - 1 + 32);
                if (i0 - high < 0 || last - low >= nodes) {
                    std::printf("D%dQ%d %d x %d x %d: cell of %d nodes at %lld reads [%lld, %lld] of %lld nodes\n", L::D, Q, nx, ny,
                                nz, count, i0, i0 - high, last - low, nodes);
                    return 1;
                }
            }
        }
    std::printf("D%dQ%d %d x %d x %d: %lld INSIDE cells\n", L::D, Q, nx, ny, nz, inside);
    return 0;
}

int main(int argc, char** argv) {
    if (argc != 5) return 2;
    const int q = std::atoi(argv[1]), nx = std::atoi(argv[2]), ny = std::atoi(argv[3]), nz = std::atoi(argv[4]);
    return q == 9 ? check<9>(nx, ny, nz) : (q == 19 ? check<19>(nx, ny, nz) : check<27>(nx, ny, nz));
}
