// Groups of 1 to 6 cells of a row and their 3 x 3 or 5 x 5 rows of neighbour cells, from standard input
// (reach, n, c0, c1, cy, cz per line): whether the tile rule takes the union, and, from every cell's own
// key, whether the keys are distinct and the rule's runs name the same keys in the same order.
#include <cinttypes>
#include <cstdio>
#include <set>
#include <vector>

#include "vfs_tile_rule.h"

int main() {
    uint32_t reach, n, c0, c1, cy, cz;
    while (std::scanf("%" SCNu32 " %" SCNu32 " %" SCNu32 " %" SCNu32 " %" SCNu32 " %" SCNu32, &reach, &n, &c0, &c1, &cy, &cz) == 6) {
        const uint64_t magic = UINT64_MAX / n + 1ull;
        const uint32_t side = 2u * reach + 1u, xa = c0 - reach, width = c1 - c0 + 1u + 2u * reach;
        std::vector<uint32_t> own, runs;
        std::vector<vfs::TileRow> rows;
        uint32_t n_first = 0u;
        bool taken = vfs::tile_first_cells(xa, width, n_first);
        for (uint32_t r = 0; r < side * side; r++) {
            const uint32_t y = cy + r % side - reach, z = cz + r / side - reach;
            for (uint32_t x = 0; x < width; x++) own.push_back(vfs::hash_cell(xa + x, y, z) % n);
            if (!taken) continue;
            const vfs::TileRow t = vfs::tile_row(xa, y, z, width, n_first, n, magic);
            for (uint32_t k = 0; k < t.l0; k++) runs.push_back(t.k0 + k);
            for (uint32_t k = 0; k < t.l1; k++) runs.push_back(t.k1 + k);
            taken = t.ok && vfs::runs_apart(t.k0, t.l0, t.k1, t.l1, n);
            for (const vfs::TileRow& q : rows)
                taken = taken && vfs::runs_apart(t.k0, t.l0, q.k0, q.l0, n) && vfs::runs_apart(t.k0, t.l0, q.k1, q.l1, n) &&
                        vfs::runs_apart(t.k1, t.l1, q.k0, q.l0, n) && vfs::runs_apart(t.k1, t.l1, q.k1, q.l1, n);
            rows.push_back(t);
        }
        const bool distinct = std::set<uint32_t>(own.begin(), own.end()).size() == own.size();
        std::printf("%d %d %d\n", taken, distinct, taken && runs == own);
    }
}
