// The spatial hash's integer arithmetic and the rule by which a group of a warp's particles walks the
// union of its neighbour cells as one tile: plain functions of integers, for the kernels and for the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define VFS_HD __host__ __device__ __forceinline__
#else
#define VFS_HD inline
#endif

namespace vfs {

// HashCell3D, assets/shaders/simulation/spatial_hash/spatial_hash_3d.slang:20-28.
VFS_HD uint32_t hash_cell(uint32_t cx, uint32_t cy, uint32_t cz) {
    const uint32_t ux = cx + 25u, uy = cy + 25u, uz = cz + 25u;
    const uint32_t lx = ux % 50u, ly = uy % 50u, lz = uz % 50u;
    const uint32_t bx = ux / 50u, by = uy / 50u, bz = uz / 50u;
    const uint32_t block_hash = bx * 15823u + by * 9737333u + bz * 440817757u;
    return lx + 50u * (ly + 50u * lz) + block_hash;
}

// KeyFromHash (spatial_hash_3d.slang:30-32): hash % n, computed as the high word of
// (magic * hash mod 2^64) * n with magic = ceil(2^64 / n) (exact for 32-bit operands).
VFS_HD uint32_t key_mod(uint32_t hash, uint64_t magic, uint32_t n) {
    const uint64_t low = magic * (uint64_t)hash;
#ifdef __CUDA_ARCH__
    return (uint32_t)__umul64hi(low, (uint64_t)n);
#else
    return (uint32_t)(((unsigned __int128)low * n) >> 64);
#endif
}

// A tile's rows of `width` cells from xa: how many of them lie in the hash block of the first. False
// when they span three blocks (the short block at the 2^32 wrap of the cells).
VFS_HD bool tile_first_cells(uint32_t xa, uint32_t width, uint32_t& n_first) {
    const uint32_t block_a = (xa + 25u) / 50u, block_b = (xa + width + 24u) / 50u;
    n_first = width;
    if (block_a != block_b) {
        n_first = 1u;
        while ((xa + n_first + 25u) / 50u == block_a) n_first++;
        if ((xa + n_first + 25u) / 50u != block_b) return false;
    }
    return true;
}

// One row's cells as runs of consecutive keys below n, in visiting order: one run, or two when the row
// crosses a hash block along x or its keys pass n - 1. ok: that is all there is to it (no hash wraps).
struct TileRow {
    uint32_t k0, l0, k1, l1;
    bool ok;
};
VFS_HD TileRow tile_row(uint32_t xa, uint32_t y, uint32_t z, uint32_t width, uint32_t n_first, uint32_t n,
                        uint64_t magic) {
    const uint32_t hash = hash_cell(xa, y, z);
    TileRow r{key_mod(hash, magic, n), n_first, 0u, 0u, hash <= 0xFFFFFFFFu - n_first};
    if (n_first != width) {
        const uint32_t hash1 = hash_cell(xa + n_first, y, z);
        r.k1 = key_mod(hash1, magic, n);
        r.l1 = width - n_first;
        r.ok = r.ok && hash1 <= 0xFFFFFFFFu - r.l1 && r.k0 + r.l0 <= n && r.k1 + r.l1 <= n;
    } else if (r.k0 + r.l0 > n) {
        r.l1 = r.k0 + r.l0 - n;  // continues at key 0
        r.l0 -= r.l1;
        r.ok = r.ok && r.l1 <= n;
    }
    return r;
}

// Runs [ka, ka + la) and [kb, kb + lb) modulo n share no key.
VFS_HD bool runs_apart(uint32_t ka, uint32_t la, uint32_t kb, uint32_t lb, uint32_t n) {
    const uint32_t up = kb >= ka ? kb - ka : kb + (n - ka), dn = ka >= kb ? ka - kb : ka + (n - kb);
    return la == 0u || lb == 0u || (up >= la && dn >= lb);
}

}  // namespace vfs
