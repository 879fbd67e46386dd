// sm_103a kernels of one WCSPH-with-boundary substep (VkFluidSim's
// WCSPHWithBoundaryModel::Step, src/models/wcsph_with_boundary_model.cpp:81-117):
//
//   k_keys_flags      key[i] = HashCell3D(floor(x_i / h)) % N, moved flags, digit histograms
//   k_onesweep        stable LSD radix pass of (key, index) with decoupled look-back
//   k_cells_reorder   cell_scan[] (lower bound of every key) + gather of x, v (and ids in x.w)
//   k_density_list    volume-map boundary terms + density + Tait EOS epilogue over the skin lists
//                     (k_skin_build builds them; k_walk_queue and k_walk walk what has none)
//   k_force           pressure + viscosity + wall penalty + symplectic Euler
//
// Data layout: particle state is float4 SoA (x,y,z,id-bits) and (vx,vy,vz,0) in sorted order;
// per-particle density products aux = (p/rho^2, m/max(rho,1e-6), rho, p/rho0^2); boundary
// bnd = (grad Psi_b, Psi_b). All arrays are 16-byte aligned and read with 128-bit loads.
//
// The neighbour loops visit exactly the reference's candidate multiset in the reference's order:
// for each (dy, dz) the keys of cells (cx-1..cx+1) are usually consecutive (HashCell3D is
// x-linear inside a 50-cell block), and consecutive keys' buckets are adjacent in the sorted
// array, so the three buckets are one contiguous range [scan[kA], scan[kA+3]). When the three
// keys are not consecutive, each bucket is walked on its own. Duplicate keys among the 27 are
// walked as often as they occur, like wcsph_with_boundary_model.slang:166-190.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>
#include <atomic>

#include "vfs_chain.h"
#include "vfs_internal.h"
#include "vfs_tile_rule.h"

namespace vfs {
namespace {

// ---------------------------------------------------------------- hashing

// GetCell3D (spatial_hash_3d.slang:16-18): IEEE division, floor, saturating conversion.
__device__ __forceinline__ uint32_t cell_coord(float x, float h) {
    return (uint32_t)__float2int_rz(floorf(__fdiv_rn(x, h)));
}

// ---------------------------------------------------------------- SPH kernel

// CubicSpline (kernels_3d.slang:62-76) at q = r / h.
__device__ __forceinline__ float cubic_w(float q, float sigma) {
    if (q <= 1.0f) {
        if (q > 0.5f) {
            const float t = 1.0f - q;
            return sigma * 2.0f * (t * t * t);
        }
        const float q2 = q * q;
        const float q3 = q2 * q;
        return sigma * (6.0f * q3 - 6.0f * q2 + 1.0f);
    }
    return 0.0f;
}

// GradCubicSpline (kernels_3d.slang:78-91); sigma already carries the extra 1/h.
__device__ __forceinline__ float cubic_dw(float r, float q, float sigma) {
    if ((r > 1e-9f) && (q <= 1.0f)) {
        if (q > 0.5f) {
            const float t = 1.0f - q;
            return -sigma * (t * t);
        }
        return sigma * q * (3.0f * q - 2.0f);
    }
    return 0.0f;
}

// ---------------------------------------------------------------- volume-map sampling
// Written with round-to-nearest intrinsics, which the compiler never fuses, so the thresholds
// of CalculateBoundaryVolume (inside-box, 0 <= dist < h, volume > 0) evaluate bit-identically
// to an unfused IEEE restatement.

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsb(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdv(float a, float b) { return __fdiv_rn(a, b); }

// One axis of SampleGrid with the cell index clamped to [0, n-2] (linear extrapolation outside;
// the reference reads out of bounds there, wcsph_with_boundary_model.slang:51-66).
__device__ __forceinline__ void grid_axis(uint32_t n, float u, uint32_t& cell, float& chi) {
    const float x = fm(fsb((float)n, 1.0f), u);
    float f = floorf(x);
    const float hi = (float)(n - 2u);
    if (!(f >= 0.0f)) f = 0.0f;
    if (f > hi) f = hi;
    cell = (uint32_t)f;
    chi = fsb(fm(2.0f, fsb(x, f)), 1.0f);
}

// A point of a grid in SampleGrid's terms: per axis the clamped cell and chi = 2 frac - 1.
struct GridPoint {
    uint32_t cell[3];
    float chi[3];
};

// Index of a point's base corner (its cell's lowest corner) in the grid array.
__device__ __forceinline__ size_t grid_base(const uint32_t* n, const GridPoint& g) {
    return g.cell[0] + (size_t)n[0] * g.cell[1] + (size_t)n[0] * n[1] * g.cell[2];
}

// The 8 corner values of a point's cell, in the shader's offsets[8] order:
// (0,0,0) (0,1,0) (0,0,1) (0,1,1) (1,0,0) ...
__device__ __forceinline__ void grid_corners(const float* __restrict__ g, const uint32_t* n,
                                             const GridPoint& p, float c[8]) {
    const size_t b = grid_base(n, p), sy = n[0], sz = (size_t)n[0] * n[1];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int ox = i >> 2, oy = i & 1, oz = (i >> 1) & 1;
        c[i] = __ldg(g + b + ox + oy * sy + oz * sz);
    }
}

// SampleGrid's weighted sum over the corner values (wcsph_with_boundary_model.slang:51-66).
__device__ __forceinline__ float grid_interp(const float c[8], const GridPoint& p) {
    float val = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int ox = i >> 2, oy = i & 1, oz = (i >> 1) & 1;
        const float fx = fa(1.0f, fm(ox ? 1.0f : -1.0f, p.chi[0]));
        const float fy = fa(1.0f, fm(oy ? 1.0f : -1.0f, p.chi[1]));
        const float fz = fa(1.0f, fm(oz ? 1.0f : -1.0f, p.chi[2]));
        val = fa(val, fm(c[i], fm(fm(fx, fy), fz)));
    }
    return fdv(val, 8.0f);
}

// SampleGrid at normalised coordinates (u, v, w).
__device__ __forceinline__ float sample_grid(const float* __restrict__ g, const uint32_t* n,
                                             float u, float v, float w) {
    GridPoint p;
    grid_axis(n[0], u, p.cell[0], p.chi[0]);
    grid_axis(n[1], v, p.cell[1], p.chi[1]);
    grid_axis(n[2], w, p.cell[2], p.chi[2]);
    float c[8];
    grid_corners(g, n, p, c);
    return grid_interp(c, p);
}

__device__ __forceinline__ void to_uvw(const DevObject& o, float x, float y, float z, float& u,
                                       float& v, float& w) {
    u = fdv(fsb(x, o.box_pos[0]), o.box_size[0]);
    v = fdv(fsb(y, o.box_pos[1]), o.box_size[1]);
    w = fdv(fsb(z, o.box_pos[2]), o.box_size[2]);
}

// Row r of a row-major 3x4 matrix applied to (x, y, z, 1), summed left to right.
__device__ __forceinline__ float mat_row(const float* M, int r, float x, float y, float z) {
    return fa(fa(fa(fm(M[4 * r], x), fm(M[4 * r + 1], y)), fm(M[4 * r + 2], z)), M[4 * r + 3]);
}

// CalculateBoundaryVolume for one particle (wcsph_with_boundary_model.slang:102-151).
__device__ __forceinline__ void boundary_terms(const SceneParams& p, float px, float py, float pz,
                                               float& bd, float& bgx, float& bgy, float& bgz) {
    bd = 0.0f;
    bgx = bgy = bgz = 0.0f;
    for (uint32_t oi = 0; oi < p.n_objects; oi++) {
        const DevObject& o = p.objects[oi];
        const float lx = mat_row(o.T, 0, px, py, pz);
        const float ly = mat_row(o.T, 1, px, py, pz);
        const float lz = mat_row(o.T, 2, px, py, pz);
        const bool outside = lx < o.box_pos[0] || ly < o.box_pos[1] || lz < o.box_pos[2] ||
                             lx > fa(o.box_pos[0], o.box_size[0]) ||
                             ly > fa(o.box_pos[1], o.box_size[1]) ||
                             lz > fa(o.box_pos[2], o.box_size[2]);
        if (outside) continue;
        float u, v, w;
        to_uvw(o, lx, ly, lz, u, v, w);
        GridPoint g0;
        grid_axis(o.res[0], u, g0.cell[0], g0.chi[0]);
        grid_axis(o.res[1], v, g0.cell[1], g0.chi[1]);
        grid_axis(o.res[2], w, g0.cell[2], g0.chi[2]);
        float c0[8];
        grid_corners(o.sdf, o.res, g0, c0);
        const float dist = grid_interp(c0, g0);
        if (!(dist >= 0.0f && dist < p.h)) continue;
        const float volume = sample_grid(o.vm, o.res, u, v, w);
        if (!(volume > 0.0f)) continue;
        // GradientVector (slang:68-85): central differences of the SDF at +-0.1 h. A sample
        // moved along one axis shares the other two axes' coordinates with the centre (the same
        // operations on the same inputs), and the centre's corner values while it stays in the
        // centre's cell; the sums are formed exactly as SampleGrid forms them.
        const float e = p.grad_eps;
        const float lc[3] = {lx, ly, lz};
        float grad[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            float s2[2];
#pragma unroll
            for (int sgn = 0; sgn < 2; sgn++) {
                const float la = sgn == 0 ? fa(lc[a], e) : fsb(lc[a], e);
                GridPoint g = g0;
                grid_axis(o.res[a], fdv(fsb(la, o.box_pos[a]), o.box_size[a]), g.cell[a], g.chi[a]);
                if (g.cell[a] == g0.cell[a]) {
                    s2[sgn] = grid_interp(c0, g);
                } else {
                    float c[8];
                    grid_corners(o.sdf, o.res, g, c);
                    s2[sgn] = grid_interp(c, g);
                }
            }
            grad[a] = fdv(fsb(s2[0], s2[1]), fm(2.0f, e));
        }
        const float gx = grad[0], gy = grad[1], gz = grad[2];
        const float modn = __fsqrt_rn(fa(fa(fm(gx, gx), fm(gy, gy)), fm(gz, gz)));
        if (!(modn > 1e-9f)) continue;
        float nx = mat_row(o.R, 0, gx, gy, gz);
        float ny = mat_row(o.R, 1, gx, gy, gz);
        float nz = mat_row(o.R, 2, gx, gy, gz);
        nx = fdv(nx, modn);
        ny = fdv(ny, modn);
        nz = fdv(nz, modn);
        const float d = fmaxf(fa(dist, p.bnd_eighth), p.bnd_half);
        const float xbx = fsb(px, fm(d, nx)), xby = fsb(py, fm(d, ny)), xbz = fsb(pz, fm(d, nz));
        const float xx = fsb(px, xbx), xy = fsb(py, xby), xz = fsb(pz, xbz);
        const float r = __fsqrt_rn(fa(fa(fm(xx, xx), fm(xy, xy)), fm(xz, xz)));
        float ux = 0.0f, uy = 0.0f, uz = 0.0f;
        if (r > 0.0f) {
            ux = fdv(xx, r);
            uy = fdv(xy, r);
            uz = fdv(xz, r);
        }
        const float q = fdv(r, p.h);
        bd = fa(bd, fm(volume, cubic_w(q, p.cubic)));
        const float s = fm(volume, cubic_dw(r, q, p.grad_over_h));
        bgx = fa(bgx, fm(s, ux));
        bgy = fa(bgy, fm(s, uy));
        bgz = fa(bgz, fm(s, uz));
    }
}

// ---------------------------------------------------------------- neighbour ranges

// ---------------------------------------------------------------- scenes

// Parameters of the scene owning particle i: the inline scene of a single-scene launch, or the
// scene-table entry of a batched one.
template <bool kBatch>
__device__ __forceinline__ const SceneParams& scene_params(const StepLaunch& L, uint32_t i) {
    if constexpr (kBatch)
        return L.scenes[__ldg(L.scene_of + i)];
    else
        return L.one;
}

// ---------------------------------------------------------------- kernels


// Per-pass digit histograms of caller-provided keys (the histogram half of k_keys).
__global__ void __launch_bounds__(256) k_digit_hist(const uint32_t* __restrict__ keys, uint32_t n,
                                                    int passes, int digit_bits,
                                                    uint32_t* __restrict__ ghist) {
    __shared__ uint32_t s_h[kMaxSortPasses * kMaxSortBins];
    const int bins = 1 << digit_bits;
    const uint32_t mask = (uint32_t)bins - 1u;
    for (int e = threadIdx.x; e < passes * bins; e += blockDim.x) s_h[e] = 0u;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t key = keys[i];
        for (int ps = 0; ps < passes; ps++)
            atomicAdd(&s_h[ps * bins + ((key >> (ps * digit_bits)) & mask)], 1u);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < passes * bins; e += blockDim.x)
        if (s_h[e]) atomicAdd(&ghist[e], s_h[e]);
}

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
    return *(const volatile uint32_t*)p;
}
__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) { *(volatile uint32_t*)p = v; }

// Exclusive scan over a 256-thread block; returns the exclusive prefix and writes the total.
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < 8 ? s_warp[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < 8) s_warp[8 + lane] = wi - w;
    }
    __syncthreads();
    const uint32_t r = s_warp[8 + warp] + incl - v;
    __syncthreads();
    return r;
}

constexpr uint32_t kLookbackSpinLimit = 1u << 20;

// Decoupled look-back of tile `tile` for digit `bin`: sums the predecessors' published counts,
// walking back until a tile with an inclusive prefix. kLookbackWide predecessors are read at a
// time: tiles that start together all begin with aggregates, and one word per L2 round trip makes
// tile t wait about t / 2 of them (a 1M-pair sort with its offsets and reorders: 152 us reading one
// at a time, 146 four, 148 eight, 159 sixteen). A predecessor that has published nothing is polled
// at most spin_limit times; then kErrLookbackTimeout is set in *err and the partial sum is returned
// (the caller's scatter is guarded, and the host reports the error word).
constexpr int kLookbackWide = 4;
__device__ __forceinline__ uint32_t lookback_exclusive(const uint32_t* status, int bins,
                                                       uint32_t tile, int bin, uint32_t spin_limit,
                                                       uint32_t* err) {
    uint32_t excl = 0u;
    uint32_t t = tile;  // predecessors below t are still to be summed
    uint32_t spins = 0u;
    while (true) {
        uint32_t w[kLookbackWide];
#pragma unroll
        for (int u = 0; u < kLookbackWide; u++)
            w[u] = (uint32_t)u < t ? ld_volatile(status + (size_t)(t - 1u - (uint32_t)u) * bins + bin) : 0u;
        bool waiting = false;
        uint32_t seen = 0u;
#pragma unroll
        for (int u = 0; u < kLookbackWide; u++) {
            const uint32_t flag = w[u] & ~kCountMask;
            if (waiting || (uint32_t)u >= t) continue;
            if (flag == 0u) {
                waiting = true;
                continue;
            }
            excl += w[u] & kCountMask;
            seen++;
            if (flag == kFlagPrefix || (uint32_t)u + 1u == t) return excl;
        }
        t -= seen;
        if (waiting) {
            if (++spins > spin_limit) {
                atomicOr(err, kErrLookbackTimeout);
                return excl;
            }
            if (seen == 0u) __nanosleep(32);
        }
    }
}

// Failure-detection self-test of the look-back wait: thread b plays tile 1 of digit b over a
// status table whose tile 0 has published (prefix b + 1) or not (nothing). exclusive[b] gets the
// look-back result.
__global__ void k_lookback_selftest(const uint32_t* status, int bins, uint32_t spin_limit,
                                    uint32_t* exclusive, uint32_t* err) {
    const int b = threadIdx.x;
    if (b < bins) exclusive[b] = lookback_exclusive(status, bins, 1u, b, spin_limit, err);
}

// One stable LSD radix pass (onesweep: Adinets & Merrill 2022). Tiles are claimed in launch
// order through an atomic counter, so every predecessor of a tile is already resident and the
// bounded look-back always terminates; a timeout sets an error bit instead of hanging.
// kMatch: ranked by match.any instead of ballots (launch_onesweep_t).
template <int BLOCK, int ITEMS, bool kMatch>
__global__ void __launch_bounds__(BLOCK)
    k_onesweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
               uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
               int shift, int bins, const uint32_t* __restrict__ ghist,
               uint32_t* __restrict__ counter, uint32_t* __restrict__ status,
               uint32_t* __restrict__ err, const uint32_t* __restrict__ n_dev) {
    VFS_CHAINED();
    static_assert(BLOCK == 256, "block scan assumes 256 threads");
    constexpr int WARPS = BLOCK / 32;
    constexpr int TILE = BLOCK * ITEMS;
    // A device-side count (at most n) sorts only that prefix; the grid is sized for n and tiles
    // past the count leave at once (no later tile waits on them: tiles are claimed in order).
    if (n_dev) n = min(n, *n_dev);
    __shared__ uint32_t s_whist[WARPS][kMaxSortBins];
    __shared__ uint32_t s_dstart[kMaxSortBins];
    __shared__ uint32_t s_gofs[kMaxSortBins];
    __shared__ uint32_t s_keys[TILE];
    __shared__ uint32_t s_vals[TILE];
    __shared__ uint32_t s_scan[16];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const uint32_t mask = (uint32_t)bins - 1u;
    const int bits = 32 - __clz((int)mask);
    if (tid == 0) s_tile = atomicAdd(counter, 1u);
    for (int e = tid; e < WARPS * kMaxSortBins; e += BLOCK) (&s_whist[0][0])[e] = 0u;
    // Global exclusive digit offsets of this pass.
    const uint32_t gcount = tid < bins ? __ldg(ghist + tid) : 0u;
    const uint32_t gbase = block_excl_scan256(gcount, s_scan);  // contains __syncthreads
    const uint32_t tile = s_tile;
    if ((uint64_t)tile * TILE >= n) return;  // block-uniform, after the last barrier of the scan
    const uint32_t base = tile * (uint32_t)TILE + (uint32_t)warp * ITEMS * 32u;
    const uint32_t lt_mask = (1u << lane) - 1u;

    uint32_t k[ITEMS], v[ITEMS], r[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t idx = base + it * 32u + lane;
        const bool valid = idx < n;
        k[it] = valid ? keys_in[idx] : 0u;
        v[it] = valid ? (vals_in ? vals_in[idx] : idx) : 0u;
    }
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t idx = base + it * 32u + lane;
        const bool valid = idx < n;
        const uint32_t d = valid ? ((k[it] >> shift) & mask) : (uint32_t)bins;
        // Lanes with the same digit. A ballot per bit (one more than a digit's: the invalid lanes'):
        // eight independent votes take less than a match.any in a sort that fills the GPU (4M pairs:
        // 309 against 336 us).
        uint32_t peers = 0xffffffffu;
        if (kMatch)
            peers = __match_any_sync(0xffffffffu, d);
        else
            for (int b = 0; b <= bits; b++) {
                const bool bit = (d >> b) & 1u;
                const uint32_t vote = __ballot_sync(0xffffffffu, bit);
                peers &= bit ? vote : ~vote;
            }
        const uint32_t pre = __popc(peers & lt_mask);
        uint32_t prev = 0u;
        if (valid) prev = s_whist[warp][d];
        __syncwarp();
        if (valid && pre == 0u) s_whist[warp][d] = prev + __popc(peers);
        __syncwarp();
        r[it] = prev + pre;
    }
    __syncthreads();
    uint32_t cnt = 0u;
    if (tid < bins) {
        uint32_t run = 0u;
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const uint32_t c = s_whist[w][tid];
            s_whist[w][tid] = run;
            run += c;
        }
        cnt = run;
    }
    const uint32_t dstart = block_excl_scan256(cnt, s_scan);
    if (tid < bins) {
        s_dstart[tid] = dstart;
        uint32_t* st = status + (size_t)tile * bins + tid;
        uint32_t excl = 0u;
        if (tile == 0u) {
            st_volatile(st, kFlagPrefix | cnt);
        } else {
            st_volatile(st, kFlagAggregate | cnt);
            excl = lookback_exclusive(status, bins, tile, tid, kLookbackSpinLimit, err);
            st_volatile(st, kFlagPrefix | ((excl + cnt) & kCountMask));
        }
        s_gofs[tid] = gbase + excl;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t idx = base + it * 32u + lane;
        if (idx < n) {
            const uint32_t d = (k[it] >> shift) & mask;
            const uint32_t lpos = s_dstart[d] + s_whist[warp][d] + r[it];
            s_keys[lpos] = k[it];
            s_vals[lpos] = v[it];
        }
    }
    __syncthreads();
    const uint32_t tile_base = tile * (uint32_t)TILE;
    const uint32_t tile_n = min((uint32_t)TILE, n - tile_base);
    for (uint32_t i = tid; i < tile_n; i += BLOCK) {
        const uint32_t kk = s_keys[i];
        const uint32_t d = (kk >> shift) & mask;
        const uint32_t g = s_gofs[d] + (i - s_dstart[d]);
        if (g < n) {  // always true unless a look-back timed out (error word set)
            keys_out[g] = kk;
            vals_out[g] = s_vals[i];
        }
    }
}

// First index in sorted keys[0, n) whose key is >= c (n when none).
__device__ __forceinline__ uint32_t lower_bound_keys(const uint32_t* __restrict__ keys, uint32_t n,
                                                    uint32_t c) {
    uint32_t lo = 0u, hi = n;
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (keys[mid] < c)
            lo = mid + 1u;
        else
            hi = mid;
    }
    return lo;
}


// Block b owns keys [256 b, 256 b + 256) of cell_scan (n + 1 entries: cell_scan[k] is the first
// sorted index with key >= k, so bucket k is [cell_scan[k], cell_scan[k + 1])) and gathers the
// particles with sorted indices in the same range. Two binary searches bound the block's slice
// of the sorted keys; each element of the slice writes the entries between its predecessor's key
// and its own, which never leave the block's range, so no thread loops over more than 256
// entries however the keys cluster.
// First index in sorted keys[0, n) whose key is >= c, searched from guess g: a gallop away from g
// (doubling steps) brackets the answer, a binary search finishes it. A few loads when g is close
// (the previous substep's answer), about twice the plain search's otherwise; exact for any g.
__device__ __forceinline__ uint32_t lower_bound_near(const uint32_t* __restrict__ keys, uint32_t n,
                                                    uint32_t c, uint32_t g) {
    g = min(g, n);
    uint32_t lo, hi;
    if (g < n && keys[g] < c) {  // the answer lies in (g, n]
        lo = g + 1u;
        hi = lo;
        uint32_t step = 1u;
        while (hi < n && keys[hi] < c) {
            lo = hi + 1u;
            hi = (n - hi > step) ? hi + step : n;
            step <<= 1;
        }
    } else {  // the answer lies in [0, g]
        hi = g;
        lo = g;
        uint32_t step = 1u;
        while (lo > 0u && keys[lo - 1u] >= c) {
            hi = lo - 1u;
            lo = lo > step ? lo - step : 0u;
            step <<= 1;
        }
    }
    // Now (lo == 0 or keys[lo - 1] < c) and (hi == n or keys[hi] >= c).
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (keys[mid] < c)
            lo = mid + 1u;
        else
            hi = mid;
    }
    return lo;
}

// The gather of particle i (every thread of the block calls it, i >= n too): position and velocity
// by the sort's permutation; with skin lists (xcur set), the position and sorted index under the
// particle's build index and its displacement since the build, flagging its scene.
__device__ __forceinline__ void reorder_particle(
    const StepLaunch& L, uint32_t i, uint32_t n, const uint32_t* __restrict__ perm,
    const float4* __restrict__ pos_in, const float4* __restrict__ vel_in, float4* __restrict__ pos_out,
    float4* __restrict__ vel_out, const uint32_t* __restrict__ b_of_id, float4* __restrict__ xcur,
    const float4* __restrict__ x_build, uint32_t* __restrict__ stale, const uint32_t* __restrict__ ctl,
    uint32_t* __restrict__ wcount) {
    bool exceed = false;  // skin lists: the particle moved past h skin / 2 since its list build
    bool jump = false;    // and as far since the last substep
    uint32_t exceed_sc = 0u;
    if (i < n) {
        uint32_t src = perm[i];
        if (src >= n) src = i;  // only after a reported sort failure
        const float4 x = __ldg(pos_in + src);
        pos_out[i] = x;
        if (!L.defer_vel) vel_out[i] = __ldg(vel_in + src);
        if (xcur) {
            const uint32_t sc = L.n_scenes > 1 ? (uint32_t)__ldg(L.scene_of + i) : 0u;
            exceed_sc = sc;
            if (ctl[sc * kSkinCtl + kCtlFresh] == 0u) {
                // No build yet, or the last build's lists have gone stale: they stay unusable
                // until the next build, so the scene is stale without a displacement check, and
                // nothing reads its positions by build index.
                exceed = true;
            } else {
                // Skin lists: the particle's current position and sorted index under its build
                // index (the list pass gathers both with one load), and its displacement since
                // the build.
                const uint32_t id = __float_as_uint(x.w);
                const uint32_t bi = id < n ? __ldg(b_of_id + id) : n;
                if (bi < n) {
                    const float4 b = __ldg(x_build + bi);
                    const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z;
                    const float lim = L.n_scenes > 1 ? L.scenes[sc].skin_half2 : L.one.skin_half2;
                    exceed = !(dx * dx + dy * dy + dz * dz <= lim);
                    if (exceed) {
                        const float4 o = xcur[bi];
                        const float ex = x.x - o.x, ey = x.y - o.y, ez = x.z - o.z;
                        jump = !(ex * ex + ey * ey + ez * ez <= lim);
                    }
                    xcur[bi] = make_float4(x.x, x.y, x.z, __uint_as_float(i));
                }
            }
        }
    }
    // Stale scenes, one atomic per warp and scene at most (most particles of a fast scene exceed).
    if (xcur) {
        const uint32_t m = __ballot_sync(0xffffffffu, exceed);
        if (exceed) {
            const uint32_t g = __match_any_sync(m, exceed_sc);
            const uint32_t word = __any_sync(g, jump) ? kSkinStale | kSkinJump : kSkinStale;
            if ((threadIdx.x & 31u) == (uint32_t)(__ffs(g) - 1) && (word & ~ld_volatile(stale + exceed_sc))) {
                atomicOr(stale + exceed_sc, word);
                if (ctl[exceed_sc * kSkinCtl + kCtlAllow]) wcount[1] = 1u;  // a build is due
            }
        }
    }
}

template <uint32_t kCellBlock>
__global__ void __launch_bounds__(kCellBlock)
    k_cells_reorder(StepLaunch L, uint32_t n, const uint32_t* __restrict__ skeys,
                    const uint32_t* __restrict__ perm, uint32_t* __restrict__ scan,
                    const float4* __restrict__ pos_in, const float4* __restrict__ vel_in,
                    float4* __restrict__ pos_out, float4* __restrict__ vel_out,
                    uint32_t* __restrict__ zero, uint32_t zero_words,
                    uint32_t* __restrict__ pkeys_out, uint32_t* guess,
                    const uint32_t* __restrict__ b_of_id, float4* __restrict__ xcur,
                    const float4* __restrict__ x_build, uint32_t* __restrict__ stale,
                    const uint32_t* __restrict__ ctl, uint32_t* __restrict__ wcount, bool late) {
    VFS_CHAINED_LATE();
    if (!late) chained_release();
    __shared__ uint32_t s_lo, s_hi;
    if (wcount && blockIdx.x == 0 && threadIdx.x == 0) wcount[0] = 0u;  // the list pass's queue
    // The sort is done with its scratch (histograms, tile counters, look-back status): clear it
    // for the next substep here instead of in a separate memset.
    for (uint32_t w = blockIdx.x * kCellBlock + threadIdx.x; w < zero_words; w += gridDim.x * kCellBlock)
        zero[w] = 0u;
    const uint32_t c0 = blockIdx.x * kCellBlock;
    const uint32_t c1 = min(c0 + kCellBlock, n + 1u);
    const uint32_t tid = threadIdx.x;
    // The block's slice of the sorted keys, searched from the previous substep's bounds (cell
    // boundaries move little per substep). guess[b] is block b's lower bound; block b reads its
    // neighbour's entry while that block may be rewriting it, and either value is a valid guess.
    if (tid == 0) {
        s_lo = guess ? lower_bound_near(skeys, n, c0, ((volatile uint32_t*)guess)[blockIdx.x])
                     : lower_bound_keys(skeys, n, c0);
        if (guess) guess[blockIdx.x] = s_lo;
    }
    if (tid == 32)
        s_hi = guess ? lower_bound_near(skeys, n, c1, ((volatile uint32_t*)guess)[blockIdx.x + 1])
                     : lower_bound_keys(skeys, n, c1);
    const uint32_t i = c0 + tid;
    reorder_particle(L, i, n, perm, pos_in, vel_in, pos_out, vel_out, b_of_id, xcur, x_build, stale, ctl, wcount);
    if (i < n && pkeys_out) pkeys_out[i] = skeys[i];
    __syncthreads();
    const uint32_t lo = s_lo, hi = max(s_lo, s_hi);
    if (lo == hi) {
        for (uint32_t c = c0 + tid; c < c1; c += kCellBlock) scan[c] = lo;
        return;
    }
    // The clamps keep writes inside [c0, c1) even if the keys were not sorted.
    for (uint32_t j = lo + tid; j < hi; j += kCellBlock) {
        const uint32_t k = min(skeys[j], c1 - 1u);
        const uint32_t start = j == lo ? c0 : max(skeys[j - 1] + 1u, c0);
        for (uint32_t c = start; c <= k; c++) scan[c] = j;
    }
    const uint32_t last = max(min(skeys[hi - 1u], c1 - 1u) + 1u, c0);
    for (uint32_t c = last + tid; c < c1; c += kCellBlock) scan[c] = hi;
}

// The gather alone, for models whose sort writes the cell starts (k_sort_small).
__global__ void __launch_bounds__(128)
    k_reorder(StepLaunch L, uint32_t n, const uint32_t* __restrict__ perm, const float4* __restrict__ pos_in,
              const float4* __restrict__ vel_in, float4* __restrict__ pos_out, float4* __restrict__ vel_out,
              const uint32_t* __restrict__ b_of_id, float4* __restrict__ xcur,
              const float4* __restrict__ x_build, uint32_t* __restrict__ stale,
              const uint32_t* __restrict__ ctl, uint32_t* __restrict__ wcount) {
    VFS_CHAINED_LATE();
    if (wcount && blockIdx.x == 0 && threadIdx.x == 0) wcount[0] = 0u;  // the list pass's queue
    reorder_particle(L, blockIdx.x * 128u + threadIdx.x, n, perm, pos_in, vel_in, pos_out, vel_out, b_of_id,
                     xcur, x_build, stale, ctl, wcount);
}

__global__ void __launch_bounds__(256)
    k_offsets(uint32_t n, uint32_t off, const uint32_t* __restrict__ scan,
              uint32_t* __restrict__ offsets) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t a = scan[off + k], b = scan[off + k + 1];
    offsets[k] = b > a ? a - off : n;
}

// ---------------------------------------------------------------- neighbour passes
// Two phases per particle. Phase A walks every candidate of the 27 buckets with a cheap,
// branch-free distance test and appends the in-range ones to a per-thread list in shared memory
// (slot-major, so a warp's lanes hit consecutive banks). Phase B runs the kernel math over the
// compacted list. Without the split a warp pays the in-range path for almost every candidate
// (only ~15% of candidates are within h, but one of 32 lanes nearly always is). The list keeps
// candidate order, so the sums are accumulated in the reference's visiting order. A list that
// fills up (dense regions) is drained early and refilled.

constexpr int kListCap = 48;
constexpr int kDrainAt = kListCap - 4;  // a batch of four never overflows the list

// Squared distance, in units of h^2, from a particle at fraction f of its cell (along one axis)
// to the neighbour cell at offset d in {-1, 0, +1} along that axis.
__device__ __forceinline__ float face_dist2(uint32_t d, float f) {
    const float l = d == 0xFFFFFFFFu ? f : (d == 1u ? 1.0f - f : 0.0f);
    const float c = fmaxf(l, 0.0f);
    return c * c;
}

// Cells whose box lies farther than h from the particle hold no in-range candidate and are
// skipped, which cannot change any sum as long as no other of the 27 neighbour cells shares
// their key (a shared key would be walked once more by the reference). The 27 keys are distinct
// when the 3x3x3 block of cells lies inside one 50^3 hash block and its hashes do not wrap past
// 2^32 (they are then hmin + d with distinct d in [0, 5102]) and n > 5102; elsewhere nothing is
// skipped. The 2e-3 margin keeps the float cell fractions conservative.
constexpr float kPruneLimit = 1.002f;

// True when the 27 neighbour cells of (cx, cy, cz) provably have 27 distinct keys (see above).
__device__ __forceinline__ bool distinct_keys(const SceneParams& p, uint32_t cx, uint32_t cy,
                                              uint32_t cz) {
    const uint32_t h_lo = hash_cell(cx - 1u, cy - 1u, cz - 1u);
    const uint32_t h_hi = hash_cell(cx + 1u, cy + 1u, cz + 1u);
    return p.n > 5102u && (cx + 24u) / 50u == (cx + 26u) / 50u &&
           (cy + 24u) / 50u == (cy + 26u) / 50u && (cz + 24u) / 50u == (cz + 26u) / 50u &&
           h_hi >= h_lo;
}

// Walks the candidates of the 27 neighbour buckets of cell (cx, cy, cz) in the reference's order
// and calls visit(j, q) for each, with q = pos[j]; four positions are fetched per iteration and
// batch_end() runs after each group of at most four (where a full list is drained).
// Rows t_begin..t_end-1 only, when given (t = (dy + 1) + 3 (dz + 1)).
template <typename Visit, typename BatchEnd>
__device__ __forceinline__ void for_each_candidate(const SceneParams& p,
                                                   const uint32_t* __restrict__ scan,
                                                   const float4* __restrict__ pos,
                                                   const float4& xi, uint32_t cx, uint32_t cy,
                                                   uint32_t cz, Visit&& visit,
                                                   BatchEnd&& batch_end, int t_begin = 0,
                                                   int t_end = 9) {
    const bool interior = distinct_keys(p, cx, cy, cz);
    const float lim = interior ? kPruneLimit : 1e30f;
    const float fx = fmaf(-(float)(int)cx, p.h, xi.x) * p.inv_h;
    const float fy = fmaf(-(float)(int)cy, p.h, xi.y) * p.inv_h;
    const float fz = fmaf(-(float)(int)cz, p.h, xi.z) * p.inv_h;
    const float dxl = face_dist2(0xFFFFFFFFu, fx), dxr = face_dist2(1u, fx);
#pragma unroll 1
    for (int t = t_begin; t < t_end; t++) {
        const uint32_t dy = (uint32_t)(t % 3) - 1u, dz = (uint32_t)(t / 3) - 1u;
        const float dyz = face_dist2(dy, fy) + face_dist2(dz, fz);
        if (dyz > lim) continue;
        const bool skip_l = dyz + dxl > lim, skip_r = dyz + dxr > lim;
        const uint32_t ry = cy + dy, rz = cz + dz;
        const uint32_t hA = hash_cell(cx - 1u, ry, rz);
        const uint32_t kA = key_mod(hA, p.mod_magic, p.n);
        uint32_t b0, e0, b1 = 0u, e1 = 0u, b2 = 0u, e2 = 0u;
        int nseg = 1;
        // Cells cx-1..cx+1 share a hash block iff (cell + 25) / 50 agrees at both ends (this also
        // covers the wrap of cell + 25 at 2^32 near cell -26).
        const bool same_block = (cx + 24u) / 50u == (cx + 26u) / 50u && hA <= 0xFFFFFFFDu;
        const uint32_t* sc = scan + p.off;  // the scene's keys are off + local key
        if (same_block && kA + 2u < p.n) {
            // Buckets kA, kA+1, kA+2 are adjacent: one range, trimmed at either end.
            b0 = __ldg(sc + kA + (skip_l ? 1u : 0u));
            e0 = __ldg(sc + kA + (skip_r ? 2u : 3u));
        } else {
            const uint32_t kB = key_mod(hash_cell(cx, ry, rz), p.mod_magic, p.n);
            const uint32_t kC = key_mod(hash_cell(cx + 1u, ry, rz), p.mod_magic, p.n);
            b0 = __ldg(sc + kA);
            e0 = skip_l ? b0 : __ldg(sc + kA + 1u);
            b1 = __ldg(sc + kB);
            e1 = __ldg(sc + kB + 1u);
            nseg = 3;
            if (!skip_r) {
                b2 = __ldg(sc + kC);
                e2 = __ldg(sc + kC + 1u);
            }
        }
#pragma unroll 1
        for (int seg = 0; seg < nseg; seg++) {
            const uint32_t b = seg == 0 ? b0 : (seg == 1 ? b1 : b2);
            const uint32_t e = seg == 0 ? e0 : (seg == 1 ? e1 : e2);
            uint32_t j = b;
            const float4* pp = pos + b;
#pragma unroll 1
            for (; j + 4u <= e; j += 4u, pp += 4) {
                const float4 q0 = __ldg(pp), q1 = __ldg(pp + 1);
                const float4 q2 = __ldg(pp + 2), q3 = __ldg(pp + 3);
                visit(j, q0);
                visit(j + 1u, q1);
                visit(j + 2u, q2);
                visit(j + 3u, q3);
                batch_end();
            }
#pragma unroll 1
            for (; j < e; j++, pp++) visit(j, __ldg(pp));
            batch_end();
        }
    }
}

// |x_j - x_i|^2 as the density pass's in-range tests evaluate it, explicitly rounded so that the
// bucket walk and the skin lists decide every pair the same way.
__device__ __forceinline__ float in_range2(const float4& xi, const float4& xj) {
    const float dx = __fsub_rn(xj.x, xi.x), dy = __fsub_rn(xj.y, xi.y), dz = __fsub_rn(xj.z, xi.z);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// Threads per block of the density pass over the skin lists.
constexpr int kListBlock = 128;

// A single scene's queue of at least this many walkers is walked in runs of 32 (where one wave of
// warps, ~2,400, has three particles each to walk a warp per walker); a smaller one a warp per walker.
// A batch's queue is walked a thread per walker above kBatchCrowd (64 scenes, 1.1M particles, density
// passes of 32 substeps with 10,000 to 44,000 walkers: 7.90 ms always per thread, 7.50 with the line at
// 16,384 or 32,768, 8.14 at 65,536).
constexpr uint32_t kWalkerCrowd = 8192;
constexpr uint32_t kBatchCrowd = 16384;
// A batch's lists of fewer particles than a line are left alone beside a crowd of walkers, or beside more
// than one in kBatchWalked of its particles: every scene walks. The line is three eighths of the batch,
// between half of kBatchListed and kBatchListed: the list pass costs ~25 us however few it sums, a walk less
// its lists' particles saves ~0.3 us for every thousand, the less the more there are (ms a pass at lines of
// 49,152 / 65,536 / 98,304: 117,906 particles 5.93 / 6.19 / 6.13, 140,822 5.53 / 5.85 / 5.80, 165,121 5.60 / 5.67 /
// 5.89, 231,700 9.49 / 9.38 / 8.84, 245,147 16.60 / 16.01 / 15.92; a third, three eighths, two fifths: 140,822
// 5.57 / 5.51 / 5.84, 22 others within 2%). The smallest batches walk in less than a wave whatever is left
// (crowds alone / one in four / six / eight: 39,742 particles 4.64 / 4.36 / 4.40 / 4.39, 40,403 4.05 / 3.52 / 3.52 /
// 3.50, 56,717 4.24 / 4.25 / 3.67 / 3.64, 49,754 4.32 / 4.33 / 4.69 / 4.67; calm batches the same).
constexpr uint32_t kBatchWalked = 6;
constexpr uint32_t kBatchListed = 98304;

// 1 / sqrt(x) for a normal x (the form without ftz spends four more instructions on denormals).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// W(|x_j - x_i|) / sigma from r2 = in_range2(x_i, x_j), explicitly rounded, so every walk and
// launch shape gives the same sums. Branch-free: 2 (1-q)^3 above q = 1/2, 6q^3 - 6q^2 + 1 below,
// 0 past 1. (A denormal r2 counts as 0: W is 1 either way.)
__device__ __forceinline__ float w_over_sigma_r2(float r2, float inv_h) {
    const float r = r2 > 1.0e-37f ? __fmul_rn(r2, rsqrt_normal(r2)) : 0.0f;
    const float q = __fmul_rn(r, inv_h);
    const float t = __fsub_rn(1.0f, q);
    const float w_out = __fmul_rn(__fmul_rn(__fmul_rn(t, t), t), 2.0f);
    const float q2 = __fmul_rn(q, q);
    const float w_in = __fmaf_rn(6.0f, __fmul_rn(q2, q), __fmaf_rn(-6.0f, q2, 1.0f));
    return q <= 1.0f ? (q > 0.5f ? w_out : w_in) : 0.0f;
}

// Particle i's density sum and neighbour list as the density pass builds them: add() takes one
// in-range neighbour, adds its W / sigma (explicitly rounded, so every launch shape and both the
// bucket walk and the skin lists give the same sums) and appends j to the list unless j == i.
struct DensitySum {
    float rho = 0.0f;
    uint32_t listed = 0;
    uint4* out;  // the next quad of i's list (stride = particles)
    uint32_t q0 = 0, q1 = 0, q2 = 0;  // the last entries, not yet stored
    __device__ __forceinline__ void add(uint32_t i, const float4& xi, uint32_t j, const float4& xj,
                                        float inv_h, uint32_t cap, uint32_t stride) {
        add_r2(i, j, in_range2(xi, xj), true, inv_h, cap, stride);
    }
    // The same with r2 = in_range2(x_i, x_j) already computed, for a candidate that counts only
    // when `in` (adding 0 leaves the sum as it is).
    __device__ __forceinline__ void add_r2(uint32_t i, uint32_t j, float r2, bool in, float inv_h,
                                           uint32_t cap, uint32_t stride) {
        rho = __fadd_rn(rho, in ? w_over_sigma_r2(r2, inv_h) : 0.0f);
        if (in && j != i) {
            if ((listed & 3u) == 3u && listed < nbr_row(cap)) {
                *out = make_uint4(q0, q1, q2, j);
                out += stride;
            }
            q0 = q1;
            q1 = q2;
            q2 = j;
            listed++;
        }
    }
    // Stores the last quad when it is not full (its other words are never read).
    __device__ __forceinline__ void flush(uint32_t cap) {
        const uint32_t m = listed & 3u;
        if (m && listed < nbr_row(cap)) *out = m == 1u ? make_uint4(q2, 0u, 0u, 0u) : m == 2u ? make_uint4(q1, q2, 0u, 0u) : make_uint4(q0, q1, q2, 0u);
    }
};

// The per-particle end of the density pass: list length word, boundary terms, density, Tait EOS
// and the force pass's record of i.
__device__ __forceinline__ void density_finish(const SceneParams& p, uint32_t i, const float4& xi,
                                               const float4* __restrict__ vel, uint32_t cx,
                                               uint32_t cy, uint32_t cz, bool distinct,
                                               const DensitySum& d, float4* __restrict__ rec,
                                               float4* __restrict__ aux, float4* __restrict__ bnd,
                                               uint32_t* __restrict__ nbr_count,
                                               float* __restrict__ host_dens, bool defer_vel) {
    nbr_count[i] = nbr_word(d.listed, cx, cy, cz, distinct);
    float bd, bgx, bgy, bgz;
    boundary_terms(p, xi.x, xi.y, xi.z, bd, bgx, bgy, bgz);
    const float rho = p.mass * p.cubic * d.rho + p.rho0 * bd;  // the factor the sum leaves out
    const float pr = p.stiffness * (powf(fmaxf(rho, p.rho0) / p.rho0, p.expoent) - 1.0f);
    const float pd = rho > 0.0f ? pr / (rho * rho) : 0.0f;
    const float mr = p.mass / fmaxf(rho, 1e-6f);
    const float pb = rho > 0.0f ? pr / (p.rho0 * p.rho0) : 0.0f;
    aux[i] = make_float4(pd, mr, rho, pb);
    if (host_dens) host_dens[i] = rho;
    // The force pass's neighbour record of i: one 32-byte sector per gathered neighbour (the
    // velocity half later, from launch_vel_records, when the velocities arrive late).
    rec[2 * (size_t)i] = make_float4(xi.x, xi.y, xi.z, pd);
    if (!defer_vel) {
        const float4 vi = __ldg(vel + i);
        rec[2 * (size_t)i + 1] = make_float4(vi.x, vi.y, vi.z, mr);
    }
    bnd[i] = make_float4(bgx, bgy, bgz, bd);
}

// ---- tiles: 32 particles of a few cells against the union of their neighbour cells

// Particles consecutive in sorted order lie in one row of cells, or in a few. A warp's 32
// particles are split into groups of one row (same scene, same y and z cell, x cells within
// kTileCells); the group's neighbour cells are rows of x runs (3 x 3 rows for the walk, 5 x 5 for a
// list build), and when the keys of the union are distinct (checked run against run), every
// particle of the group meets each of its candidates exactly once among the union's buckets.
//   Stage: the union's particles are loaded 32 at a time in visiting order, and those within the
//     radius of the group's bounding box are kept, packed, in shared memory.
//   Filter: |x_j - x_i|^2 - limit of 32 particles x 128 candidates comes from the tensor cores:
//     (-2 x_i, 1) . (x_j, |x_j|^2) + (|x_i|^2 - limit) with m16n8k4 TF32 MMAs. Only its sign is
//     kept, one funnel shift per value, as a bit per (particle, candidate). TF32 rounds to 2^-11
//     relative. With coordinates from the group's centre, at most M_a for its particles on axis a
//     and M_a + R for a candidate within the radius R, rounding them moves a pair's distance by at
//     most e = 2^-11 |2 M + R| and its square by 2 R e + e^2, and rounding |x_j|^2 adds
//     2^-11 |M + R|^2. The limit is raised by that bound (~0.013 h^2 for a group of four cells, 1.8%
//     more candidates), so no candidate within the radius is missed; the few beyond it are what a
//     second, exact test (the walk) or a slightly longer list (the build) is for. Two TF32 terms per
//     value (m16n8k8) would keep only 0.7% too many, but took the build from 470 to 660 us at 1M.
//   Each lane then goes through its own particle's bits, in visiting order.
// What bounds it: issue slots. Per 32 particles with ~500 kept candidates the filter costs ~1.7
// instructions per candidate, where a thread's own distance test costs ~12 over the ~165
// candidates left by its pruning. The MMA columns are permuted so that lane (g, q) of a quad holds
// candidates [32 q, 32 q + 32) of its four rows: whole words in visiting order. Lane 4 g + q owns
// particle g + 8 q, the row order of the accumulators.
constexpr int kTileWarps = 4;          // warps per block; a warp works alone
constexpr int kTileBlocks = 4;         // MMA blocks (128 candidates) of a fill
constexpr int kTileWordStride = 34;    // staged candidates per word: 32 and 2 of padding (bank conflicts)
constexpr int kTileMaskStride = 132;   // words per MMA block: 4 rows of 33 (bank conflicts)
constexpr uint32_t kTileCells = 6;     // x cells of a group
constexpr int kTileGroups = 8;         // more groups than this in a warp: no tiles
constexpr float kTileSlack = 0.03f;    // of h: how far a particle may lie outside its cell's place

struct TileSmem {
    union {
        struct {
            float4 cand[kTileBlocks * 4 * kTileWordStride];  // x, y, z, |x - centre|^2 (rounded to TF32)
            uint32_t id[kTileBlocks * 4 * kTileWordStride];  // sorted index
            uint32_t mask[kTileBlocks * kTileMaskStride];    // word q' of particle g + 8 p: 33 p + 4 g + q'
        } t;
        uint32_t j[kListCap * 32];  // per-thread walk: slot-major candidate lists
    };
};

// Blocks of a tile kernel that an SM's shared memory holds (1 KB a block is the system's): a bound of five
// would only take registers away (96 instead of 128: 1.5% of a substep of the 4.6M stress cloud).
constexpr int kTileResident = 4;
static_assert(kTileResident * (kTileWarps * sizeof(TileSmem) + 1024) <= 228u * 1024u &&
                  (kTileResident + 1) * (kTileWarps * sizeof(TileSmem) + 1024) > 228u * 1024u,
              "kTileResident is what fits");

__device__ __forceinline__ float to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

__device__ __forceinline__ void mma_m16n8k4(float d[4], float a0, float a1, float b, float c0, float c1) {
    asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%8,%8};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(b)), "f"(c0), "f"(c1));
}

__device__ __forceinline__ float warp_min(float x) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float warp_max(float x) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// A fill in progress: `blocks` MMA blocks are done (their masks written), `pending` candidates of
// the current group are staged behind them.
struct TileFill {
    int blocks = 0, pending = 0;
};

// The group's side of the MMAs: A fragments, accumulator seeds and the centre component of lane
// (g, q)'s B column.
struct TileRows {
    float a[4], c[4], oq;
};

// Filters the pending candidates: pads them to whole blocks and writes their mask words.
__device__ __forceinline__ void tile_filter(TileSmem& S, TileFill& f, const TileRows& R) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, q = lane & 3u;
    const int nb = (f.pending + 127) >> 7;
    float4* cand = S.t.cand + f.blocks * 4 * kTileWordStride;
    for (int k = f.pending + (int)lane; k < nb * 128; k += 32)
        cand[k + 2 * (k >> 5)] = make_float4(0.0f, 0.0f, 0.0f, 1.0e30f);
    __syncwarp();
    const float* fb = reinterpret_cast<const float*>(cand) + 4u * ((g >> 1) * kTileWordStride + (g & 1u)) + q;
    uint32_t* mw = S.t.mask + f.blocks * kTileMaskStride + lane;
    for (int b = 0; b < nb; b++, fb += 16 * kTileWordStride, mw += kTileMaskStride) {
        uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float bv = to_tf32(fb[8 * k] - R.oq);
            float d[4];
            mma_m16n8k4(d, R.a[0], R.a[1], bv, R.c[0], R.c[1]);
            m[0] = __funnelshift_l(__float_as_uint(d[0]), m[0], 1);
            m[0] = __funnelshift_l(__float_as_uint(d[1]), m[0], 1);
            m[1] = __funnelshift_l(__float_as_uint(d[2]), m[1], 1);
            m[1] = __funnelshift_l(__float_as_uint(d[3]), m[1], 1);
            mma_m16n8k4(d, R.a[2], R.a[3], bv, R.c[2], R.c[3]);
            m[2] = __funnelshift_l(__float_as_uint(d[0]), m[2], 1);
            m[2] = __funnelshift_l(__float_as_uint(d[1]), m[2], 1);
            m[3] = __funnelshift_l(__float_as_uint(d[2]), m[3], 1);
            m[3] = __funnelshift_l(__float_as_uint(d[3]), m[3], 1);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) mw[33 * k] = m[k];
    }
    f.blocks += nb;
    f.pending = 0;
}

// The mask words of this lane's particle: word k at [(k >> 2) * kTileMaskStride + (k & 3)].
__device__ __forceinline__ const uint32_t* tile_masks(const TileSmem& S) {
    const uint32_t lane = threadIdx.x & 31u;
    return S.t.mask + 33u * (lane & 3u) + (lane & ~3u);
}

// Stages and filters one group (mask `grp` of the warp's lanes; cells cx in [c0, c1], cy, cz) of
// particles at xi against everything within `radius` (radius <= reach h) of them. consume(blocks)
// is called whenever a fill is full; what is left in `f` at the end is the caller's to consume.
// Returns false, with nothing staged, when the group does not qualify: its union's keys are not
// distinct, or a particle lies far outside its cell's place (a saturated cell coordinate). p is the
// group's scene's; every argument but xi is warp-uniform.
template <uint32_t kReach, typename Consume>
__device__ __forceinline__ bool tile_group(TileSmem& S, TileFill& f, uint32_t grp, const SceneParams& p,
                                           const uint32_t* __restrict__ scan,
                                           const float4* __restrict__ pos, const float4& xi,
                                           uint32_t c0, uint32_t c1, uint32_t cy, uint32_t cz,
                                           float radius2, Consume&& consume) {
    constexpr uint32_t kSide = 2u * kReach + 1u, kRows = kSide * kSide;
    const uint32_t lane = threadIdx.x & 31u;
    const bool mine = (grp >> lane) & 1u;
    const float h = p.h;
    // Centre of the group's cells; every particle must be near its cell.
    const float hw = 0.5f * (float)(c1 - c0 + 1u);
    const float ox = ((float)(int)c0 + hw) * h;
    const float oy = ((float)(int)cy + 0.5f) * h, oz = ((float)(int)cz + 0.5f) * h;
    const float rx = xi.x - ox, ry = xi.y - oy, rz = xi.z - oz;
    const bool near = fabsf(rx) <= (hw + 0.02f) * h && fabsf(ry) <= 0.52f * h && fabsf(rz) <= 0.52f * h;
    if (!__all_sync(0xffffffffu, !mine || near)) return false;
    // Lane r holds row r of the union's cells, in visiting order: one run of keys or two.
    const uint32_t xa = c0 - kReach, width = c1 - c0 + 1u + 2u * kReach;
    uint32_t n_first;  // cells of a row in the hash block of its first cell
    if (!tile_first_cells(xa, width, n_first)) return false;
    const uint32_t row_y = lane % kSide, row_z = lane / kSide;  // cell offsets from -kReach
    TileRow row{0u, 0u, 0u, 0u, true};
    if (lane < kRows)
        row = tile_row(xa, cy + row_y - kReach, cz + row_z - kReach, width, n_first, p.n, p.mod_magic);
    const uint32_t k0 = row.k0, l0 = row.l0, k1 = row.k1, l1 = row.l1;
    bool ok = row.ok;
    const bool two = __any_sync(0xffffffffu, l1 != 0u);
    // Pairwise disjoint runs modulo n, so every key of the union is met once.
    auto apart = [&](uint32_t ka, uint32_t la, uint32_t kb, uint32_t lb) { return runs_apart(ka, la, kb, lb, p.n); };
    if (two) ok = ok && apart(k0, l0, k1, l1);
    for (uint32_t s = 1u; s <= kRows / 2u; s++) {
        const int o = (int)((lane + s >= kRows ? lane + s - kRows : lane + s) & 31u);
        const uint32_t ka = __shfl_sync(0xffffffffu, k0, o), la = __shfl_sync(0xffffffffu, l0, o);
        bool fine = apart(k0, l0, ka, la);
        if (two) {
            const uint32_t kb = __shfl_sync(0xffffffffu, k1, o), lb = __shfl_sync(0xffffffffu, l1, o);
            fine = fine && apart(k0, l0, kb, lb) && apart(k1, l1, ka, la) && apart(k1, l1, kb, lb);
        }
        ok = ok && (lane >= kRows || fine);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    // The group's bounding box (from its centre), and how much of each row lies within the radius
    // of it; a particle may lie kTileSlack h outside its cell's place.
    const float big = 3.0e38f;
    const float bx0 = warp_min(mine ? rx : big), bx1 = warp_max(mine ? rx : -big);
    const float by0 = warp_min(mine ? ry : big), by1 = warp_max(mine ? ry : -big);
    const float bz0 = warp_min(mine ? rz : big), bz1 = warp_max(mine ? rz : -big);
    uint32_t b0 = 0u, n0 = 0u, b1 = 0u, n1 = 0u;
    if (lane < kRows) {
        const float sy = ((float)row_y - (float)kReach - 0.5f) * h, sz = ((float)row_z - (float)kReach - 0.5f) * h;
        const float dy = fmaxf(fmaxf(by0 - (sy + h), sy - by1) - kTileSlack * h, 0.0f);
        const float dz = fmaxf(fmaxf(bz0 - (sz + h), sz - bz1) - kTileSlack * h, 0.0f);
        const float left = radius2 - dy * dy - dz * dz;
        if (left >= 0.0f) {
            const float half = sqrtf(left) + kTileSlack * h;
            // Cells [ta, tb) of the row, counted from xa.
            const float fa_ = floorf((bx0 - half) * p.inv_h + hw) + (float)kReach;
            const float fb_ = floorf((bx1 + half) * p.inv_h + hw) + (float)kReach;
            const uint32_t ta = (uint32_t)fminf(fmaxf(fa_, 0.0f), (float)width);
            const uint32_t tb = (uint32_t)fminf(fmaxf(fb_ + 1.0f, 0.0f), (float)width);
            const uint32_t* sc = scan + p.off;
            const uint32_t a0 = min(ta, l0), e0 = min(tb, l0);
            if (a0 < e0) {
                b0 = __ldg(sc + k0 + a0);
                n0 = __ldg(sc + k0 + e0) - b0;
            }
            const uint32_t a1 = ta > l0 ? ta - l0 : 0u, e1 = tb > l0 ? tb - l0 : 0u;
            if (a1 < e1 && l1) {
                b1 = __ldg(sc + k1 + a1);
                n1 = __ldg(sc + k1 + min(e1, l1)) - b1;
            }
        }
    }
    // Rows are loaded in words of at most 32 consecutive particles: the words before row r.
    const uint32_t w0 = (n0 + 31u) >> 5, w_row = w0 + ((n1 + 31u) >> 5);
    uint32_t first_word = w_row;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, first_word, o);
        if ((int)lane >= o) first_word += v;
    }
    const uint32_t n_words = __shfl_sync(0xffffffffu, first_word, 31);
    first_word -= w_row;
    // Rows g, g + 8 of the first MMA and g + 16, g + 24 of the second are particles g + 8 p, owned by
    // lanes 4 g + p. Lanes outside the group have no candidate.
    const uint32_t g = lane >> 2, q = lane & 3u;
    TileRows R;
    {
        const float tx = to_tf32(rx), ty = to_tf32(ry), tz = to_tf32(rz);
        // The filter's error bound (see above), and 5% and 2^-13 R^2 for its own single precision.
        const float R_ = sqrtf(radius2);
        const float mx = fmaxf(-bx0, bx1), my = fmaxf(-by0, by1), mz = fmaxf(-bz0, bz1);
        const float sx = 2.0f * mx + R_, sy = 2.0f * my + R_, sz = 2.0f * mz + R_;
        const float e = 4.8828125e-4f * sqrtf(fmaf(sx, sx, fmaf(sy, sy, sz * sz)));
        const float wx = mx + R_, wy = my + R_, wz = mz + R_;
        const float err = fmaf(e, 2.0f * R_ + e, 4.8828125e-4f * fmaf(wx, wx, fmaf(wy, wy, wz * wz)));
        const float lim = radius2 * 1.00012207f + 1.05f * err;
        const float own = mine ? fmaf(tx, tx, fmaf(ty, ty, fmaf(tz, tz, -lim))) : big;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int src = (int)(4u * g) + r;
            const float ax = __shfl_sync(0xffffffffu, tx, src), ay = __shfl_sync(0xffffffffu, ty, src),
                        az = __shfl_sync(0xffffffffu, tz, src);
            R.c[r] = __shfl_sync(0xffffffffu, own, src);
            const float v = q == 0u ? ax : (q == 1u ? ay : az);
            R.a[r] = q == 3u ? 1.0f : (R.c[r] < big ? -2.0f * v : 0.0f);
        }
        R.oq = q == 0u ? ox : (q == 1u ? oy : (q == 2u ? oz : 0.0f));
    }
    const float keep2 = 1.001f * radius2;
    for (uint32_t w32 = 0; w32 < n_words; w32 += 32u) {
        // Lane l describes word w32 + l: its row is the last one starting at or before it.
        uint32_t r = 0u;
#pragma unroll
        for (uint32_t step = 16u; step >= 1u; step >>= 1) {
            const uint32_t probe = __shfl_sync(0xffffffffu, first_word, (int)((r + step) & 31u));
            if (r + step < kRows && probe <= w32 + lane) r += step;
        }
        const uint32_t lw = w32 + lane - __shfl_sync(0xffffffffu, first_word, (int)r);
        const uint32_t rw0 = __shfl_sync(0xffffffffu, w0, (int)r);
        const uint32_t rb0 = __shfl_sync(0xffffffffu, b0, (int)r), rn0 = __shfl_sync(0xffffffffu, n0, (int)r);
        const uint32_t rb1 = __shfl_sync(0xffffffffu, b1, (int)r), rn1 = __shfl_sync(0xffffffffu, n1, (int)r);
        const bool second = lw >= rw0;
        const uint32_t in_run = 32u * (second ? lw - rw0 : lw);
        const uint32_t wj = (second ? rb1 : rb0) + in_run;            // its first particle
        const uint32_t run_n = second ? rn1 : rn0;
        const uint32_t wn = w32 + lane < n_words && run_n > in_run ? run_n - in_run : 0u;  // and how many (or more than 31)
        const uint32_t here = min(32u, n_words - w32);
        for (uint32_t v = 0; v < here; v += 4u) {
            float4 x[4];
            uint32_t j[4];
            bool in[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                j[u] = __shfl_sync(0xffffffffu, wj, (int)(v + u)) + lane;
                in[u] = lane < __shfl_sync(0xffffffffu, wn, (int)(v + u));
                x[u] = in[u] ? __ldg(pos + j[u]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float ux = x[u].x - ox, uy = x[u].y - oy, uz = x[u].z - oz;
                const float ex = fmaxf(fmaxf(bx0 - ux, ux - bx1), 0.0f), ey = fmaxf(fmaxf(by0 - uy, uy - by1), 0.0f),
                            ez = fmaxf(fmaxf(bz0 - uz, uz - bz1), 0.0f);
                in[u] = in[u] && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= keep2;
                const uint32_t kept = __ballot_sync(0xffffffffu, in[u]);
                const int n_kept = __popc(kept);
                if (128 * f.blocks + f.pending + n_kept > 128 * kTileBlocks) {
                    tile_filter(S, f, R);
                    consume(f.blocks);
                    f.blocks = 0;
                }
                if (in[u]) {
                    const int k = 128 * f.blocks + f.pending + __popc(kept & ((1u << lane) - 1u));
                    const float tx = to_tf32(ux), ty = to_tf32(uy), tz = to_tf32(uz);
                    x[u].w = to_tf32(fmaf(tx, tx, fmaf(ty, ty, tz * tz)));
                    S.t.cand[k + 2 * (k >> 5)] = x[u];
                    S.t.id[k + 2 * (k >> 5)] = j[u];
                }
                f.pending += n_kept;
            }
        }
    }
    tile_filter(S, f, R);
    return true;
}

// The groups of a warp's particles (lanes in `todo`, at cells cx, cy, cz of scene sc): calls
// group(mask of its lanes, leader lane, lowest and highest x cell) for each, one row of cells from
// its lowest x cell up. Returns false, with nothing called, when there are more than kTileGroups
// (sparse or scattered particles).
template <typename Group>
__device__ __forceinline__ bool for_each_tile_group(uint32_t todo, uint32_t cx, uint32_t cy, uint32_t cz,
                                                    uint32_t sc, Group&& group) {
    const uint32_t lane = threadIdx.x & 31u;
    for (int pass = 0; pass < 2; pass++) {
        int k = 0;
        for (uint32_t left = todo; left; k++) {
            if (k == kTileGroups) return false;  // in the counting pass
            const int lead = __ffs((int)left) - 1;
            const uint32_t ly = __shfl_sync(0xffffffffu, cy, lead), lz = __shfl_sync(0xffffffffu, cz, lead);
            const uint32_t ls = __shfl_sync(0xffffffffu, sc, lead);
            const bool row = ((left >> lane) & 1u) && cy == ly && cz == lz && sc == ls;
            // Lowest cell of the row (as signed cells) and the lanes within kTileCells of it.
            const int lo = __reduce_min_sync(0xffffffffu, row ? (int)cx : INT_MAX);
            const bool in = row && cx - (uint32_t)lo < kTileCells;
            const uint32_t grp = __ballot_sync(0xffffffffu, in);
            left &= ~grp;
            if (pass == 0) continue;
            const int hi = __reduce_max_sync(0xffffffffu, in ? (int)cx : INT_MIN);
            group(grp, lead, (uint32_t)lo, (uint32_t)hi, ly, lz);
        }
    }
    return true;
}

// The per-thread state of a density walk: particle i at xi, its sum and list so far.
struct WalkState {
    uint32_t i;
    float4 xi;
    DensitySum d;
};

// The walk's sums over the filled blocks: every lane goes through its mask words in order and
// tests, sums and lists the candidates with in_range2 and DensitySum, as the per-thread walk does:
// the same in-range candidates in the same order, so the densities and lists are the same bit
// for bit. The next candidate's load runs ahead of the current one's arithmetic.
__device__ __forceinline__ void tile_sum(const TileSmem& S, int blocks, const SceneParams& p,
                                         uint32_t total, WalkState& w) {
    __syncwarp();
    const uint32_t* m = tile_masks(S);
    const float h2 = p.h2, inv_h = p.inv_h;
    const uint32_t nbr_cap = p.nbr_cap;
    uint32_t nz = 0u;  // words with a bit set, first word highest
    for (int k = 0; k < 4 * blocks; k += 4) {
#pragma unroll
        for (int u = 0; u < 4; u++) nz |= m[33 * k + u] ? 0x80000000u >> (k + u) : 0u;
    }
    uint32_t bits = 0u, at = 0u, j = 0u;
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto next = [&]() {
        if (!bits) {
            if (!nz) return false;
            const uint32_t k = (uint32_t)__clz((int)nz);
            nz ^= 0x80000000u >> k;
            bits = m[(k >> 2) * kTileMaskStride + (k & 3u)];
            at = k * kTileWordStride;
        }
        const uint32_t b = (uint32_t)__clz((int)bits);
        bits ^= 0x80000000u >> b;
        x = S.t.cand[at + b];
        j = S.t.id[at + b];
        return true;
    };
    bool more = next();
    while (more) {
        const float r2 = in_range2(w.xi, x);
        const uint32_t cj = j;
        more = next();
        w.d.add_r2(w.i, cj, r2, r2 <= h2, inv_h, nbr_cap, total);
    }
    __syncwarp();
}
static_assert(kTileMaskStride == 33 * 4, "tile_sum steps 33 words per mask word of a block");

// The lists of the last build are summed this substep (a scene that is stale and may rebuild has
// just rebuilt them).
__device__ __forceinline__ bool lists_in_use(const SkinLists& sk, uint32_t sc) {
    return sk.stale[sc] ? sk.ctl[sc * kSkinCtl + kCtlAllow] != 0u : true;
}

// The same for a single scene's passes, where a scene whose last build left most lists unusable is
// walked in index order until its next build.
__device__ __forceinline__ bool sums_lists(const SkinLists& sk) {
    return sk.stale[0] ? sk.ctl[kCtlAllow] != 0u : sk.ctl[kCtlPoor] == 0u;
}

// The list build: for every particle of a scene that is stale and may rebuild, the candidates
// within h (1 + skin) (and a few just beyond: the filter's margin), in visiting order, under its
// sorted index of this substep, which becomes its build index; its position; and its current
// position and sorted index for the list pass of this substep. A particle whose group is no tile
// or that has more than sk.cap candidates gets no usable list. Other scenes are left alone, and
// the launch returns at its top when no build is due.
template <bool kBatch>
__global__ void __launch_bounds__(kTileWarps * 32, kTileResident)
    k_skin_build(StepLaunch L, const float4* __restrict__ pos, const uint32_t* __restrict__ scan, SkinLists sk) {
    VFS_CHAINED_LATE();
    static_assert(kSkinCap * 32 * sizeof(uint16_t) <= sizeof(float4) * kTileBlocks * 4 * kTileWordStride,
                  "the lists of a fill take the staged positions' place");
    extern __shared__ __align__(16) unsigned char s_raw[];
    TileSmem& S = reinterpret_cast<TileSmem*>(s_raw)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t slot_of = (lane >> 2) + 8u * (lane & 3u);  // lane 4 g + q owns slot g + 8 q of a run
    // The list pass's blocks beside a build's run with what on-chip memory its tiles leave as L1: let in
    // at once only where a build is rarely due (1M flow, building every few substeps: 6.67 ms, let in
    // always 6.74; 97,336 particles 66.1 us a substep, let in late 67.5).
    if (!kBatch && L.total < kSkinFullScene) chained_release();
    if (sk.wcount[1] == 0u) {  // no scene's build is due
        chained_release();
        return;
    }
    const uint32_t runs = (L.total + 31u) / 32u;
    for (uint32_t run = blockIdx.x * (uint32_t)kTileWarps + (threadIdx.x >> 5); run < runs;
         run += gridDim.x * (uint32_t)kTileWarps) {
        const uint32_t i = min(run * 32u + slot_of, L.total - 1u);
        bool act = run * 32u + slot_of < L.total;
        const uint32_t sc = kBatch ? (uint32_t)__ldg(L.scene_of + i) : 0u;
        if (kBatch) act = act && sk.stale[sc] != 0u && sk.ctl[sc * kSkinCtl + kCtlAllow] != 0u;
        const uint32_t todo = __ballot_sync(0xffffffffu, act);
        if (todo == 0u) continue;
        const SceneParams& p = scene_params<kBatch>(L, i);
        const float4 xi = __ldg(pos + i);
        const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h), cz = cell_coord(xi.z, p.h);
        uint32_t c = 0u;  // candidates listed so far
        TileFill f;
        uint32_t refused = 0u;
        auto list = [&](int blocks) {
            __syncwarp();
            const uint32_t* m = tile_masks(S);
            uint16_t* at = reinterpret_cast<uint16_t*>(S.t.cand) + lane;  // slot-major, 32 lanes a slot
            uint32_t n = 0u;
            for (int k = 0; k < 4 * blocks; k++) {
                uint32_t bits = m[(k >> 2) * kTileMaskStride + (k & 3)];
                while (bits) {
                    const uint32_t b = (uint32_t)__clz((int)bits);
                    bits ^= 0x80000000u >> b;
                    if (n < kSkinCap) at[32u * n] = (uint16_t)(k * kTileWordStride + (int)b);
                    n++;
                }
            }
            // A quad at a time (a fill that begins inside one: its words first), so that a warp's
            // lanes store nearby sectors.
            const uint32_t room = c < kSkinCap ? kSkinCap - c : 0u, stored = min(n, room);
            uint32_t k = 0u;
            for (; k < stored && ((c + k) & 3u); k++) sk.list[nbr_word_at(c + k, L.total, i)] = S.t.id[at[32u * k]];
            uint4* out = reinterpret_cast<uint4*>(sk.list) + (size_t)((c + k) >> 2) * L.total + i;
            for (; k + 4u <= stored; k += 4u, out += L.total)
                *out = make_uint4(S.t.id[at[32u * k]], S.t.id[at[32u * (k + 1u)]], S.t.id[at[32u * (k + 2u)]],
                                  S.t.id[at[32u * (k + 3u)]]);
            for (; k < stored; k++) sk.list[nbr_word_at(c + k, L.total, i)] = S.t.id[at[32u * k]];
            c += n;
            __syncwarp();
        };
        if (for_each_tile_group(todo, cx, cy, cz, sc, [&](uint32_t grp, int lead, uint32_t lo, uint32_t hi,
                                                          uint32_t ly, uint32_t lz) {
                const uint32_t li = __shfl_sync(0xffffffffu, i, lead);
                const SceneParams& pl = scene_params<kBatch>(L, li);
                if (!tile_group<2>(S, f, grp, pl, scan, pos, xi, lo, hi, ly, lz, pl.skin_r2, list)) refused |= grp;
            })) {
            if (f.blocks) list(f.blocks);
        } else {
            refused = todo;
        }
        if (act) {
            const bool usable = !((refused >> lane) & 1u) && c <= kSkinCap;
            sk.x_build[i] = xi;
            sk.b_of_id[__float_as_uint(xi.w)] = i;
            sk.xcur[i] = make_float4(xi.x, xi.y, xi.z, __uint_as_float(i));
            sk.count[i] = usable ? c | kSkinUsable : 0u;
            // The scene's usable lists, one atomic per warp and scene.
            const uint32_t gm = __match_any_sync(__activemask(), sc);
            const uint32_t u = __ballot_sync(gm, usable);
            if (lane == (uint32_t)(__ffs((int)gm) - 1) && u)
                atomicAdd(sk.ctl + sc * kSkinCtl + kCtlUsable, (uint32_t)__popc(u));
        }
        __syncwarp();
    }
}

// The walk of one particle by a whole warp (a single scene's few particles without a usable list),
// so that its ~280 candidates are tested 32 at a time instead of in one thread's chain of dependent
// loads. Lane r < 27 holds candidate segment r of the walk (row r / 3, part r % 3 of the rows of
// for_each_candidate: the same buckets, the same pruning), the segments' candidates are numbered in
// visiting order and taken in chunks of 32, and the in-range ones are summed in visiting order
// (every lane adds them one by one through shuffles) and listed in visiting order: exactly the sum
// and the list of the per-thread walk.
__device__ __forceinline__ void walk_by_warp(const SceneParams& p, uint32_t i, uint32_t total_n,
                                             const float4* __restrict__ pos, const float4* __restrict__ vel,
                                             float4* __restrict__ rec, const uint32_t* __restrict__ scan,
                                             float4* __restrict__ aux, float4* __restrict__ bnd,
                                             uint32_t* __restrict__ nbr, uint32_t* __restrict__ nbr_count,
                                             float* __restrict__ host_dens, bool defer_vel) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t* sc = scan + p.off;
    const float4 xi = __ldg(pos + i);
    const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h),
                   cz = cell_coord(xi.z, p.h);
    const bool distinct = distinct_keys(p, cx, cy, cz);
    // Segment r of the walk: [b, b + len).
    uint32_t b = 0u, len = 0u;
    if (lane < 27) {
        const float lim = distinct ? kPruneLimit : 1e30f;
        const float fx = fmaf(-(float)(int)cx, p.h, xi.x) * p.inv_h;
        const float fy = fmaf(-(float)(int)cy, p.h, xi.y) * p.inv_h;
        const float fz = fmaf(-(float)(int)cz, p.h, xi.z) * p.inv_h;
        const int t = lane / 3, part = lane % 3;
        const uint32_t dy = (uint32_t)(t % 3) - 1u, dz = (uint32_t)(t / 3) - 1u;
        const float dyz = face_dist2(dy, fy) + face_dist2(dz, fz);
        if (dyz <= lim) {
            const bool skip_l = dyz + face_dist2(0xFFFFFFFFu, fx) > lim;
            const bool skip_r = dyz + face_dist2(1u, fx) > lim;
            const uint32_t ry = cy + dy, rz = cz + dz;
            const uint32_t hA = hash_cell(cx - 1u, ry, rz);
            const uint32_t kA = key_mod(hA, p.mod_magic, p.n);
            const bool same_block = (cx + 24u) / 50u == (cx + 26u) / 50u && hA <= 0xFFFFFFFDu;
            uint32_t e = 0u;
            if (same_block && kA + 2u < p.n) {
                if (part == 0) {
                    b = __ldg(sc + kA + (skip_l ? 1u : 0u));
                    e = __ldg(sc + kA + (skip_r ? 2u : 3u));
                }
            } else if (part == 0) {
                b = __ldg(sc + kA);
                e = skip_l ? b : __ldg(sc + kA + 1u);
            } else if (part == 1) {
                const uint32_t kB = key_mod(hash_cell(cx, ry, rz), p.mod_magic, p.n);
                b = __ldg(sc + kB);
                e = __ldg(sc + kB + 1u);
            } else if (!skip_r) {
                const uint32_t kC = key_mod(hash_cell(cx + 1u, ry, rz), p.mod_magic, p.n);
                b = __ldg(sc + kC);
                e = __ldg(sc + kC + 1u);
            }
            len = e > b ? e - b : 0u;
        }
    }
    // Exclusive prefix of the segment lengths: the visiting-order number of each segment's
    // first candidate.
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t start = incl - len;
    float rho = 0.0f;
    uint32_t listed = 0u;
    for (uint32_t base = 0; base < total; base += 32u) {
        const uint32_t f = base + (uint32_t)lane;
        // The segment holding candidate f: the last one starting at or before f.
        int r = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const uint32_t s_probe = __shfl_sync(0xffffffffu, start, (r + step) & 31);
            if (r + step < 27 && s_probe <= f) r += step;
        }
        const uint32_t rb = __shfl_sync(0xffffffffu, b, r);
        const uint32_t rs = __shfl_sync(0xffffffffu, start, r);
        const bool valid = f < total;
        const uint32_t j = rb + (f - rs);
        float4 xj = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) xj = __ldg(pos + j);
        const float r2 = in_range2(xi, xj);
        const bool inr = valid && r2 <= p.h2;
        const float wv = inr ? w_over_sigma_r2(r2, p.inv_h) : 0.0f;
        uint32_t mask = __ballot_sync(0xffffffffu, inr);
        const uint32_t listm = __ballot_sync(0xffffffffu, inr && j != i);
        if (inr && j != i) {
            const uint32_t slot = listed + (uint32_t)__popc(listm & lt);
            if (slot < p.nbr_cap) nbr[nbr_word_at(slot, total_n, i)] = j;
        }
        listed += (uint32_t)__popc(listm);
        while (mask) {
            const int l = __ffs(mask) - 1;
            rho = __fadd_rn(rho, __shfl_sync(0xffffffffu, wv, l));
            mask &= mask - 1u;
        }
    }
    if (lane == 0) {
        DensitySum d;
        d.rho = rho;
        d.listed = listed;
        density_finish(p, i, xi, vel, cx, cy, cz, distinct, d, rec, aux, bnd, nbr_count, host_dens,
                   defer_vel);
    }
}

// The walk of the particles k_density_list queued in a single scene (no usable list this substep): a
// crowd (kWalkerCrowd) in runs of 32, a smaller queue a warp per particle (walk_by_warp). One
// resident wave whose warps claim the runs. A warp walks its particles as tiles (tile_group) where they qualify and per
// thread (for_each_candidate) where not. In a crowd dense enough to overflow the skin lists the
// tiles pay most: the filter's cost per candidate is a seventh of a thread's own test (419,000
// particles with ~900 neighbours each: 3.1 ms against 7.5 ms a warp per particle and 8.7 ms a thread
// per particle).
__global__ void __launch_bounds__(kTileWarps * 32, kTileResident)
    k_walk_queue(StepLaunch L, const float4* __restrict__ pos, const float4* __restrict__ vel,
                 float4* __restrict__ rec, const uint32_t* __restrict__ scan,
                 float4* __restrict__ aux, float4* __restrict__ bnd, uint32_t* __restrict__ nbr,
                 uint32_t* __restrict__ nbr_count, SkinLists sk, uint32_t* __restrict__ sched) {
    VFS_CHAINED();
    extern __shared__ __align__(16) unsigned char s_raw[];
    TileSmem& S = reinterpret_cast<TileSmem*>(s_raw)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t slot_of = (lane >> 2) + 8u * (lane & 3u);  // lane 4 g + q owns slot g + 8 q of a run
    if (!sums_lists(sk)) return;  // k_walk walks every particle
    const SceneParams& p = L.one;
    const uint32_t slots = min(*sk.wcount, L.total);
    if (slots < kWalkerCrowd) {
        for (uint32_t k = blockIdx.x * (uint32_t)kTileWarps + (threadIdx.x >> 5); k < slots;
             k += gridDim.x * (uint32_t)kTileWarps)
            walk_by_warp(p, __ldg(sk.queue + k), L.total, pos, vel, rec, scan, aux, bnd, nbr, nbr_count,
                         L.host_dens, L.defer_vel);
        return;
    }
    // Every warp takes runs of 32 slots: first the run of its own index, then runs claimed from
    // the launch's counter (sched[0]), until none is left. Walks differ widely in length (dense and
    // sparse regions), and a warp that finishes early takes the next run. No lane leaves a run
    // before the warp's collective steps: inactive lanes carry act = false.
    const uint32_t runs = (slots + 31u) / 32u;
    const uint32_t warps = gridDim.x * (uint32_t)kTileWarps;
    uint32_t run = blockIdx.x * (uint32_t)kTileWarps + (threadIdx.x >> 5);
    for (; run < runs;) {
        const uint32_t t = run * 32u + slot_of;
        const bool act = t < slots;
        WalkState w{};
        w.i = act ? __ldg(sk.queue + t) : 0u;
        // The next run, claimed now so that the counter's latency hides behind this one.
        uint32_t next = 0u;
        if (lane == 0u) next = warps + atomicAdd(sched, 1u);
        next = __shfl_sync(0xffffffffu, next, 0);
        const uint32_t todo = __ballot_sync(0xffffffffu, act);
        w.xi = act ? __ldg(pos + w.i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w.d.out = reinterpret_cast<uint4*>(nbr) + w.i;
        const uint32_t cx = cell_coord(w.xi.x, p.h), cy = cell_coord(w.xi.y, p.h), cz = cell_coord(w.xi.z, p.h);
        uint32_t single = 0u;  // lanes that walk per thread
        TileFill f;
        auto sum = [&](int blocks) { tile_sum(S, blocks, p, L.total, w); };
        if (for_each_tile_group(todo, cx, cy, cz, 0u, [&](uint32_t grp, int, uint32_t lo, uint32_t hi,
                                                                   uint32_t ly, uint32_t lz) {
                if (!tile_group<1>(S, f, grp, p, scan, pos, w.xi, lo, hi, ly, lz, p.h2, sum)) single |= grp;
            })) {
            if (f.blocks) sum(f.blocks);
        } else {
            single = todo;
        }
        if ((single >> lane) & 1u) {
            // The per-thread walk. Scene constants used per candidate, in registers.
            const float s_inv_h = p.inv_h, h2 = p.h2;
            const uint32_t s_nbr_cap = p.nbr_cap;
            uint32_t s_end = lane;  // word one past the last kept candidate (stride 32)
            auto drain = [&]() {
#pragma unroll 2
                for (uint32_t o = lane; o < s_end; o += 32u) {
                    const uint32_t j = S.j[o];
                    w.d.add(w.i, w.xi, j, __ldg(pos + j), s_inv_h, s_nbr_cap, L.total);
                }
                s_end = lane;
            };
            // Branch-free append: every candidate is stored at the list's end and kept only when
            // in range (the next one overwrites it otherwise). Lists are drained above kDrainAt,
            // so the slot index stays below kListCap.
            for_each_candidate(p, scan, pos, w.xi, cx, cy, cz, [&](uint32_t j, const float4& xj) {
                S.j[s_end] = j;
                s_end += in_range2(w.xi, xj) <= h2 ? 32u : 0u;
            }, [&]() {
                if (s_end > lane + kDrainAt * 32u) drain();
            });
            drain();
        }
        run = next;
        if (act) {
            w.d.flush(p.nbr_cap);
            density_finish(p, w.i, w.xi, vel, cx, cy, cz, distinct_keys(p, cx, cy, cz), w.d, rec, aux, bnd,
                           nbr_count, L.host_dens, L.defer_vel);
        }
        __syncwarp();
    }
    // The last warp out puts the counter back to zero for the next launch (every other warp has
    // made its last claim before it counts itself out).
    if (lane == 0u) {
        __threadfence();
        if (atomicAdd(sched + 1, 1u) == warps - 1u) {
            atomicExch(sched, 0u);
            atomicExch(sched + 1, 0u);
        }
    }
}

// CalculateBoundaryVolume + CalculateDensities + the per-particle part of PressureFromDensityEOS
// (wcsph_with_boundary_model.slang:102-203), by a walk of the neighbour cells, one thread per
// particle. Besides the density products it writes particle i's neighbour list: every in-range j
// except i itself, in visiting order, in quads (nbr_word_at), and its length in nbr_count[i] (a length above nbr_cap means the list
// overflowed and was truncated). Positions do not change before the force pass, so that list is
// exactly the force pass's neighbour set. It walks whole scenes in index order (no skin lists; a
// single scene that is stale and may not rebuild, or whose lists are mostly unusable; a batch whose lists
// are left alone) and a batch's queue. A single scene whose lists are summed returns at the kernel's top. One
// resident wave whose warps claim runs of 32 slots; a single scene's shapes of 768 threads an SM are held
// to the 72 registers that let 28 warps in (74, 24 warps: 130,000 particles walking 92 us, 72 76). The tiles above are no faster for a fluid's ~43
// neighbours: 515 us against 450 us for 1M particles (their sum phase runs at 16 warps per SM, this
// kernel at 27, and it tests only ~200 candidates per particle after pruning).
template <bool kBatch, int kNbrBlock, int kMinBlocks>
__global__ void __launch_bounds__(kNbrBlock, kBatch || kMinBlocks * kNbrBlock > 768 ? kMinBlocks : 896 / kNbrBlock)
    k_walk(StepLaunch L, const float4* __restrict__ pos, const float4* __restrict__ vel,
           float4* __restrict__ rec, const uint32_t* __restrict__ scan,
           float4* __restrict__ aux, float4* __restrict__ bnd, uint32_t* __restrict__ nbr,
           uint32_t* __restrict__ nbr_count, SkinLists sk, uint32_t* __restrict__ sched) {
    VFS_CHAINED_LATE();
    static_assert(kNbrBlock % 32 == 0, "whole warps");
    __shared__ uint32_t s_j[kListCap * kNbrBlock];
    const int tid = threadIdx.x;
    const uint32_t lane = (uint32_t)(tid & 31);
    // The force pass's blocks beside a walk run with what on-chip memory its lists leave as L1: let in
    // only where there is nothing to walk (64 scenes 27.1 ms, late 25.7; 87,386 particles walking 111 us a
    // substep, late 106).
    if (!kBatch && sk.list && sums_lists(sk)) {
        chained_release();
        return;
    }
    // Every warp takes runs of 32 slots: first the run of its own index, then runs claimed from
    // the launch's counter (sched[0]), until none is left. Walks differ widely in length (the
    // queued walkers of a batch, dense and sparse regions), and a warp that finishes early takes
    // the next run.
    uint32_t slots = L.total;
    const uint32_t warps = gridDim.x * (uint32_t)(kNbrBlock / 32);
    const bool queued = kBatch && sk.list && sk.wcount[2] == 0u;  // (else every particle, in index order)
    if (queued) {
        slots = min(*sk.wcount, L.total);
        if (slots == 0u) chained_release();
        if (slots <= kBatchCrowd) {
            for (uint32_t k = blockIdx.x * (uint32_t)(kNbrBlock / 32) + (uint32_t)(tid >> 5); k < slots; k += warps) {
                const uint32_t i = __ldg(sk.queue + k);
                walk_by_warp(scene_params<kBatch>(L, i), i, L.total, pos, vel, rec, scan, aux, bnd, nbr, nbr_count,
                             L.host_dens, L.defer_vel);
            }
            return;
        }
    }
    const uint32_t runs = (slots + 31u) / 32u;
    uint32_t run = blockIdx.x * (uint32_t)(kNbrBlock / 32) + (uint32_t)(tid >> 5);
    for (; run < runs;) {
        const uint32_t t = run * 32u + lane;
        const bool act = t < slots;
        uint32_t i = act ? t : 0u;
        if (queued && act) i = __ldg(sk.queue + t);
        // The next run, claimed now so that the counter's latency hides behind this one.
        uint32_t next = 0u;
        if (lane == 0u) next = warps + atomicAdd(sched, 1u);
        run = __shfl_sync(0xffffffffu, next, 0);
        if (!act) continue;
        const SceneParams& p = scene_params<kBatch>(L, i);
        const float4 xi = __ldg(pos + i);
        const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h), cz = cell_coord(xi.z, p.h);
        DensitySum d;
        d.out = reinterpret_cast<uint4*>(nbr) + i;
        uint32_t s_end = tid;  // shared-memory word one past the last kept candidate (stride kNbrBlock)
        // Scene constants used per candidate, in registers (a batched launch reads its scene's
        // parameters from a device table).
        const float s_inv_h = p.inv_h, h2 = p.h2;
        const uint32_t s_nbr_cap = p.nbr_cap;
        auto drain = [&]() {
#pragma unroll 2
            for (uint32_t o = tid; o < s_end; o += kNbrBlock) {
                const uint32_t j = s_j[o];
                d.add(i, xi, j, __ldg(pos + j), s_inv_h, s_nbr_cap, L.total);
            }
            s_end = tid;
        };
        // Branch-free append: every candidate is stored at the list's end and kept only when in
        // range (the next one overwrites it otherwise). Lists are drained above kDrainAt, so the
        // slot index stays below kListCap.
        for_each_candidate(p, scan, pos, xi, cx, cy, cz, [&](uint32_t j, const float4& xj) {
            s_j[s_end] = j;
            s_end += in_range2(xi, xj) <= h2 ? kNbrBlock : 0u;
        }, [&]() {
            if (s_end > tid + kDrainAt * kNbrBlock) drain();
        });
        drain();
        d.flush(s_nbr_cap);
        density_finish(p, i, xi, vel, cx, cy, cz, distinct_keys(p, cx, cy, cz), d, rec, aux, bnd, nbr_count,
                       L.host_dens, L.defer_vel);
    }
    // The last warp out puts the counter back to zero for the next launch (every other warp has
    // made its last claim before it counts itself out).
    if (lane == 0u) {
        __threadfence();
        if (atomicAdd(sched + 1, 1u) == warps - 1u) {
            atomicExch(sched, 0u);
            atomicExch(sched + 1, 0u);
        }
    }
}

// The density pass over the skin lists: a particle of a scene that is not stale, whose list is
// usable, sums the in-range members of its list (the same in-range set as the walk: every
// pair within h was within h (1 + skin) at the build; each once: the particle has moved less than
// h / 4 since the build, so its 27 cells lie in the build's 5x5x5 block, whose keys were
// distinct), in the list's order. Every other particle goes to the queue for k_walk_queue (a
// batch's: k_walk).
// Bound by the chains of dependent loads and by L1: the gathers' and the list stores' wavefronts. The
// in-range indices wait in a ring of two quads per thread in shared memory and leave as whole quads,
// at most one per four candidates: 1M falling particles 117 -> 104 us (quads gathered in registers
// and stored as they fill: 109 to 116). Nine blocks an SM: ten spill (112 us), eight have fewer loads
// in flight (108).
template <bool kBatch>
__global__ void __launch_bounds__(kListBlock, 9)
    k_density_list(StepLaunch L, const float4* __restrict__ pos, const float4* __restrict__ vel,
                   float4* __restrict__ rec, float4* __restrict__ aux, float4* __restrict__ bnd,
                   uint32_t* __restrict__ nbr, uint32_t* __restrict__ nbr_count, SkinLists sk, bool late) {
    VFS_CHAINED_LATE();
    if (!late) chained_release();
    __shared__ uint32_t s_ring[8 * kListBlock];
    const uint32_t i = blockIdx.x * kListBlock + threadIdx.x;
    // A single scene that is stale and waits, or whose last build left most lists unusable, or a batch whose
    // lists are left alone: k_walk walks it in index order (queueing all of a batch took 7 to 11 us a substep).
    if (kBatch ? sk.wcount[2] != 0u : !sums_lists(sk)) return;
    bool walk = false;
    if (i < L.total) {
        const SceneParams& p = scene_params<kBatch>(L, i);
        uint32_t c = 0u, row = 0u;
        const uint32_t scene = kBatch ? (uint32_t)__ldg(L.scene_of + i) : 0u;
        const bool built = sk.stale[scene] != 0u;  // this substep, unless the scene is walked
        walk = !lists_in_use(sk, scene);
        // A particle of a stale scene only joins the queue: its position is not read.
        const float4 xi = walk ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : __ldg(pos + i);
        if (!walk) {
            row = built ? i : __ldg(sk.b_of_id + __float_as_uint(xi.w));
            c = __ldg(sk.count + row);
            walk = (c & kSkinUsable) == 0u;
        }
        if (!walk) {
            const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h),
                           cz = cell_coord(xi.z, p.h);
            const uint32_t n_list = c & ~kSkinUsable;
            const float h2 = p.h2, s_inv_h = p.inv_h;
            const uint32_t s_nbr_cap = p.nbr_cap;
            DensitySum d;
            d.out = reinterpret_cast<uint4*>(nbr) + i;
            const size_t stride = L.total;
            const uint4* q = reinterpret_cast<const uint4*>(sk.list) + row;
            uint32_t quads = 0u;
            uint32_t* ring = s_ring + threadIdx.x;
            auto add = [&](uint32_t jj, float r2, bool in) {
                d.rho = __fadd_rn(d.rho, in ? w_over_sigma_r2(r2, s_inv_h) : 0.0f);
                ring[(d.listed & 7u) * kListBlock] = jj;
                d.listed += in && jj != i ? 1u : 0u;
            };
            auto put = [&]() {
                const uint32_t* r = ring + (quads & 1u) * (4u * kListBlock);
                if (4u * quads < nbr_row(s_nbr_cap))
                    *d.out = make_uint4(r[0], r[kListBlock], r[2 * kListBlock], r[3 * kListBlock]);
                d.out += L.total;
                quads++;
            };
            // The next quad of build indices loads while the current one is resolved and summed.
            uint4 next = make_uint4(0u, 0u, 0u, 0u);
            if (n_list) next = __ldg(q);
            uint32_t k = 0;
#pragma unroll 1
            for (; k + 4u <= n_list; k += 4u) {
                const uint32_t j[4] = {next.x, next.y, next.z, next.w};
                q += stride;
                if (k + 4u < n_list) next = __ldg(q);
                float4 xj[4];
#pragma unroll
                for (int u = 0; u < 4; u++) xj[u] = __ldg(sk.xcur + j[u]);  // position, sorted index
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const float r2 = in_range2(xi, xj[u]);
                    add(__float_as_uint(xj[u].w), r2, r2 <= h2);
                }
                if ((d.listed >> 2) != quads) put();
            }
            if (k < n_list) {
                const uint32_t m = n_list - k;  // 1 to 3
                const uint32_t j[3] = {next.x, m > 1u ? next.y : next.x, m > 2u ? next.z : next.x};
                float4 xj[3];
#pragma unroll
                for (int u = 0; u < 3; u++) xj[u] = __ldg(sk.xcur + j[u]);
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    const float r2 = in_range2(xi, xj[u]);
                    add(__float_as_uint(xj[u].w), r2, (uint32_t)u < m && r2 <= h2);
                }
            }
            if ((d.listed >> 2) != quads) put();
            if (d.listed & 3u) put();
            density_finish(p, i, xi, vel, cx, cy, cz, distinct_keys(p, cx, cy, cz), d, rec, aux,
                           bnd, nbr_count, L.host_dens, L.defer_vel);
        }
    }
    // The walkers go to the queue, packed from 0 in blocks claimed by one atomic each, in index order
    // within the block.
    __shared__ uint32_t s_cnt[kListBlock / 32];
    __shared__ uint32_t s_base;
    const uint32_t m = __ballot_sync(0xffffffffu, walk);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) s_cnt[warp] = (uint32_t)__popc(m);
    __syncthreads();
    uint32_t base = 0u, total = 0u;
#pragma unroll
    for (int w = 0; w < kListBlock / 32; w++) {
        base += w < warp ? s_cnt[w] : 0u;
        total += s_cnt[w];
    }
    if (threadIdx.x == 0) s_base = total ? atomicAdd(sk.wcount, total) : 0u;
    __syncthreads();
    base += s_base;  // at most L.total walkers in all: the slots stay inside the queue
    if (walk) sk.queue[base + (uint32_t)__popc(m & ((1u << lane) - 1u))] = i;
}

// Small models, where three lanes per particle still fit one wave of the GPU and one lane per
// particle would leave the SMs waiting on each thread's chain of candidate loads: the density pass
// with the 27-cell walk split over three lanes of one warp, lane r walking the rows of the z-plane
// dz = r - 1 (rows 3r..3r+2). Each lane sums its plane in visiting order and the particle's density
// is (plane 0 + plane 1) + plane 2, whatever the list capacity. The neighbour list is the planes'
// entries one after the other, the reference's visiting order as in k_walk, so the force pass
// is the same in both modes. A plane whose shared list fills mid-walk keeps summing but its
// entries are not listed (the list length is then reported above the capacity, and the force
// pass walks the candidates again).
constexpr int kPlaneBlock = 96;  // 3 warps x 10 particles x 3 lanes (2 lanes of each warp idle)

template <bool kBatch>
__global__ void __launch_bounds__(kPlaneBlock)
    k_density_planes(StepLaunch L, const float4* __restrict__ pos, const float4* __restrict__ vel,
                     float4* __restrict__ rec, const uint32_t* __restrict__ scan,
                     float4* __restrict__ aux, float4* __restrict__ bnd,
                     uint32_t* __restrict__ nbr, uint32_t* __restrict__ nbr_count) {
    VFS_CHAINED_LATE();
    __shared__ uint32_t s_j[kListCap * kPlaneBlock];
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u, pw = lane / 3u, pl = lane - 3u * pw;
    const uint32_t lead = lane - pl;
    const uint32_t i = (blockIdx.x * (kPlaneBlock / 32u) + (tid >> 5)) * 10u + pw;
    const bool active = lane < 30u && i < L.total;
    float rho = 0.0f;
    uint32_t n_pl = 0u;  // this plane's entries other than the particle itself
    bool lost = false;   // entries summed mid-walk and not kept for the list
    uint32_t s_end = tid;
    float4 xi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (active) {
        const SceneParams& p = scene_params<kBatch>(L, i);
        xi = __ldg(pos + i);
        const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h),
                       cz = cell_coord(xi.z, p.h);
        const float s_inv_h = p.inv_h, h2 = p.h2;
        auto sum_list = [&]() {
#pragma unroll 2
            for (uint32_t o = tid; o < s_end; o += kPlaneBlock) {
                const uint32_t j = s_j[o];
                rho = __fadd_rn(rho, w_over_sigma_r2(in_range2(xi, __ldg(pos + j)), s_inv_h));
                n_pl += j != i ? 1u : 0u;
            }
        };
        for_each_candidate(p, scan, pos, xi, cx, cy, cz, [&](uint32_t j, const float4& xj) {
            const float dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
            const float r2 = dx * dx + dy * dy + dz * dz;
            s_j[s_end] = j;
            s_end += r2 <= h2 ? kPlaneBlock : 0u;
        }, [&]() {
            if (s_end > tid + kDrainAt * kPlaneBlock) {
                sum_list();
                lost = true;
                s_end = tid;
            }
        }, 3 * (int)pl, 3 * (int)pl + 3);
        sum_list();
    }
    // The three planes of a particle meet in its lead lane (lanes 30 and 31 exchange nothing
    // that is used).
    const uint32_t n0 = __shfl_sync(0xffffffffu, n_pl, lead);
    const uint32_t n1 = __shfl_sync(0xffffffffu, n_pl, lead + 1u);
    const uint32_t n2 = __shfl_sync(0xffffffffu, n_pl, lead + 2u);
    const float rho1 = __shfl_sync(0xffffffffu, rho, lead + 1u);
    const float rho2 = __shfl_sync(0xffffffffu, rho, lead + 2u);
    const uint32_t lost_bits = __ballot_sync(0xffffffffu, lost);
    if (!active) return;
    const SceneParams& p = scene_params<kBatch>(L, i);
    const bool any_lost = ((lost_bits >> lead) & 7u) != 0u;
    const uint32_t total = n0 + n1 + n2;
    if (!any_lost) {
        uint32_t k = (pl >= 1u ? n0 : 0u) + (pl >= 2u ? n1 : 0u);
        for (uint32_t o = tid; o < s_end; o += kPlaneBlock) {
            const uint32_t j = s_j[o];
            if (j == i) continue;
            if (k < p.nbr_cap) nbr[nbr_word_at(k, L.total, i)] = j;
            k++;
        }
    }
    if (pl != 0u) return;
    const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h), cz = cell_coord(xi.z, p.h);
    const uint32_t listed = any_lost ? max(total, p.nbr_cap + 1u) : total;
    nbr_count[i] = nbr_word(listed, cx, cy, cz, distinct_keys(p, cx, cy, cz));
    float bd, bgx, bgy, bgz;
    boundary_terms(p, xi.x, xi.y, xi.z, bd, bgx, bgy, bgz);
    rho = __fadd_rn(__fadd_rn(rho, rho1), rho2);
    rho = p.mass * p.cubic * rho + p.rho0 * bd;
    const float pr = p.stiffness * (powf(fmaxf(rho, p.rho0) / p.rho0, p.expoent) - 1.0f);
    const float pd = rho > 0.0f ? pr / (rho * rho) : 0.0f;
    const float mr = p.mass / fmaxf(rho, 1e-6f);
    const float pb = rho > 0.0f ? pr / (p.rho0 * p.rho0) : 0.0f;
    aux[i] = make_float4(pd, mr, rho, pb);
    if (L.host_dens) L.host_dens[i] = rho;
    rec[2 * (size_t)i] = make_float4(xi.x, xi.y, xi.z, pd);
    if (!L.defer_vel) {
        const float4 vi = __ldg(vel + i);
        rec[2 * (size_t)i + 1] = make_float4(vi.x, vi.y, vi.z, mr);
    }
    bnd[i] = make_float4(bgx, bgy, bgz, bd);
}

struct ForceAcc {
    float Px, Py, Pz, Vx, Vy, Vz;
};

// Pressure and viscosity contributions of one in-range neighbour (PressureAccel slang:234-249,
// ViscousAccel slang:301-318) with the constant factors taken out of the sums. With
// dW = grad_over_h * c(q) (c = -(1-q)^2 above q = 1/2, q (3q - 2) below, 0 outside the support or
// at r <= 1e-9) and u = c(q) / r, the reference's terms are
//   pressure:   mass * (pd_i + pd_j) * dW * x_ij / r  = (mass * grad_over_h) * [(pd_i + pd_j) u x_ij]
//   viscosity:  mr_j (v_ij . x_ij) dW x_ij / r / (r^2 + 0.01 h^2) = grad_over_h * [mr_j (v_ij . x_ij) u x_ij / (r^2 + eps)]
// and only the bracketed parts are summed here; k_force applies the factors once per particle.
// Every operation is an explicit round-to-nearest intrinsic, so no fusion is left to the
// compiler and every launch shape of the force pass gives bit-identical results.
__device__ __forceinline__ void force_term(const SceneParams& p, const float4& xi, const float4& vi,
                                           float pdi, const float4& xj, const float2& aj,
                                           const float4& vj, ForceAcc& f) {
    const float xx = __fsub_rn(xi.x, xj.x), xy = __fsub_rn(xi.y, xj.y), xz = __fsub_rn(xi.z, xj.z);
    const float r2 = __fmaf_rn(xz, xz, __fmaf_rn(xy, xy, __fmul_rn(xx, xx)));
    const float ir = rsqrtf(fmaxf(r2, 1e-30f));  // finite at r2 = 0, where u is 0 below
    const float r = __fmul_rn(r2, ir);
    const float q = __fmul_rn(r, p.inv_h);
    const float t = __fsub_rn(1.0f, q);
    const float c_out = -__fmul_rn(t, t);
    const float c_in = __fmul_rn(q, __fmaf_rn(3.0f, q, -2.0f));
    const float c = q > 0.5f ? c_out : c_in;
    const float u = (r > 1e-9f && q <= 1.0f) ? __fmul_rn(c, ir) : 0.0f;
    const float sp = __fmul_rn(__fadd_rn(pdi, aj.x), u);
    f.Px = __fmaf_rn(sp, xx, f.Px);
    f.Py = __fmaf_rn(sp, xy, f.Py);
    f.Pz = __fmaf_rn(sp, xz, f.Pz);
    const float dv = __fmaf_rn(__fsub_rn(vi.z, vj.z), xz,
                               __fmaf_rn(__fsub_rn(vi.y, vj.y), xy, __fmul_rn(__fsub_rn(vi.x, vj.x), xx)));
    const float iden = __fdividef(1.0f, __fadd_rn(r2, p.visc_eps));
    const float sv = __fmul_rn(__fmul_rn(__fmul_rn(aj.y, dv), u), iden);
    f.Vx = __fmaf_rn(sv, xx, f.Vx);
    f.Vy = __fmaf_rn(sv, xy, f.Vy);
    f.Vz = __fmaf_rn(sv, xz, f.Vz);
}

// A 32-byte force record in one 256-bit load (sm_100+; rec + 2j is 32-byte aligned because the
// buffer comes from cudaMalloc and each record is 32 bytes).
__device__ __forceinline__ void load_record(const float4* __restrict__ rec, uint32_t j, float4& a,
                                            float4& b) {
    const float4* q = rec + 2 * (size_t)j;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(q));
}

// One neighbour's term from its force record: rec[2j] = (x, y, z, p/rho^2), rec[2j+1] =
// (vx, vy, vz, m/max(rho, 1e-6)), the same values as pos, vel and aux hold.
__device__ __forceinline__ void force_term_rec(const SceneParams& p, const float4& xi,
                                               const float4& vi, float pdi,
                                               const float4* __restrict__ rec, uint32_t j,
                                               ForceAcc& f) {
    float4 r0, r1;
    load_record(rec, j, r0, r1);
    force_term(p, xi, vi, pdi, r0, make_float2(r0.w, r1.w), r1, f);
}

// The rest of CalculatePressureAccel + CalculateViscousAccel + UpdatePositions for particle i
// once its sums are complete: the constant factors, the boundary term, gravity, the wall, and
// symplectic Euler.
__device__ __forceinline__ void force_finish(const SceneParams& p, uint32_t i, const float4& xi,
                                             const float4& vi, const float4& ai, ForceAcc f,
                                             const float4* __restrict__ bnd,
                                             float4* __restrict__ pos_out,
                                             float4* __restrict__ vel_out,
                                             float4* __restrict__ acc_out, float3& x_new,
                                             float3& v_new) {
    const float pdi = ai.x;
    // The factors force_term leaves out of the sums.
    const float cp = p.mass * p.grad_over_h, cv = p.visc_scale * p.grad_over_h;
    f.Px *= cp;
    f.Py *= cp;
    f.Pz *= cp;
    const float4 bi = __ldg(bnd + i);
    const float sb = (pdi + ai.w) * p.rho0;
    f.Px += sb * bi.x;
    f.Py += sb * bi.y;
    f.Pz += sb * bi.z;

    float ax = p.gx + -f.Px, ay = p.gy + -f.Py, az = p.gz + -f.Pz;
    ax += cv * f.Vx;
    ay += cv * f.Vy;
    az += cv * f.Vz;
    // WallAcceleration, wcsph_with_boundary_model.slang:336-347.
    const float dx = fminf(xi.x - p.lo[0], 0.0f) - fminf(p.hi[0] - xi.x, 0.0f);
    const float dyw = fminf(xi.y - p.lo[1], 0.0f) - fminf(p.hi[1] - xi.y, 0.0f);
    const float dzw = fminf(xi.z - p.lo[2], 0.0f) - fminf(p.hi[2] - xi.z, 0.0f);
    if (fabsf(dx) > 1e-9f || fabsf(dyw) > 1e-9f || fabsf(dzw) > 1e-9f) {
        ax += -p.wall_k * dx;
        ay += -p.wall_k * dyw;
        az += -p.wall_k * dzw;
    }
    if (acc_out) acc_out[i] = make_float4(ax, ay, az, 0.0f);
    const float nvx = vi.x + ax * p.dt, nvy = vi.y + ay * p.dt, nvz = vi.z + az * p.dt;
    v_new = make_float3(nvx, nvy, nvz);
    x_new = make_float3(xi.x + nvx * p.dt, xi.y + nvy * p.dt, xi.z + nvz * p.dt);
    vel_out[i] = make_float4(nvx, nvy, nvz, 0.0f);
    pos_out[i] = make_float4(x_new.x, x_new.y, x_new.z, xi.w);
}

// CalculatePressureAccel + CalculateViscousAccel + UpdatePositions
// (wcsph_with_boundary_model.slang:205-360), fused: both sums are accumulated separately in the
// reference's visiting order, then a = ((g - P) + V) + wall, v += a dt, x += v dt.
// Fresh lists have gone stale, `age` substeps after their build, in a jump or by drift: the substep of the
// run that has just begun at which to build lists that reach both its ends, if it is like the last one and
// they can (0: no such build).
__device__ __forceinline__ uint32_t skin_middle(uint32_t* c, uint32_t age, bool jump) {
    if (c[kCtlTried]) {
        const uint32_t fails = age > kSkinMiddleKept ? 0u : min(c[kCtlFails] + 1u, 6u);
        c[kCtlTried] = 0u;
        c[kCtlFails] = fails;
        c[kCtlPass] = fails ? 1u << fails : 0u;
    }
    if (!jump) {
        c[kCtlLife] = age;
        return 0u;
    }
    const uint32_t run = c[kCtlRun], life = c[kCtlLife];
    c[kCtlRun] = c[kCtlLife] = 0u;
    if (c[kCtlPass]) {
        c[kCtlPass]--;
        return 0u;
    }
    if (life == 0u || run > 2u * life + 1u || c[kCtlPoor]) return 0u;
    c[kCtlTried] = 1u;
    return run / 2u;
}

template <bool kBatch, int kNbrBlock, int kMinBlocks>
__global__ void __launch_bounds__(kNbrBlock, kMinBlocks)
    k_force(StepLaunch L, const float4* __restrict__ pos, const float4* __restrict__ vel,
            const float4* __restrict__ aux, const float4* __restrict__ rec,
            const float4* __restrict__ bnd,
            const uint32_t* __restrict__ scan, const uint32_t* __restrict__ nbr,
            const uint32_t* __restrict__ nbr_count, float4* __restrict__ pos_out,
            float4* __restrict__ vel_out, float4* __restrict__ acc_out,
            uint32_t* __restrict__ skin_stale, uint32_t* __restrict__ skin_ctl,
            uint32_t* __restrict__ skin_due, HostOut ho) {
    VFS_CHAINED();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // The density pass is done with the skin lists' flags: run each scene's build policy and clear
    // the flags for the next substep.
    if (skin_stale && blockIdx.x == 0) {
        __shared__ uint32_t s_listed;  // batch: particles of the scenes with lists to sum or to build
        uint32_t listed = 0u;
        if (kBatch && threadIdx.x == 0) s_listed = 0u;
        if (threadIdx.x == 0) *skin_due = 0u;
        for (uint32_t sc = threadIdx.x; sc < L.n_scenes; sc += blockDim.x) {
            uint32_t* c = skin_ctl + sc * kSkinCtl;
            const bool stale = skin_stale[sc] != 0u;
            const uint32_t n = L.n_scenes > 1 ? L.scenes[sc].n : L.one.n;
            const uint32_t min_life = n < kSkinSmallScene ? kSkinMinLifeSmall
                                      : n < kSkinFullScene ? kSkinMinLife
                                                           : kSkinMinLifeFull;
            const uint32_t grace = n < kSkinFullScene ? 0u : kSkinGrace;
            uint32_t age = c[kCtlAge], wait = c[kCtlWait], since = c[kCtlSince], young = c[kCtlYoung];
            uint32_t middle = c[kCtlMiddle];
            if (stale && c[kCtlFresh]) {  // the last build's lists just went stale: were they worth it?
                middle = n >= kSkinSmallScene ? skin_middle(c, age, (skin_stale[sc] & kSkinJump) != 0u) : 0u;
                if (middle && !c[kCtlAllow]) {  // not rebuilt now: it walks until then
                    wait = middle;
                    middle = 0u;
                } else if (age < min_life || c[kCtlPoor]) {
                    young++;
                    if (young > grace || c[kCtlPoor]) wait = min(max(2u * wait, kSkinMinWait), kSkinMaxWait);
                } else {
                    young = wait = 0u;
                }
                c[kCtlFresh] = 0u;
                since = 0u;
            }
            if (stale && c[kCtlAllow]) {  // the density pass rebuilt
                c[kCtlBuilds]++;
                c[kCtlFresh] = 1u;
                c[kCtlPoor] = c[kCtlUsable] < n - n / kSkinPoorPart ? 1u : 0u;
                c[kCtlUsable] = 0u;
                age = 0u;
            } else {
                age++;
                if (stale) since++;
            }
            if (middle && --middle == 0u) {  // the lists rebuilt at the jump have served
                c[kCtlFresh] = 0u;
                wait = since = 0u;
            }
            skin_stale[sc] = 0u;
            c[kCtlRun]++;
            c[kCtlMiddle] = middle;
            c[kCtlAge] = age;
            c[kCtlWait] = wait;
            c[kCtlSince] = since;
            c[kCtlYoung] = young;
            // Lists that have lived long enough are rebuilt in the very substep they go stale in
            // (a small scene's, which walks beside the others of its batch, one substep later).
            const bool at_once = n >= kSkinSmallScene && (age >= min_life || young < grace) && !c[kCtlPoor];
            c[kCtlAllow] = (c[kCtlFresh] ? at_once : since >= wait) ? 1u : 0u;
            if (kBatch && (c[kCtlFresh] ? c[kCtlPoor] == 0u : since >= wait)) listed += n;
        }
        if (kBatch) {
            __syncthreads();
            if (listed) atomicAdd(&s_listed, listed);
            __syncthreads();
            const uint32_t line = min(kBatchListed, max(kBatchListed / 2u, L.total / 8u * 3u));
            const bool off = s_listed < line && L.total - s_listed > min(kBatchCrowd, L.total / kBatchWalked);
            if (threadIdx.x == 0) skin_due[1] = off ? 1u : 0u;
            if (off)
                for (uint32_t sc = threadIdx.x; sc < L.n_scenes; sc += blockDim.x) skin_ctl[sc * kSkinCtl + kCtlAllow] = 0u;
        }
    }
    // The particle's new position and velocity and its density, for the host outputs.
    float3 x_new = make_float3(0.0f, 0.0f, 0.0f), v_new = x_new;
    float dens_i = 0.0f;
    if (i < L.total) {
        const SceneParams& p = scene_params<kBatch>(L, i);
        const float4 xi = __ldg(pos + i);
        const float4 vi = __ldg(vel + i);
        const float4 ai = __ldg(aux + i);
        const float pdi = ai.x;

        ForceAcc f{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        const uint32_t listed = nbr_count[i] & kNbrCountMask;
        if (listed <= p.nbr_cap) {
            // The density pass's list: the in-range neighbours in the reference's visiting order.
            // A quad of indices is one load, made under the previous quad's gathers, so each quad
            // waits on one dependent load (the records) instead of two, the last, partial one too.
            const uint4* nl = reinterpret_cast<const uint4*>(nbr) + i;
            const size_t stride = L.total;
            uint4 next = make_uint4(0u, 0u, 0u, 0u);
            if (listed) next = __ldg(nl);
            uint32_t k = 0;
#pragma unroll 1
            for (; k + 4u <= listed; k += 4u) {
                const uint32_t j[4] = {next.x, next.y, next.z, next.w};
                nl += stride;
                if (k + 4u < listed) next = __ldg(nl);
                float4 a[4], b[4];
#pragma unroll
                for (int u = 0; u < 4; u++) load_record(rec, j[u], a[u], b[u]);
#pragma unroll
                for (int u = 0; u < 4; u++) force_term(p, xi, vi, pdi, a[u], make_float2(a[u].w, b[u].w), b[u], f);
            }
            if (k < listed) {
                const uint32_t m = listed - k;  // 1 to 3
                const uint32_t j[3] = {next.x, m > 1u ? next.y : next.x, m > 2u ? next.z : next.x};
                float4 a[3], b[3];
#pragma unroll
                for (int u = 0; u < 3; u++) load_record(rec, j[u], a[u], b[u]);
#pragma unroll
                for (int u = 0; u < 3; u++)
                    if ((uint32_t)u < m) force_term(p, xi, vi, pdi, a[u], make_float2(a[u].w, b[u].w), b[u], f);
            }
        } else {
            // Overflowed list (very dense neighbourhood): walk the candidates again and add every
            // in-range one as it comes, in the same order. This path needs no shared memory, so
            // the pass keeps the whole on-chip memory as L1 for its record gathers.
            const uint32_t cx = cell_coord(xi.x, p.h), cy = cell_coord(xi.y, p.h),
                           cz = cell_coord(xi.z, p.h);
            for_each_candidate(p, scan, pos, xi, cx, cy, cz, [&](uint32_t j, const float4& xj) {
                const float xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
                const float r2 = xx * xx + xy * xy + xz * xz;
                if (r2 <= p.h2 && j != i) force_term_rec(p, xi, vi, pdi, rec, j, f);
            }, [&]() {});
        }
        force_finish(p, i, xi, vi, ai, f, bnd, pos_out, vel_out, acc_out, x_new, v_new);
        dens_i = ai.z;
    }
    if (ho.pos3 || ho.vel3 || ho.dens) {
        // Host outputs (a single scene; the launch gives 7 floats of dynamic shared memory per
        // thread): the block's particles are consecutive slots, so each array's part is staged
        // and written out as contiguous words, whole lines over the host link.
        extern __shared__ float s_io[];
        const uint32_t t = threadIdx.x, base = blockIdx.x * (uint32_t)kNbrBlock;
        const uint32_t m = min((uint32_t)kNbrBlock, L.total - base);
        s_io[3 * t] = x_new.x;
        s_io[3 * t + 1] = x_new.y;
        s_io[3 * t + 2] = x_new.z;
        s_io[3 * kNbrBlock + 3 * t] = v_new.x;
        s_io[3 * kNbrBlock + 3 * t + 1] = v_new.y;
        s_io[3 * kNbrBlock + 3 * t + 2] = v_new.z;
        s_io[6 * kNbrBlock + t] = dens_i;
        __syncthreads();
        const size_t b3 = 3 * (size_t)base;
        for (uint32_t k = t; k < 3 * m; k += kNbrBlock) {
            if (ho.pos3) ho.pos3[b3 + k] = s_io[k];
            if (ho.vel3) ho.vel3[b3 + k] = s_io[3 * kNbrBlock + k];
        }
        if (ho.dens && t < m) ho.dens[base + t] = s_io[6 * kNbrBlock + t];
    }
}

// ---------------------------------------------------------------- incremental sort
// Particles move little per substep, so most keep the key they had in the previous substep, whose
// stably sorted keys `pkeys` line up with the current (reordered) particles. The particles whose
// key changed ("moved", in index order) are sorted stably by key and merged with the others by
// (key, index): exactly the stable sort of all (key, index) pairs. The unmoved particles' keys are
// pkeys[i], a subsequence of a sorted array, so they are already in order; this holds for any
// sorted pkeys (all moved when pkeys is the all-ones fill of a fresh model), so no step ever
// needs to know whether pkeys is current.

// Keys, moved flags and the moved particles' compaction, in two or three launches without a chain
// between tiles: the moved flags as a bitmask with one word per 32 particles, bits[w], and the
// number of moved particles before each word, pre[w] (pre[W] = total = *mcount, W = ceil(n / 32),
// pre = bits + W); (mkeys, midx)[rank] for the moved ones in index order; and the digit
// histograms of the moved keys. A tile is 256 threads x kDeltaItems particles (particle
// tile * kDeltaTile + item * 256 + thread, so every load is coalesced, and a warp's 32 particles
// of one item are one bitmask word: the tile's words are bits[32 tile, 32 tile + 32), in (item,
// warp) order).
//   k_keys_flags:    keys, moved flags, each tile's moved count (tile_cnt), histograms;
//   k_tile_scan:     one block: the tiles' exclusive prefixes in place, the total (only above
//                    kFoldTiles tiles; below, each compaction block sums its predecessors' counts);
//   k_moved_compact: per tile, each word's prefix and the moved particles' (key, index) pairs
//                    at their ranks (the key recomputed from the position: the same arithmetic).
// One launch would have to chain its tiles by a decoupled look-back, which resolves ~32 tiles per
// L2 round trip: ~22 us for the 1,024 tiles of a 1M-particle model, whatever the bytes.
constexpr int kDeltaItems = 4;
constexpr uint32_t kDeltaTile = 256u * kDeltaItems;

template <bool kBatch>
__device__ __forceinline__ uint32_t particle_key(const StepLaunch& L, uint32_t i, const float4& x) {
    const SceneParams& p = scene_params<kBatch>(L, i);
    return p.off + key_mod(hash_cell(cell_coord(x.x, p.h), cell_coord(x.y, p.h), cell_coord(x.z, p.h)),
                           p.mod_magic, p.n);
}

// kHostIn (a single scene's host round trip): the positions come from page-locked host memory,
// packed float3 in slot order (host3, its device address), and the kernel also stores them as the
// model's positions (pos_out, id = slot) and zeroes the densities, as the state upload does (with
// b_next, the build index under each slot's old id is stored under its new id first); the tile's
// 12 KB are read into shared memory with coalesced loads first.
template <bool kBatch, bool kHostIn>
__global__ void __launch_bounds__(256)
    k_keys_flags(StepLaunch L, const float4* __restrict__ pos, const uint32_t* __restrict__ pkeys,
                 uint32_t* __restrict__ bits, int passes, int digit_bits,
                 uint32_t* __restrict__ ghist, uint32_t* __restrict__ tile_cnt,
                 const float* __restrict__ host3, float4* __restrict__ pos_out,
                 float4* __restrict__ aux, const uint32_t* __restrict__ b_of_id,
                 uint32_t* __restrict__ b_next) {
    VFS_CHAINED();
    __shared__ uint32_t s_h[kMaxSortPasses * kMaxSortBins];
    __shared__ uint32_t s_n[8];
    __shared__ float s_p[kHostIn ? 3 * kDeltaTile : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bins = 1 << digit_bits;
    const uint32_t mask = (uint32_t)bins - 1u;
    for (int e = tid; e < passes * bins; e += 256) s_h[e] = 0u;
    const uint32_t t0 = blockIdx.x * kDeltaTile;
    if (kHostIn) {
        const uint32_t m3 = 3u * min(kDeltaTile, L.total - t0);
        const float* src = host3 + 3 * (size_t)t0;
        for (uint32_t k = (uint32_t)tid; k < m3; k += 256u) s_p[k] = src[k];
    }
    __syncthreads();
    const uint32_t base = t0 + (uint32_t)tid;
    const uint32_t W = (L.total + 31u) >> 5;
    // All of the thread's loads first (positions and previous keys), then the key arithmetic.
    float4 xs[kDeltaItems];
    uint32_t pks[kDeltaItems];
#pragma unroll
    for (int k = 0; k < kDeltaItems; k++) {
        const uint32_t i = base + (uint32_t)k * 256u;
        if (i < L.total) {
            if (kHostIn) {
                const uint32_t l = 3u * ((uint32_t)k * 256u + (uint32_t)tid);
                xs[k] = make_float4(s_p[l], s_p[l + 1u], s_p[l + 2u], __uint_as_float(i));
                if (b_next) {
                    const uint32_t old = __float_as_uint(pos_out[i].w);
                    b_next[i] = old < L.total ? b_of_id[old] : 0u;
                }
                pos_out[i] = xs[k];
                aux[i].z = 0.0f;
            } else {
                xs[k] = __ldg(pos + i);
            }
            pks[k] = __ldg(pkeys + i);
        }
    }
    uint32_t cnt = 0u;
#pragma unroll
    for (int k = 0; k < kDeltaItems; k++) {
        const uint32_t i = base + (uint32_t)k * 256u;
        bool moved = false;
        if (i < L.total) {
            const uint32_t key = particle_key<kBatch>(L, i, xs[k]);
            moved = key != pks[k];
            if (moved)
                for (int ps = 0; ps < passes; ps++)
                    atomicAdd(&s_h[ps * bins + ((key >> (ps * digit_bits)) & mask)], 1u);
        }
        const uint32_t ball = __ballot_sync(0xffffffffu, moved);
        const uint32_t word = (i - (uint32_t)lane) >> 5;
        if (lane == 0 && word < W) bits[word] = ball;
        cnt += (uint32_t)__popc(ball);
    }
    if (lane == 0) s_n[warp] = cnt;
    __syncthreads();
    if (tid == 0) {
        uint32_t t = 0u;
#pragma unroll
        for (int w = 0; w < 8; w++) t += s_n[w];
        tile_cnt[blockIdx.x] = t;
    }
    for (int e = tid; e < passes * bins; e += 256)
        if (s_h[e]) atomicAdd(&ghist[e], s_h[e]);
}

// Exclusive prefix sums of the tiles' moved counts, in place, by one block in chunks of 1,024
// tiles (one chunk up to 1M particles); the total goes to *mcount and pre[W].
__global__ void __launch_bounds__(1024)
    k_tile_scan(uint32_t tiles, uint32_t* __restrict__ tile_cnt, uint32_t* __restrict__ bits,
                uint32_t W, uint32_t* __restrict__ mcount) {
    VFS_CHAINED();
    __shared__ uint32_t s_w[32];
    __shared__ uint32_t s_carry;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) s_carry = 0u;
    __syncthreads();
    for (uint32_t b = 0; b < tiles; b += 1024u) {
        const uint32_t t = b + tid;
        const uint32_t v = t < tiles ? tile_cnt[t] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += y;
        }
        if (lane == 31u) s_w[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t y = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
                if ((int)lane >= o) y += z;
            }
            s_w[lane] = y;
        }
        __syncthreads();
        const uint32_t incl = s_carry + (warp ? s_w[warp - 1] : 0u) + x;
        if (t < tiles) tile_cnt[t] = incl - v;
        __syncthreads();  // every thread has read s_carry and s_w
        if (tid == 1023u) s_carry = incl;
        __syncthreads();
    }
    if (tid == 0) {
        *mcount = s_carry;
        bits[2u * W] = s_carry;  // pre[W]
    }
}

// Up to this many tiles (4M particles) the compaction's blocks sum the earlier tiles' counts
// themselves (at most 16 loads per thread) and the scan kernel is not launched.
constexpr uint32_t kFoldTiles = 4096u;

// kFolded: tile_cnt holds the tiles' counts (k_tile_scan did not run): the block sums those of
// the tiles before its own, and the last tile writes the total. Otherwise tile_cnt holds the
// exclusive prefixes.
template <bool kBatch, bool kFolded>
__global__ void __launch_bounds__(256)
    k_moved_compact(StepLaunch L, const float4* __restrict__ pos, uint32_t* __restrict__ bits,
                    const uint32_t* __restrict__ tile_cnt, uint32_t* __restrict__ mkeys,
                    uint32_t* __restrict__ midx, uint32_t* __restrict__ mcount) {
    VFS_CHAINED();
    __shared__ uint32_t s_bits[32], s_off[32], s_sum[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t W = (L.total + 31u) >> 5;
    uint32_t excl;
    if (kFolded) {
        uint32_t part = 0u;
        for (uint32_t u = tid; u < blockIdx.x; u += 256u) part += tile_cnt[u];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0u) s_sum[warp] = part;
        __syncthreads();
        excl = 0u;
#pragma unroll
        for (int w = 0; w < 8; w++) excl += s_sum[w];
        if (tid == 0u && blockIdx.x == gridDim.x - 1u) {
            const uint32_t total = excl + tile_cnt[blockIdx.x];
            *mcount = total;
            bits[2u * W] = total;  // pre[W]
        }
    } else {
        excl = tile_cnt[blockIdx.x];
    }
    if (warp == 0) {
        const uint32_t w = blockIdx.x * 32u + lane;
        const uint32_t b = w < W ? bits[w] : 0u;
        const uint32_t c = (uint32_t)__popc(b);
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) x += y;
        }
        const uint32_t off = excl + x - c;
        s_bits[lane] = b;
        s_off[lane] = off;
        if (w < W) bits[W + w] = off;
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < kDeltaItems; k++) {
        const uint32_t i = blockIdx.x * kDeltaTile + (uint32_t)k * 256u + tid;
        const uint32_t b = s_bits[k * 8 + warp];
        if (i < L.total && ((b >> lane) & 1u)) {
            const uint32_t rank = s_off[k * 8 + warp] + (uint32_t)__popc(b & lt);
            mkeys[rank] = particle_key<kBatch>(L, i, __ldg(pos + i));
            midx[rank] = i;
        }
    }
}

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* a, uint32_t n, uint32_t v) {
    uint32_t lo = 0u, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1u; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t upper_bound_u32(const uint32_t* a, uint32_t n, uint32_t v) {
    uint32_t lo = 0u, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] <= v) lo = mid + 1u; else hi = mid;
    }
    return lo;
}

// Merge of the unmoved particles (keys pkeys[i], in index order) with the sorted moved ones
// (mk, mi) by (key, index). Thread t < n places unmoved particle t; thread n + r places the moved
// particle of sorted rank r. Every output position is computed independently.
// Moved particles with index < i (0 <= i <= n) from the bitmask and per-word prefix.
__device__ __forceinline__ uint32_t moved_before(const uint32_t* __restrict__ bits, uint32_t W,
                                                 uint32_t i) {
    const uint32_t w = i >> 5;
    if (w >= W) return bits[W + W];
    return bits[W + w] + __popc(bits[w] & ((1u << (i & 31u)) - 1u));
}

__global__ void __launch_bounds__(256)
    k_merge(uint32_t n, const uint32_t* __restrict__ pkeys, const uint32_t* __restrict__ bits,
            const uint32_t* __restrict__ mcount, const uint32_t* __restrict__ mk,
            const uint32_t* __restrict__ mi, uint32_t* __restrict__ out_keys,
            uint32_t* __restrict__ out_perm) {
    VFS_CHAINED();
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t m = min(*mcount, n);
    const uint32_t W = (n + 31u) >> 5;
    uint32_t key, idx, pos;
    if (t < n) {
        idx = (uint32_t)t;
        const uint32_t word = bits[idx >> 5];
        if ((word >> (idx & 31u)) & 1u) return;  // moved: placed by its sorted rank
        const uint32_t before = bits[W + (idx >> 5)] + __popc(word & ((1u << (idx & 31u)) - 1u));
        key = pkeys[idx];
        uint32_t lo = 0u, hi = m;  // moved particles ordered before (key, idx)
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            const uint32_t k2 = mk[mid];
            if (k2 < key || (k2 == key && mi[mid] < idx)) lo = mid + 1u; else hi = mid;
        }
        pos = (idx - before) + lo;
    } else if (t < (uint64_t)n + m) {
        const uint32_t r = (uint32_t)(t - n);
        key = mk[r];
        idx = mi[r];
        // Unmoved particles ordered before (key, idx): pkeys is sorted and unmoved j has key
        // pkeys[j], so they are the unmoved j below lower_bound(key) plus the unmoved j < idx in
        // the equal-key range [L, R).
        const uint32_t lb = lower_bound_u32(pkeys, n, key), ub = upper_bound_u32(pkeys, n, key);
        const uint32_t e = idx > lb ? min(idx, ub) : lb;
        const uint32_t mlb = moved_before(bits, W, lb);
        pos = r + (lb - mlb) + ((e - lb) - (moved_before(bits, W, e) - mlb));
    } else {
        return;
    }
    if (pos < n) {
        out_keys[pos] = key;
        out_perm[pos] = idx;
    }
}

// ---------------------------------------------------------------- small models: one kernel
// Keys, stable sort and cell starts of a model of up to kSmallSort particles in one cluster of 8 or
// 16 blocks, everything in (distributed) shared memory: a key and an index, 16 bits each, in one
// word. The incremental sort and the cell starts cost such a model six launches and 39 to 44 us under
// ncu, nearly all of it launch and dependent-load latency (8 bytes a particle take under a
// microsecond to move); this kernel and the gather take 15 us at 5,000 particles, 26 at 47,000 (30
// with eight blocks), 28 at 65,536: block barriers, cluster barriers (five, a microsecond or so each:
// seven made the substep of 17,576 particles 38.5 us instead of 36.7) and the ranking of up to four items
// per thread. More than 65,536 particles would need two words an item.
// Block c holds positions [c S, c S + S) of the array being sorted, S = ceil(n / blocks / 32) 32. Each of one
// or two LSD passes ranks its items as the moved particles' sort does (per-warp histograms, match.any), exchanges
// the blocks' digit counts, and stores every item straight into its place in the owner's shared
// memory. The heads of equal keys are then stored into a table over the keys, and a suffix minimum
// over it gives every key's first position; what a block's last keys take from the blocks after it,
// the element where the owner of the keys changes has stored into its `s_rest`.
constexpr uint32_t kSmallSort = 65536;

template <bool kBatch, bool kHostIn, int kBlocks, int ITEMS>
__global__ void __launch_bounds__(1024, 1)
    k_sort_small(StepLaunch L, const float4* __restrict__ pos, int digit_bits, int passes,
                 uint32_t* __restrict__ skeys, uint32_t* __restrict__ perm, uint32_t* __restrict__ scan,
                 const float* __restrict__ host3, float4* __restrict__ pos_out, float4* __restrict__ aux,
                 const uint32_t* __restrict__ b_of_id, uint32_t* __restrict__ b_next) {
    VFS_CHAINED();
    namespace cg = cooperative_groups;
    constexpr uint32_t kSeg = 1024u * ITEMS;
    extern __shared__ uint32_t s_mem[];
    uint32_t* const s_buf = s_mem;                      // [2][kSeg] key << 16 | index
    uint32_t* const s_head = s_mem + 2 * kSeg;          // [kSeg] first position of each key of this block's
    uint32_t* const s_whist = s_mem + 3 * kSeg;         // [32][256] per-warp digit counts, then prefixes
    __shared__ uint32_t s_cnt[256], s_base[256], s_warp[32], s_rest;
    __shared__ float s_p[kHostIn ? 3072 : 1];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t n = L.total, c = cluster.block_rank();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr uint32_t kUnit = 32u * kBlocks;
    const uint32_t S = ((n + kUnit - 1u) / kUnit) * 32u;
    const uint32_t magic = 0xFFFFFFFFu / S + 1u;  // pos / S = umulhi(pos, magic) for pos < 2^16
    const uint32_t first = c * S, mine = first < n ? min(S, n - first) : 0u;
    const uint32_t lt = (1u << lane) - 1u;
    // Keys of the block's particles, in index order.
    for (uint32_t t0 = 0; t0 < mine; t0 += 1024u) {
        const uint32_t t = t0 + tid, i = first + t;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (kHostIn) {
            // Page-locked positions of a host round trip, stored as the state upload stores them
            // (see k_keys_flags): coalesced through shared memory.
            const uint32_t m3 = 3u * min(1024u, mine - t0);
            const float* src = host3 + 3 * (size_t)(first + t0);
            __syncthreads();
            for (uint32_t k = tid; k < m3; k += 1024u) s_p[k] = src[k];
            __syncthreads();
            if (t < mine) {
                x = make_float4(s_p[3u * tid], s_p[3u * tid + 1u], s_p[3u * tid + 2u], __uint_as_float(i));
                if (b_next) {
                    const uint32_t old = __float_as_uint(pos_out[i].w);
                    b_next[i] = old < n ? b_of_id[old] : 0u;
                }
                pos_out[i] = x;
                aux[i].z = 0.0f;
            }
        } else if (t < mine) {
            x = __ldg(pos + i);
        }
        if (t < mine) s_buf[t] = particle_key<kBatch>(L, i, x) << 16 | i;
    }
    for (uint32_t k = tid; k < S; k += 1024u) s_head[k] = 0xFFFFFFFFu;
    if (tid == 0u) s_rest = n;
    const uint32_t bins = 1u << digit_bits, mask = bins - 1u;
    uint32_t* cur = s_buf;
    uint32_t* nxt = s_buf + kSeg;
    for (int ps = 0; ps < passes; ps++) {
        const int shift = 16 + ps * digit_bits;
        for (uint32_t k = tid; k < 32u * bins; k += 1024u) s_whist[k] = 0u;
        __syncthreads();
        uint32_t v[ITEMS], r[ITEMS];
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            const uint32_t t = (warp * ITEMS + it) * 32u + lane;
            const bool valid = t < mine;
            v[it] = valid ? cur[t] : 0u;
            const uint32_t d = valid ? (v[it] >> shift) & mask : bins;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            const uint32_t pre = (uint32_t)__popc(peers & lt);
            uint32_t prev = 0u;
            if (valid) prev = s_whist[warp * bins + d];
            __syncwarp();
            if (valid && pre == 0u) s_whist[warp * bins + d] = prev + (uint32_t)__popc(peers);
            __syncwarp();
            r[it] = prev + pre;
        }
        __syncthreads();
        // Per digit, the prefix over the warps: four threads a digit, eight warps each.
        if (tid < 4u * bins) {
            const uint32_t d = tid >> 2, w0 = 8u * (tid & 3u);
            uint32_t sum = 0u;
#pragma unroll
            for (uint32_t w = 0; w < 8u; w++) sum += s_whist[(w0 + w) * bins + d];
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o, 4);
                if ((int)(tid & 3u) >= o) incl += t;
            }
            uint32_t run = incl - sum;
#pragma unroll
            for (uint32_t w = 0; w < 8u; w++) {
                const uint32_t t = s_whist[(w0 + w) * bins + d];
                s_whist[(w0 + w) * bins + d] = run;
                run += t;
            }
            if ((tid & 3u) == 3u) s_cnt[d] = run;
        }
        cluster.sync();
        // A digit's first position: all blocks' smaller digits, then the earlier blocks' same digit.
        uint32_t lower = 0u, total = 0u;
        if (tid < bins) {
#pragma unroll
            for (uint32_t b = 0; b < (uint32_t)kBlocks; b++) {
                const uint32_t k = cluster.map_shared_rank(s_cnt, b)[tid];
                lower += b < c ? k : 0u;
                total += k;
            }
        }
        uint32_t incl = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += t;
        }
        if (lane == 31u) s_warp[warp] = incl;
        __syncthreads();
        if (tid < bins) {
            uint32_t before = 0u;
            for (uint32_t w = 0; w < warp; w++) before += s_warp[w];  // at most 7
            s_base[tid] = before + incl - total + lower;
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < ITEMS; it++) {
            if ((warp * ITEMS + it) * 32u + lane < mine) {
                const uint32_t d = (v[it] >> shift) & mask;
                const uint32_t to = s_base[d] + s_whist[warp * bins + d] + r[it];
                const uint32_t b = __umulhi(to, magic);
                cluster.map_shared_rank(nxt, b)[to - b * S] = v[it];
            }
        }
        cluster.sync();
        uint32_t* const t = cur;
        cur = nxt;
        nxt = t;
    }
    // The sorted arrays; the heads of equal keys into the table of their keys' owner (owner b holds keys
    // [b S, b S + S)); and, where the owner changes, the position into the owners passed: the first
    // past all their keys.
    for (uint32_t t = tid; t < mine; t += 1024u) {
        const uint32_t i = first + t, key = cur[t] >> 16;
        skeys[i] = key;
        perm[i] = cur[t] & 0xFFFFu;
        uint32_t before = 0xFFFFFFFFu;
        if (t) before = cur[t - 1u] >> 16;
        else if (i) before = cluster.map_shared_rank(cur, c - 1u)[S - 1u] >> 16;
        if (key != before) {
            const uint32_t b = __umulhi(key, magic);
            cluster.map_shared_rank(s_head, b)[key - b * S] = i;
            for (uint32_t q = i ? __umulhi(before, magic) : 0u; q < b; q++) *cluster.map_shared_rank(&s_rest, q) = i;
        }
    }
    cluster.sync();  // the last use of other blocks' shared memory is behind it
    // scan[k] = the smallest head of the keys >= k (n when none): a suffix minimum, ITEMS keys a thread.
    uint32_t h[ITEMS];
    uint32_t low = 0xFFFFFFFFu;
#pragma unroll
    for (int it = ITEMS - 1; it >= 0; it--) {
        const uint32_t k = tid * ITEMS + it;
        if (k < S) low = min(low, s_head[k]);
        h[it] = low;
    }
    uint32_t after = low;  // over this thread and the later ones of its warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_down_sync(0xffffffffu, after, o);
        if (lane + (uint32_t)o < 32u) after = min(after, t);
    }
    if (lane == 0u) s_warp[warp] = after;
    __syncthreads();
    uint32_t rest = s_rest;
    for (uint32_t w = warp + 1u; w < 32u; w++) rest = min(rest, s_warp[w]);
    const uint32_t later = __shfl_down_sync(0xffffffffu, after, 1);
    if (lane < 31u) rest = min(rest, later);
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t k = tid * ITEMS + it;
        if (k < S && first + k < n) scan[first + k] = min(h[it], rest);
    }
    if (c == 0u && tid == 0u) scan[n] = n;
}

constexpr int kSortBlock = 256;

template <int ITEMS>
cudaError_t launch_onesweep_t(uint32_t n, const SortConfig& sc, const SortScratch& scr, int pass,
                              const uint32_t* kin, const uint32_t* vin, uint32_t* kout,
                              uint32_t* vout, const uint32_t* n_dev, cudaStream_t s) {
    // The few moved particles of a substep (*n_dev of n) are one tile's chain or a few, where match.any is
    // shorter than ballots: us a substep by ballots and match.any, 66,751 particles 88.7 / 85.7, 83,607
    // 84.7 / 79.8, 150,000 172.5 / 168.7, 1M 646.6 / 644.6. Above kMatchMost that is lost beside a substep
    // of milliseconds, and a whole new state (every particle moved) sorts the sooner by ballots.
    constexpr uint32_t kMatchMost = 1u << 21;
    auto* const kernel = n_dev && n <= kMatchMost ? k_onesweep<kSortBlock, ITEMS, true> : k_onesweep<kSortBlock, ITEMS, false>;
    launch_chained(kernel, sc.tiles, kSortBlock, 0, s, kin, vin, kout, vout, n, pass * sc.digit_bits, sc.bins, scr.ghist + pass * sc.bins,
        scr.counters + pass, scr.status + (size_t)pass * sc.tiles * sc.bins, scr.err, n_dev);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_lookback_selftest(bool published, uint32_t spin_limit, uint32_t* d_work,
                                     uint32_t* err, cudaStream_t s) {
    constexpr int bins = 32;
    uint32_t h[2 * bins];
    for (int b = 0; b < bins; b++) {
        h[b] = published ? (kFlagPrefix | (uint32_t)(b + 1)) : 0u;  // tile 0
        h[bins + b] = 0u;                                           // tile 1 (the waiter)
    }
    cudaError_t e = cudaMemcpyAsync(d_work, h, sizeof(h), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    e = cudaStreamSynchronize(s);  // h is a stack buffer
    if (e != cudaSuccess) return e;
    k_lookback_selftest<<<1, bins, 0, s>>>(d_work, bins, spin_limit, d_work + 2 * bins, err);
    return cudaGetLastError();
}


int key_bits_for(uint32_t max_key) {
    int bits = 1;
    while (bits < 32 && (((uint64_t)1 << bits) <= (uint64_t)max_key)) bits++;
    return bits;
}

SortConfig make_sort_config(uint32_t n, int digit_bits, int tile_items, int key_bits) {
    SortConfig c{};
    if (digit_bits < 4) digit_bits = 4;
    if (digit_bits > 8) digit_bits = 8;
    if (tile_items != 8 && tile_items != 12 && tile_items != 16) tile_items = 16;
    // Spatial-hash keys are < n.
    const int bits = key_bits > 0 ? (key_bits > 32 ? 32 : key_bits)
                                  : key_bits_for(n > 0 ? n - 1u : 0u);
    while ((bits + digit_bits - 1) / digit_bits > kMaxSortPasses) digit_bits++;  // <= 8 covers 32 bits
    c.digit_bits = digit_bits;
    c.passes = (bits + digit_bits - 1) / digit_bits;
    c.bins = 1 << digit_bits;
    c.tile = kSortBlock * tile_items;
    c.tiles = (uint32_t)(((uint64_t)n + c.tile - 1) / c.tile);
    if (c.tiles == 0) c.tiles = 1;
    c.delta_blocks = (uint32_t)(((uint64_t)n + kDeltaTile - 1u) / kDeltaTile);
    if (c.delta_blocks == 0) c.delta_blocks = 1;
    return c;
}

size_t sort_scratch_words(const SortConfig& c) {
    return (size_t)c.passes * c.bins + (size_t)c.passes + (size_t)c.passes * c.tiles * c.bins +
           1u + (size_t)c.delta_blocks;
}


cudaError_t launch_keys_delta(const StepLaunch& L, const float4* pos, const uint32_t* pkeys,
                              uint32_t* mkeys, uint32_t* midx, uint32_t* bits,
                              const SortConfig& sc, const SortScratch& scr, cudaStream_t s,
                              const float* host3, float4* pos_out, float4* aux,
                              const uint32_t* b_of_id, uint32_t* b_next) {
    if (L.total == 0) return cudaSuccess;
    const uint32_t tiles = sc.delta_blocks, W = (L.total + 31u) >> 5;
    if (L.n_scenes > 1)
        launch_chained(k_keys_flags<true, false>, tiles, 256, 0, s, L, pos, pkeys, bits, sc.passes, sc.digit_bits,
                                                        scr.ghist, scr.dstatus, nullptr, nullptr, nullptr,
                                                        nullptr, nullptr);
    else if (host3)
        launch_chained(k_keys_flags<false, true>, tiles, 256, 0, s, L, pos, pkeys, bits, sc.passes, sc.digit_bits,
                                                        scr.ghist, scr.dstatus, host3, pos_out, aux,
                                                        b_of_id, b_next);
    else
        launch_chained(k_keys_flags<false, false>, tiles, 256, 0, s, L, pos, pkeys, bits, sc.passes, sc.digit_bits,
                                                         scr.ghist, scr.dstatus, nullptr, nullptr, nullptr,
                                                         nullptr, nullptr);
    if (tiles <= kFoldTiles) {
        if (L.n_scenes > 1)
            launch_chained(k_moved_compact<true, true>, tiles, 256, 0, s, L, pos, bits, scr.dstatus, mkeys, midx, scr.mcount);
        else
            launch_chained(k_moved_compact<false, true>, tiles, 256, 0, s, L, pos, bits, scr.dstatus, mkeys, midx, scr.mcount);
        return cudaGetLastError();
    }
    launch_chained(k_tile_scan, 1, 1024, 0, s, tiles, scr.dstatus, bits, W, scr.mcount);
    if (L.n_scenes > 1)
        launch_chained(k_moved_compact<true, false>, tiles, 256, 0, s, L, pos, bits, scr.dstatus, mkeys, midx, scr.mcount);
    else
        launch_chained(k_moved_compact<false, false>, tiles, 256, 0, s, L, pos, bits, scr.dstatus, mkeys, midx, scr.mcount);
    return cudaGetLastError();
}

bool small_sort(uint32_t total) { return total <= kSmallSort; }

namespace {
// A cluster of 16 blocks is more than every device need schedule: asked once per device.
template <bool kBatch, bool kHostIn, int kBlocks, int ITEMS>
cudaError_t sort_small_items(const StepLaunch& L, const float4* pos, int bits, int passes, uint32_t* skeys,
                             uint32_t* perm, uint32_t* scan, const float* host3, float4* pos_out, float4* aux,
                             const uint32_t* b_of_id, uint32_t* b_next, cudaStream_t s) {
    auto* const kernel = k_sort_small<kBatch, kHostIn, kBlocks, ITEMS>;
    cudaLaunchAttribute attrs[2] = {};
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim = {kBlocks, 1, 1};
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see vfs_chain.h
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kBlocks);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = (3u * 1024u * ITEMS + 32u * 256u) * sizeof(uint32_t);
    cfg.stream = s;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    static std::atomic<int> state[16];  // 0: not asked, 1: this cluster size, 2: eight blocks instead
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int st = dev < 16 ? state[dev].load(std::memory_order_relaxed) : 0;
    if (st == 0) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
        if (e != cudaSuccess) return e;
        st = 1;
        if (kBlocks > 8) {
            int clusters = 0;
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
                cudaGetLastError();
                st = 2;
            }
        }
        if (dev < 16) state[dev].store(st, std::memory_order_relaxed);
    }
    if constexpr (kBlocks > 8) {
        if (st == 2)
            return sort_small_items<kBatch, kHostIn, 8, 2 * ITEMS>(L, pos, bits, passes, skeys, perm, scan, host3,
                                                                   pos_out, aux, b_of_id, b_next, s);
    }
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, L, pos, bits, passes, skeys, perm, scan, host3, pos_out, aux, b_of_id, b_next);
}

template <bool kBatch, bool kHostIn>
cudaError_t sort_small(const StepLaunch& L, const float4* pos, uint32_t* skeys, uint32_t* perm, uint32_t* scan,
                       const float* host3, float4* pos_out, float4* aux, const uint32_t* b_of_id,
                       uint32_t* b_next, cudaStream_t s) {
    // At least 3 bits a digit: the kernel's four threads a digit then fill whole warps.
    const int key_bits = key_bits_for(L.total - 1u), passes = (key_bits + 7) / 8;
    const int bits = std::max(3, (key_bits + passes - 1) / passes);
    if (L.total <= 8192u) return sort_small_items<kBatch, kHostIn, 8, 1>(L, pos, bits, passes, skeys, perm, scan, host3, pos_out, aux, b_of_id, b_next, s);
    if (L.total <= 16384u) return sort_small_items<kBatch, kHostIn, 16, 1>(L, pos, bits, passes, skeys, perm, scan, host3, pos_out, aux, b_of_id, b_next, s);
    if (L.total <= 32768u) return sort_small_items<kBatch, kHostIn, 16, 2>(L, pos, bits, passes, skeys, perm, scan, host3, pos_out, aux, b_of_id, b_next, s);
    return sort_small_items<kBatch, kHostIn, 16, 4>(L, pos, bits, passes, skeys, perm, scan, host3, pos_out, aux, b_of_id, b_next, s);
}
}  // namespace

cudaError_t launch_sort_small(const StepLaunch& L, const float4* pos, uint32_t* skeys, uint32_t* perm,
                              uint32_t* cell_scan, cudaStream_t s, const float* host3, float4* pos_out,
                              float4* aux, const uint32_t* b_of_id, uint32_t* b_next) {
    if (L.total == 0) return cudaSuccess;
    if (L.n_scenes > 1) return sort_small<true, false>(L, pos, skeys, perm, cell_scan, nullptr, nullptr, nullptr, nullptr, nullptr, s);
    if (host3) return sort_small<false, true>(L, pos, skeys, perm, cell_scan, host3, pos_out, aux, b_of_id, b_next, s);
    return sort_small<false, false>(L, pos, skeys, perm, cell_scan, nullptr, nullptr, nullptr, nullptr, nullptr, s);
}

cudaError_t launch_reorder(const StepLaunch& L, uint32_t n, const uint32_t* perm, const float4* pos_in,
                           const float4* vel_in, float4* pos_out, float4* vel_out, const SkinLists& sk,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    launch_chained(k_reorder, (n + 127u) / 128u, 128, 0, s, L, n, perm, pos_in, vel_in, pos_out, vel_out, sk.b_of_id, sk.xcur,
                                                sk.x_build, sk.stale, sk.ctl, sk.wcount);
    return cudaGetLastError();
}

cudaError_t launch_merge(uint32_t n, const uint32_t* pkeys, const uint32_t* bits,
                         const uint32_t* mcount, const uint32_t* mk, const uint32_t* mi,
                         uint32_t* out_keys, uint32_t* out_perm, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint64_t threads = 2ull * n;
    launch_chained(k_merge, (unsigned)((threads + 255u) / 256u), 256, 0, s, n, pkeys, bits, mcount, mk, mi,
                                                                 out_keys, out_perm);
    return cudaGetLastError();
}

cudaError_t launch_digit_hist(const uint32_t* keys, uint32_t n, const SortConfig& sc,
                              uint32_t* ghist, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    // Few blocks: each adds its passes x bins counters to the global ones with atomics (1M keys: 15 us
    // with 1,216 blocks, 6 with 304).
    uint32_t blocks = (n + 1023u) / 1024u;
    if (blocks > 152u * 2u) blocks = 152u * 2u;
    k_digit_hist<<<blocks, 256, 0, s>>>(keys, n, sc.passes, sc.digit_bits, ghist);
    return cudaGetLastError();
}

cudaError_t launch_sort_pass(uint32_t n, const SortConfig& sc, const SortScratch& scr, int pass,
                             const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout,
                             const uint32_t* n_dev, cudaStream_t s) {
    const int items = sc.tile / kSortBlock;
    if (items == 8) return launch_onesweep_t<8>(n, sc, scr, pass, kin, vin, kout, vout, n_dev, s);
    if (items == 12) return launch_onesweep_t<12>(n, sc, scr, pass, kin, vin, kout, vout, n_dev, s);
    return launch_onesweep_t<16>(n, sc, scr, pass, kin, vin, kout, vout, n_dev, s);
}

cudaError_t launch_sort(uint32_t n, const SortConfig& sc, const SortScratch& scr, uint32_t* keys,
                        uint32_t* keys_alt, uint32_t* vals, uint32_t* vals_alt,
                        uint32_t** sorted_keys, uint32_t** sorted_perm, cudaStream_t s,
                        bool vals_given, const uint32_t* n_dev) {
    const uint32_t* kin = keys;
    const uint32_t* vin = vals_given ? vals : nullptr;  // nullptr: pass 0 ranks (key, index)
    uint32_t* kout = keys_alt;
    uint32_t* vout = vals_alt;
    for (int pass = 0; pass < sc.passes; pass++) {
        const cudaError_t e = launch_sort_pass(n, sc, scr, pass, kin, vin, kout, vout, n_dev, s);
        if (e != cudaSuccess) return e;
        kin = kout;
        vin = vout;
        kout = (kout == keys_alt) ? keys : keys_alt;
        vout = (vout == vals_alt) ? vals : vals_alt;
    }
    *sorted_keys = const_cast<uint32_t*>(kin);
    *sorted_perm = const_cast<uint32_t*>(vin);
    return cudaSuccess;
}

namespace {
__global__ void __launch_bounds__(256)
    k_vel_records(uint32_t n, const uint32_t* __restrict__ perm, const float* __restrict__ vel3,
                  float4* __restrict__ vel_out, const float4* __restrict__ aux,
                  float4* __restrict__ rec) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    uint32_t src = perm[i];
    if (src >= n) src = i;  // only after a reported sort failure, as in the cell pass
    const float* v = vel3 + 3 * (size_t)src;
    const float vx = __ldg(v), vy = __ldg(v + 1), vz = __ldg(v + 2);
    vel_out[i] = make_float4(vx, vy, vz, 0.0f);
    rec[2 * (size_t)i + 1] = make_float4(vx, vy, vz, __ldg(aux + i).y);
}
}  // namespace

cudaError_t launch_vel_records(uint32_t n, const uint32_t* perm, const float* vel3,
                               float4* vel_out, const float4* aux, float4* rec, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_vel_records<<<(n + 255u) / 256u, 256, 0, s>>>(n, perm, vel3, vel_out, aux, rec);
    return cudaGetLastError();
}

// SMs of the current device (0 if unknown), cached per device.
static int sm_count() {
    static std::atomic<int> sms[16];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
    int n = sms[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// A walk of n particles has less than a resident wave of blocks (768 to 896 threads an SM in most of its
// shapes). Let in while the kernel before it fills the SMs unevenly, they crowd a few of them.
static bool walk_below_wave(uint32_t n) { return n < (uint32_t)sm_count() * 768u; }

cudaError_t launch_cells_reorder(const StepLaunch& L, uint32_t n, const uint32_t* skeys, const uint32_t* perm,
                                 uint32_t* cell_scan, const float4* pos_in, const float4* vel_in,
                                 float4* pos_out, float4* vel_out, uint32_t* zero,
                                 uint32_t zero_words, uint32_t* pkeys_out, uint32_t* guess,
                                 const SkinLists& sk, const KernelConfig& kc, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    // Without lists the walk comes next: us a substep let in early and late, 71,402 particles 110.4 /
    // 99.4, 90,000 112.6 / 109.4, 110,000 117.4 / 116.8, 150,000 173.7 / 175.4.
    const bool late = !sk.list && walk_below_wave(n);
    switch (kc.cell_block) {
        case 128:
            launch_chained(k_cells_reorder<128>, (n + 128u) / 128u, 128, 0, s, L, n, skeys, perm, cell_scan, pos_in,
                                                                 vel_in, pos_out, vel_out, zero, zero_words, pkeys_out, guess, sk.b_of_id, sk.xcur, sk.x_build, sk.stale, sk.ctl, sk.wcount, late);
            break;
        case 512:
            launch_chained(k_cells_reorder<512>, (n + 512u) / 512u, 512, 0, s, L, n, skeys, perm, cell_scan, pos_in,
                                                                 vel_in, pos_out, vel_out, zero, zero_words, pkeys_out, guess, sk.b_of_id, sk.xcur, sk.x_build, sk.stale, sk.ctl, sk.wcount, late);
            break;
        default:
            launch_chained(k_cells_reorder<256>, (n + 256u) / 256u, 256, 0, s, L, n, skeys, perm, cell_scan, pos_in,
                                                                 vel_in, pos_out, vel_out, zero, zero_words, pkeys_out, guess, sk.b_of_id, sk.xcur, sk.x_build, sk.stale, sk.ctl, sk.wcount, late);
    }
    return cudaGetLastError();
}

constexpr size_t kTileSmemBytes = kTileWarps * sizeof(TileSmem);

// Blocks of one resident wave of a tile kernel over `total` particles (fewer when they cover them).
// Residency per SM is asked of the occupancy calculator once per kernel and device.
template <typename Kernel>
cudaError_t tile_blocks(Kernel* kernel, std::atomic<int>* per_sm, uint32_t total, uint32_t& blocks) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int r = dev < 16 ? per_sm[dev].load(std::memory_order_relaxed) : 0;
    if (r == 0) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemBytes);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kernel, kTileWarps * 32, kTileSmemBytes);
        if (e != cudaSuccess) return e;
        if (r < 1) r = 1;
        if (dev < 16) per_sm[dev].store(r, std::memory_order_relaxed);
    }
    const int sms = sm_count();
    blocks = (total + kTileWarps * 32 - 1) / (kTileWarps * 32);
    if (sms > 0) blocks = min(blocks, (uint32_t)sms * (uint32_t)r);
    return cudaSuccess;
}

template <bool kBatch>
cudaError_t launch_build(const StepLaunch& L, const float4* pos, const uint32_t* cell_scan,
                         const SkinLists& sk, cudaStream_t s) {
    static std::atomic<int> per_sm[16];
    uint32_t blocks = 0u;
    const cudaError_t e = tile_blocks(k_skin_build<kBatch>, per_sm, L.total, blocks);
    if (e != cudaSuccess) return e;
    launch_chained(k_skin_build<kBatch>, blocks, kTileWarps * 32, kTileSmemBytes, s, L, pos, cell_scan, sk);
    return cudaGetLastError();
}

cudaError_t launch_walk_queue(const StepLaunch& L, const float4* pos, const float4* vel, float4* rec,
                              const uint32_t* cell_scan, float4* aux, float4* bnd, uint32_t* nbr,
                              uint32_t* nbr_count, const SkinLists& sk, uint32_t* sched, cudaStream_t s) {
    static std::atomic<int> per_sm[16];
    uint32_t blocks = 0u;
    const cudaError_t e = tile_blocks(k_walk_queue, per_sm, L.total, blocks);
    if (e != cudaSuccess) return e;
    launch_chained(k_walk_queue, blocks, kTileWarps * 32, kTileSmemBytes, s, L, pos, vel, rec, cell_scan, aux, bnd, nbr,
                                                                 nbr_count, sk, sched);
    return cudaGetLastError();
}

// One resident wave of the walk kernel: its blocks take runs of slots until none is left, so
// more blocks would only start after the work is gone. Residency per SM is asked of the
// occupancy calculator once per instantiation.
template <bool kBatch, int B, int M>
cudaError_t launch_walk(const StepLaunch& L, const float4* pos, const float4* vel, float4* rec,
                        const uint32_t* cell_scan, float4* aux, float4* bnd, uint32_t* nbr,
                        uint32_t* nbr_count, const SkinLists& sk, uint32_t* sched, cudaStream_t s) {
    static std::atomic<int> per_sm{0};
    int r = per_sm.load(std::memory_order_relaxed);
    if (r == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_walk<kBatch, B, M>, B, 0) == cudaSuccess && r > 0)
            per_sm.store(r, std::memory_order_relaxed);
        else
            r = M;
    }
    const int sms = sm_count();
    const uint32_t all_blocks = (L.total + B - 1) / B;
    const uint32_t blocks = sms > 0 ? min(all_blocks, (uint32_t)sms * (uint32_t)r) : all_blocks;
    launch_chained(k_walk<kBatch, B, M>, blocks, B, 0, s, L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, sched);
    return cudaGetLastError();
}

// The walk in the density pass's launch shape.
template <bool kBatch>
cudaError_t launch_walk_shaped(int shape, const StepLaunch& L, const float4* pos, const float4* vel,
                               float4* rec, const uint32_t* cell_scan, float4* aux, float4* bnd,
                               uint32_t* nbr, uint32_t* nbr_count, const SkinLists& sk, uint32_t* sched,
                               cudaStream_t s) {
    switch (shape) {
        case kNbr128x8: return launch_walk<kBatch, 128, 8>(L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, sched, s);
        case kNbr96x8: return launch_walk<kBatch, 96, 8>(L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, sched, s);
        case kNbr64x12: return launch_walk<kBatch, 64, 12>(L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, sched, s);
        default: return launch_walk<kBatch, 128, 6>(L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, sched, s);
    }
}

template <int B, int M>
void force_shape(const StepLaunch& L, const float4* pos, const float4* vel, const float4* aux,
                 const float4* rec, const float4* bnd, const uint32_t* cell_scan, const uint32_t* nbr,
                 const uint32_t* nbr_count, float4* pos_out, float4* vel_out, float4* acc_out,
                 const SkinLists& sk, cudaStream_t s, const HostOut& ho) {
    const uint32_t blocks = (L.total + B - 1) / B;
    if (L.n_scenes > 1)
        launch_chained(k_force<true, B, M>, blocks, B, 0, s, L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count,
                                                 pos_out, vel_out, acc_out, sk.stale, sk.ctl,
                                                 sk.wcount + 1, HostOut{});
    else  // shared memory only for host outputs: without them the whole on-chip memory stays L1
        launch_chained(k_force<false, B, M>, blocks, B, ho.any() ? 7 * B * sizeof(float) : 0, s, L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count, pos_out, vel_out, acc_out,
            sk.stale, sk.ctl, sk.wcount + 1, ho);
}

bool planes_mode(uint32_t total) {
    const int n = sm_count();
    return n > 0 && (uint64_t)total * 3u <= (uint64_t)n * 768u;
}

cudaError_t launch_density(const StepLaunch& L, const float4* pos, const float4* vel, float4* rec,
                           const uint32_t* cell_scan, float4* aux, float4* bnd, uint32_t* nbr,
                           uint32_t* nbr_count, const SkinLists& sk, uint32_t* walk_sched,
                           const KernelConfig& kc, cudaStream_t s) {
    if (L.total == 0) return cudaSuccess;
    if (planes_mode(L.total)) {
        const uint32_t blocks = (L.total + 29u) / 30u;
        if (L.n_scenes > 1)
            launch_chained(k_density_planes<true>, blocks, kPlaneBlock, 0, s, L, pos, vel, rec, cell_scan, aux, bnd,
                                                                  nbr, nbr_count);
        else
            launch_chained(k_density_planes<false>, blocks, kPlaneBlock, 0, s, L, pos, vel, rec, cell_scan, aux, bnd,
                                                                   nbr, nbr_count);
        return cudaGetLastError();
    }
    const bool batch = L.n_scenes > 1;
    if (sk.list) {
        // Skin lists: the build where it is due, then the list pass, then the walk of the queue it
        // leaves (a batch's below).
        cudaError_t e = batch ? launch_build<true>(L, pos, cell_scan, sk, s) : launch_build<false>(L, pos, cell_scan, sk, s);
        if (e != cudaSuccess) return e;
        const uint32_t lb = (L.total + kListBlock - 1) / kListBlock;
        if (batch) {
            // The walk comes next, as after launch_cells_reorder's pass: us a substep let in early and late,
            // 13 scenes of 1,579 to 23,237 particles 184 / 172, 8 of up to 20,766 232 / 223 (the batches' host
            // copies included).
            const bool late = walk_below_wave(L.total);
            launch_chained(k_density_list<true>, lb, kListBlock, 0, s, L, pos, vel, rec, aux, bnd, nbr, nbr_count, sk, late);
        } else {
            launch_chained(k_density_list<false>, lb, kListBlock, 0, s, L, pos, vel, rec, aux, bnd, nbr, nbr_count, sk, false);
            e = launch_walk_queue(L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, walk_sched, s);
            if (e != cudaSuccess) return e;
        }
    }
    return batch ? launch_walk_shaped<true>(kc.nbr_shape, L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, walk_sched, s)
                 : launch_walk_shaped<false>(kc.nbr_shape, L, pos, vel, rec, cell_scan, aux, bnd, nbr, nbr_count, sk, walk_sched, s);
}

cudaError_t launch_force(const StepLaunch& L, const float4* pos, const float4* vel,
                         const float4* aux, const float4* rec, const float4* bnd, const uint32_t* cell_scan,
                         const uint32_t* nbr, const uint32_t* nbr_count, float4* pos_out,
                         float4* vel_out, float4* acc_out, const SkinLists& sk,
                         const KernelConfig& kc, cudaStream_t s, const HostOut& ho) {
    if (L.total == 0) return cudaSuccess;
    switch (kc.force_shape) {
        case kNbr128x8:
            force_shape<128, 8>(L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count, pos_out, vel_out, acc_out, sk, s, ho);
            break;
        case kNbr96x8:
            force_shape<96, 8>(L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count, pos_out, vel_out, acc_out, sk, s, ho);
            break;
        case kNbr64x12:
            force_shape<64, 12>(L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count, pos_out, vel_out, acc_out, sk, s, ho);
            break;
        default:
            force_shape<128, 6>(L, pos, vel, aux, rec, bnd, cell_scan, nbr, nbr_count, pos_out, vel_out, acc_out, sk, s, ho);
    }
    return cudaGetLastError();
}

cudaError_t launch_offsets(uint32_t n, uint32_t off, const uint32_t* cell_scan, uint32_t* offsets,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_offsets<<<(n + 255u) / 256u, 256, 0, s>>>(n, off, cell_scan, offsets);
    return cudaGetLastError();
}

}  // namespace vfs
