// ref_kernels.cu -- the reference engine's math on sm_100a, FP64 as in the
// reference (all particle and voxel state is CudaVec<double>).
//
// Each kernel restates one reference kernel with the same arithmetic so that
// integer outputs are bit-exact and floating-point outputs agree to rounding.
// What changes is the execution shape: one CTA of 128 threads per occupied
// root cell instead of 32, the three axes of P2G/G2P/divergence/projection in
// one launch instead of three, the voxel-activation predicate evaluated once
// (its 512-bit mask is kept for the compaction) instead of twice, and the
// tile-local red-black SOR iterated in shared memory for a whole convergence
// check interval instead of two launches per iteration.
//
// The reference's behaviours that change results are kept:
//   - the activation solid test takes the tile origin from the key of
//     particle blockIdx.x (not the node's first particle) and computes the
//     voxel's y index as (i % 8 * 8) / 8, which equals its x index
//     (particles.cu:99,118);
//   - the z-apron copy of the divergence indexes x with the z coordinate
//     (voxelSolveFunctions.cu:85);
//   - the y-row table stores root-cell ids that are later compared with node
//     counts (particleToGridFunctions.cu:369, voxelSolveFunctions.cu:138-156);
//   - G2P skips voxels whose velocity is exactly zero (particles.cu:649).
#include "common.cuh"
#include "ref_kernels.cuh"
#include <curand_kernel.h>

namespace flip {

__device__ __forceinline__ uint32_t sat_u32_d(double v) {
    return (uint32_t)__double2uint_rz(v);  // saturating: negative/NaN -> 0
}
__device__ __forceinline__ uint32_t sat_u32_f(float v) { return (uint32_t)__float2uint_rz(v); }

__device__ __forceinline__ double ref_dist(double dx, double dy, double dz) {
    return sqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
}
__device__ __forceinline__ double ref_scw(const flip_grid& g) { return (double)(g.cellSize / 4.0f); }
__device__ __forceinline__ double ref_local(double p, float neg, uint32_t gid, float cell, double scw) {
    double t = p - (double)neg;
    float prod = __fmul_rn((float)gid, cell);
    t = t - (double)prod;
    return t + 2.0 * scw;
}
__device__ __forceinline__ void ref_decompose(uint32_t key, const flip_grid& g, uint32_t& gx, uint32_t& gy, uint32_t& gz) {
    uint32_t xy = g.sizeX * g.sizeY;
    uint32_t m = key % xy;
    gz = key / xy;
    gy = m / g.sizeX;
    gx = m % g.sizeX;
}

// ----------------------------------------------------------------- keys
// rootCell (particleToGridFunctions.cu:19-45)
__global__ void ref_keys_kernel(double* __restrict__ px, double* __restrict__ py, double* __restrict__ pz, uint64_t n,
                                flip_grid g, uint32_t* __restrict__ keys, uint32_t* __restrict__ idx) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float ux = fmaf((float)g.sizeX, g.cellSize, g.negX);
    const float uy = fmaf((float)g.sizeY, g.cellSize, g.negY);
    const float uz = fmaf((float)g.sizeZ, g.cellSize, g.negZ);
    double x = px[i], y = py[i], z = pz[i];
    if (x < (double)g.negX) { x = g.negX; px[i] = x; } else if (x > (double)ux) { x = ux; px[i] = x; }
    if (y < (double)g.negY) { y = g.negY; py[i] = y; } else if (y > (double)uy) { y = uy; py[i] = y; }
    if (z < (double)g.negZ) { z = g.negZ; pz[i] = z; } else if (z > (double)uz) { z = uz; pz[i] = z; }
    uint32_t kx = sat_u32_f(floorf(__double2float_rn(__ddiv_rn(x - (double)g.negX, (double)g.cellSize))));
    uint32_t ky = sat_u32_f(floorf(__double2float_rn(__ddiv_rn(y - (double)g.negY, (double)g.cellSize))));
    uint32_t kz = sat_u32_f(floorf(__double2float_rn(__ddiv_rn(z - (double)g.negZ, (double)g.cellSize))));
    keys[i] = kx + ky * g.sizeX + kz * g.sizeX * g.sizeY;
    if (idx) idx[i] = (uint32_t)i;
}

// ------------------------------------------------------------ y-row table
__global__ void ref_ydim_fill_kernel(uint32_t* table, uint32_t rows, uint32_t nodes) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < rows) table[i] = nodes;
}
// getYDimPositionFirstInRow (particleToGridFunctions.cu:355-372)
__global__ void ref_ydim_rows_kernel(const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes,
                                     flip_grid g, uint32_t* __restrict__ table) {
    uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nodes) return;
    uint32_t prev = idx ? keys[starts[idx - 1]] : nodes;
    uint32_t cur = keys[starts[idx]];
    uint32_t pr = prev / g.sizeX, cr = cur / g.sizeX;
    if (pr != cr && cr < g.sizeY * g.sizeZ) table[cr] = cur;
}

// ------------------------------------------------------- voxel activation
constexpr int kNodeThreads = 128;

// solid test of local voxel i of the tile whose origin comes from particle
// b's key (particles.cu:97-130, 203-247), y index computed as written (Q3)
__device__ __forceinline__ bool ref_tile_solid(uint32_t i, uint32_t gx, uint32_t gy, uint32_t gz, const flip_grid& g) {
    uint32_t vx = i % 8u, vy = (i % 8u * 8u) / 8u, vz = i / 64u;
    uint32_t gvx = gx * 8u + vx, gvy = gy * 8u + vy, gvz = gz * 8u + vz;
    const double fr = 2.0;
    if ((double)gvx < fr || (double)gvy < fr || (double)gvz < fr) return true;
    if ((double)gvx > (double)(g.sizeX * 8u) + fr || (double)gvy > (double)(g.sizeY * 8u) + fr ||
        (double)gvz > (double)(g.sizeZ * 8u) + fr)
        return true;
    return false;
}

// true when ref_tile_solid is false for every voxel of the tile: its voxel
// coordinates run over gx*8 .. gx*8+7 in x and y (the y index is the x index)
// and gz*8 .. gz*8+7 in z, and the test is monotone in each, so the tile's
// corners decide (tiles away from the domain faces, nearly all of them)
__device__ __forceinline__ bool ref_tile_clear(uint32_t gx, uint32_t gy, uint32_t gz, const flip_grid& g) {
    const double fr = 2.0;
    if ((double)(gx * 8u) < fr || (double)(gy * 8u) < fr || (double)(gz * 8u) < fr) return false;
    if ((double)(gx * 8u + 7u) > (double)(g.sizeX * 8u) + fr || (double)(gy * 8u + 7u) > (double)(g.sizeY * 8u) + fr ||
        (double)(gz * 8u + 7u) > (double)(g.sizeZ * 8u) + fr)
        return false;
    return true;
}

// ref_dist(dx, dy, dz) < R without the square root where the sum of squares
// s decides it: the square root is correctly rounded and monotone, so it
// comes out below R exactly when s lies below the square of the midpoint
// between R and the double below R, which is within a relative 2^-52 of R^2.
// s below lo = R^2 (1 - 2^-48) is inside, s at or above hi = R^2 (1 + 2^-48)
// is outside (both bounds hold with the roundings of R^2 and of the
// products); in the band between, the square root decides, as in ref_dist.
__device__ __forceinline__ bool ref_within(double dx, double dy, double dz, double R, double lo, double hi) {
    const double s = fma(dx, dx, fma(dy, dy, dz * dz));
    if (s < lo) return true;
    if (s >= hi) return false;
    return sqrt(s) < R;
}

struct RefLocal {
    double lx, ly, lz;
    uint32_t sx, sy, sz;
};
__device__ __forceinline__ RefLocal ref_particle_local(const double* px, const double* py, const double* pz,
                                                      const uint32_t* keys, uint32_t idx, const flip_grid& g, double scw) {
    uint32_t qx, qy, qz;
    ref_decompose(keys[idx], g, qx, qy, qz);
    RefLocal r;
    r.lx = ref_local(px[idx], g.negX, qx, g.cellSize, scw);
    r.ly = ref_local(py[idx], g.negY, qy, g.cellSize, scw);
    r.lz = ref_local(pz[idx], g.negZ, qz, g.cellSize, scw);
    r.sx = sat_u32_d(floor(r.lx / scw));
    r.sy = sat_u32_d(floor(r.ly / scw));
    r.sz = sat_u32_d(floor(r.lz / scw));
    return r;
}

// The voxels of a particle's stencil in the tile, one word per z plane (bit
// x + 8 y), for the planes sz - 1, sz, sz + 1.
//
// The reference tests 4 x 4 x 4 points at three offsets with FP64 distances.
// In units of the voxel, f = l / scw - s in [0, 1): a point k = -2 .. 1 voxels
// away lies at f - k or, with the half-voxel offset, f - k + 1/2 on each axis,
// so the column k = -2 is never nearer than the radius 2 and 27 points
// remain.  Their distances are taken in FP32: with f rounded once, every
// square and sum stays within 5e-6 of the exact value, so a squared distance
// at least 1e-5 away from 4 decides as the reference's FP64 test does.  The
// column k = -2 counts with its smallest distance, 4 f + (f' - 1/2)^2 +
// (f'' - 1/2)^2 above 4.  False (one particle in about 10^4): a distance
// nearer to 4 than that, or a position outside the root cell; the caller
// then runs the reference's own test.
//
// FP64 tests of all 64 points by a warp per particle took 33 ms for 64M
// particles in 29.5M nodes.
__device__ __forceinline__ bool ref_marks(double qx, double qy, double qz, uint32_t sx, uint32_t sy, uint32_t sz,
                                          unsigned long long (&plane)[3]) {
    const float fx = (float)(qx - (double)sx), fy = (float)(qy - (double)sy), fz = (float)(qz - (double)sz);
    const float kNear = 1e-5f;
    if (sx - 2u > 4u || sy - 2u > 4u || sz - 2u > 4u) return false;
    // squares of f + 1, f, f - 1 (a) and of those plus 1/2 (b), k = -1, 0, 1
    float ax[3], bx[3], ay[3], by[3], az[3], bz[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float o = 1.0f - (float)k;
        ax[k] = (fx + o) * (fx + o) - 4.0f;
        bx[k] = (fx + o + 0.5f) * (fx + o + 0.5f) - 4.0f;
        ay[k] = (fy + o) * (fy + o);
        by[k] = (fy + o + 0.5f) * (fy + o + 0.5f);
        az[k] = (fz + o) * (fz + o);
        bz[k] = (fz + o + 0.5f) * (fz + o + 0.5f);
    }
    const float hx = (fx - 0.5f) * (fx - 0.5f), hy = (fy - 0.5f) * (fy - 0.5f), hz = (fz - 0.5f) * (fz - 0.5f);
    float near = fminf(4.0f * fx + (hy + hz), fminf(4.0f * fy + (hx + hz), 4.0f * fz + (hx + hy)));
    const uint32_t shift = (sx - 1u) + 8u * (sy - 1u);
#pragma unroll
    for (int z = 0; z < 3; ++z) {
        uint32_t bits = 0;  // nine sign bits, the last pushed lowest
#pragma unroll
        for (int y = 2; y >= 0; --y) {
            const float p = by[y] + bz[z], q = fminf(ay[y] + bz[z], by[y] + az[z]);
#pragma unroll
            for (int x = 2; x >= 0; --x) {
                const float d = fminf(ax[x] + p, bx[x] + q);
                near = fminf(near, fabsf(d));
                bits = __funnelshift_l(__float_as_uint(d), bits, 1);
            }
        }
        plane[z] = (unsigned long long)((bits & 7u) | ((bits & 0x38u) << 5) | ((bits & 0x1C0u) << 10)) << shift;
    }
    return near > kNear;
}

// what the particles of one node share: the node's corner and the voxel size
struct RefNode {
    double neg[3], corner[3], scw, R, lo, hi;
};
__device__ __forceinline__ RefNode ref_node(uint32_t key, const flip_grid& g) {
    RefNode N;
    uint32_t gx, gy, gz;
    ref_decompose(key, g, gx, gy, gz);
    N.neg[0] = (double)g.negX; N.neg[1] = (double)g.negY; N.neg[2] = (double)g.negZ;
    N.corner[0] = (double)__fmul_rn((float)gx, g.cellSize);
    N.corner[1] = (double)__fmul_rn((float)gy, g.cellSize);
    N.corner[2] = (double)__fmul_rn((float)gz, g.cellSize);
    N.scw = ref_scw(g);
    N.R = 2.0 * N.scw;
    N.lo = N.R * N.R * (1.0 - 0x1p-48);
    N.hi = N.R * N.R * (1.0 + 0x1p-48);
    return N;
}
// ref_local with the node's part taken once
__device__ __forceinline__ double ref_node_local(const RefNode& N, int a, double p) {
    return ((p - N.neg[a]) - N.corner[a]) + 2.0 * N.scw;
}

// ORs the voxels of particles i0, i0 + step, ... below `last` (each lane its
// own range and node) into the lane's words planes[z * kVoxStride + lane].  The
// whole warp calls; a particle that ref_marks leaves open is tested by all of
// its lanes, two of the 64 points each.
constexpr int kVoxStride = 33;  // words of eight planes, plane-major: lane l's plane z at z * 33 + l
__device__ __forceinline__ void ref_mark_particles(const RefNode& N, uint32_t i0, uint32_t last, uint32_t step,
                                                   const double* __restrict__ px, const double* __restrict__ py,
                                                   const double* __restrict__ pz, unsigned long long* planes) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = i0; __any_sync(0xffffffffu, i < last); i += step) {
        double lx = 0.0, ly = 0.0, lz = 0.0;
        uint32_t sx = 0, sy = 0, sz = 0;
        bool open = false;
        if (i < last) {
            lx = ref_node_local(N, 0, px[i]);
            ly = ref_node_local(N, 1, py[i]);
            lz = ref_node_local(N, 2, pz[i]);
            const double qx = lx / N.scw, qy = ly / N.scw, qz = lz / N.scw;
            sx = sat_u32_d(floor(qx));
            sy = sat_u32_d(floor(qy));
            sz = sat_u32_d(floor(qz));
            unsigned long long plane[3];
            if (ref_marks(qx, qy, qz, sx, sy, sz, plane)) {
#pragma unroll
                for (int k = 0; k < 3; ++k) planes[(sz - 1u + (uint32_t)k) * kVoxStride + lane] |= plane[k];
            } else {
                // The reference's loops run x from sx - 2 while (unsigned) x < sx + 2,
                // so a stencil coordinate below 2 on any axis leaves a particle
                // without marks, and points outside the 8^3 tile never mark.
                open = !(sx < 2u || sy < 2u || sz < 2u);
            }
        }
        const double hs = N.scw / 2.0;
        for (uint32_t rest = __ballot_sync(0xffffffffu, open); rest; rest &= rest - 1u) {
            const int j = __ffs(rest) - 1;
            const double ax = __shfl_sync(0xffffffffu, lx, j), ay = __shfl_sync(0xffffffffu, ly, j), az = __shfl_sync(0xffffffffu, lz, j);
            const uint32_t tx = __shfl_sync(0xffffffffu, sx, j), ty = __shfl_sync(0xffffffffu, sy, j), tz = __shfl_sync(0xffffffffu, sz, j);
#pragma unroll
            for (uint32_t c = lane; c < 64u; c += 32u) {
                const int vx = (int)(tx - 2u) + (int)(c >> 4), vy = (int)(ty - 2u) + (int)((c >> 2) & 3u),
                          vz = (int)(tz - 2u) + (int)(c & 3u);
                if ((uint32_t)vx >= 8u || (uint32_t)vy >= 8u || (uint32_t)vz >= 8u) continue;
                const double dx = ax - vx * N.scw, dy = ay - vy * N.scw, dz = az - vz * N.scw;
                if (ref_within(dx, dy + hs, dz + hs, N.R, N.lo, N.hi) || ref_within(dx + hs, dy, dz + hs, N.R, N.lo, N.hi) ||
                    ref_within(dx + hs, dy + hs, dz, N.R, N.lo, N.hi))
                    atomicOr(&planes[vz * kVoxStride + j], 1ull << (vx + 8 * vy));
            }
        }
        __syncwarp();
    }
}
// ref_tile_solid over a tile: a voxel (x, y, z) is solid when bit x of `row`
// or bit z of `planes` is set (Q3: the y test reads the x index)
struct RefSolid {
    uint32_t row, planes;
    __device__ __forceinline__ unsigned long long plane(uint32_t z) const {
        return (planes >> z) & 1u ? ~0ull : (unsigned long long)row * 0x0101010101010101ull;
    }
    __device__ __forceinline__ uint32_t at(uint32_t id) const { return ((row >> (id & 7u)) | (planes >> (id >> 6))) & 1u; }
};
__device__ __forceinline__ RefSolid ref_solid(uint32_t key, const flip_grid& g) {
    uint32_t gx, gy, gz;
    ref_decompose(key, g, gx, gy, gz);
    RefSolid S{0u, 0u};
    if (ref_tile_clear(gx, gy, gz, g)) return S;
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k) {
        const uint32_t x = gx * 8u + k, y = gy * 8u + k, z = gz * 8u + k;
        if (x < 2u || y < 2u || x > (uint64_t)(g.sizeX * 8u) + 2u || y > (uint64_t)(g.sizeY * 8u) + 2u) S.row |= 1u << k;
        if (z < 2u || z > (uint64_t)(g.sizeZ * 8u) + 2u) S.planes |= 1u << k;
    }
    return S;
}

// getNumberVoxelsUsedPerNode (particles.cu:88-190): mask + count per node,
// kNodeLanes lanes a node: 32 or 8 take a node's particles in turn, 1 leaves a
// node to a lane (sparse nodes, whose long ones the whole warp takes first).
// Every lane gathers in words of its own.  A node of more than `giant`
// particles (positions clamped to a domain face pile up in its nodes) gets
// its solid voxels here and the others from ref_voxel_giants_kernel: left to
// one warp, such nodes were 25 of 38 ms at 64M particles.
constexpr int kVoxWarps = 8;
// Particles above which the warp takes a sparse variant's node together: at 4, 8,
// 16 and never, 24 million nodes of 2.5 took 3.27, 2.35, 2.37 and 2.38 ms, and with a
// tenth of the positions clamped to the faces 2.51, 2.46, 2.47 and 8.63 ms.
constexpr uint32_t kVoxLong = 8;
// ... and above which several warps do: at 256, 1,024 and 4,096, 59 million
// particles took 2.47, 2.35 and 2.31 ms, clamped ones 2.56, 2.46 and 3.82 ms.
constexpr uint32_t kVoxGiant = 1024;
struct VoxWarp {
    unsigned long long planes[8 * kVoxStride];
    uint32_t mask[32 * 17];  // rows of 16 words, padded: the masks of the warp's nodes
};
template <int kNodeLanes>
__global__ void __launch_bounds__(32 * kVoxWarps) ref_voxel_counts_kernel(
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes, uint64_t n,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz, flip_grid g, uint32_t giant,
    uint32_t* __restrict__ counts, uint32_t* __restrict__ masks) {
    extern __shared__ __align__(16) unsigned char vox_smem[];
    VoxWarp& W = reinterpret_cast<VoxWarp*>(vox_smem)[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    constexpr uint32_t kNodes = 32u / kNodeLanes;  // nodes a warp
    const uint32_t b0 = (blockIdx.x * kVoxWarps + (threadIdx.x >> 5)) * kNodes;
    if (b0 >= nodes) return;  // a whole warp; nothing below synchronises the CTA
    unsigned long long* mine = W.planes + lane;
    auto clear = [&]() {
#pragma unroll
        for (int z = 0; z < 8; ++z) mine[z * kVoxStride] = 0ull;
    };
    // the node's mask from the 32 lanes' words, into row r
    auto gather = [&](uint32_t r) {
        uint32_t word = 0;
#pragma unroll
        for (int z = 0; z < 8; ++z) {
            const unsigned long long v = mine[z * kVoxStride];
            const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
            if (lane == 2u * z) word = lo;
            if (lane == 2u * z + 1u) word = hi;
        }
        if (lane < 16u) W.mask[17u * r + lane] = word;
    };
    const uint32_t r = lane / kNodeLanes, b = b0 + r;  // the lane's node
    uint32_t first = 0, last = 0;
    if (b < nodes) {
        first = starts[b];
        last = b == nodes - 1u ? (uint32_t)n : starts[b + 1u];
    }
    RefNode N = ref_node(b < nodes ? keys[first] : 0u, g);
    if (last - first > giant) last = first;
    if (kNodeLanes > 1) {
        clear();
        __syncwarp();
        ref_mark_particles(N, first + lane % kNodeLanes, last, kNodeLanes, px, py, pz, W.planes);
        if (kNodeLanes == 32) {
            gather(0);
        } else {
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                unsigned long long v = mine[z * kVoxStride];
#pragma unroll
                for (int o = 1; o < kNodeLanes; o <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
                if (lane % kNodeLanes == 0u) {
                    W.mask[17u * r + 2u * z] = (uint32_t)v;
                    W.mask[17u * r + 2u * z + 1u] = (uint32_t)(v >> 32);
                }
            }
        }
    } else {
        const bool is_long = last - first > kVoxLong;
        for (uint32_t rest = __ballot_sync(0xffffffffu, is_long); rest; rest &= rest - 1u) {
            const int j = __ffs(rest) - 1;
            const uint32_t f = __shfl_sync(0xffffffffu, first, j), l = __shfl_sync(0xffffffffu, last, j);
            clear();
            __syncwarp();
            ref_mark_particles(ref_node(keys[f], g), f + lane, l, 32u, px, py, pz, W.planes);
            gather((uint32_t)j);
        }
        clear();
        __syncwarp();
        ref_mark_particles(N, first, is_long ? first : last, 1u, px, py, pz, W.planes);
        if (!is_long) {
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                const unsigned long long v = mine[z * kVoxStride];
                W.mask[17u * lane + 2u * z] = (uint32_t)v;
                W.mask[17u * lane + 2u * z + 1u] = (uint32_t)(v >> 32);
            }
        }
    }
    __syncwarp();
    // solid voxels of tiles on the domain's faces, then the counts
    if (b < nodes && lane % kNodeLanes == 0u) {
        uint32_t c = 0;
        const RefSolid sol = ref_solid(keys[b], g);  // Q3: particle b's key, not the node's
        if (sol.row | sol.planes)
            for (uint32_t z = 0; z < 8u; ++z) {
                const unsigned long long v = sol.plane(z);
                W.mask[17u * r + 2u * z] |= (uint32_t)v;
                W.mask[17u * r + 2u * z + 1u] |= (uint32_t)(v >> 32);
            }
#pragma unroll
        for (int k = 0; k < 16; ++k) c += __popc(W.mask[17u * r + k]);
        counts[b] = c;
    }
    __syncwarp();
    const uint32_t words = 16u * min(kNodes, nodes - b0);
    for (uint32_t i = lane; i < words; i += 32u) masks[(size_t)b0 * 16u + i] = W.mask[17u * (i >> 4) + (i & 15u)];
}

// the last node whose first particle is at most p (starts ascend from 0): 32
// probes a step
__device__ __forceinline__ uint32_t ref_node_of(const uint32_t* __restrict__ starts, uint32_t nodes, uint32_t p) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = nodes;
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u, at = lo + lane * step;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, at < hi && (lane == 0u || starts[at] <= p)));
        lo += (c - 1u) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}
// The nodes of more than kVoxGiant particles: a warp takes kVoxGiant
// consecutive particles, so a giant node among them holds the first or the
// last one.  The bits that an atomic OR finds unset are the ones to count.
__global__ void __launch_bounds__(32 * kVoxWarps) ref_voxel_giants_kernel(
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes, uint64_t n,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz, flip_grid g,
    uint32_t* __restrict__ counts, uint32_t* __restrict__ masks) {
    __shared__ unsigned long long planes[kVoxWarps][8 * kVoxStride];
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t p0 = ((uint64_t)blockIdx.x * kVoxWarps + (threadIdx.x >> 5)) * kVoxGiant;
    if (p0 >= n) return;  // a whole warp
    const uint32_t p1 = (uint32_t)min(p0 + kVoxGiant, n);
    unsigned long long* mine = planes[threadIdx.x >> 5] + lane;
    uint32_t b = ref_node_of(starts, nodes, (uint32_t)p0);
    for (int end = 0; end < 2; ++end) {
        if (end) {
            const uint32_t e = ref_node_of(starts, nodes, p1 - 1u);
            if (e == b) return;
            b = e;
        }
        const uint32_t first = starts[b], last = b == nodes - 1u ? (uint32_t)n : starts[b + 1u];
        if (last - first <= kVoxGiant) continue;
#pragma unroll
        for (int z = 0; z < 8; ++z) mine[z * kVoxStride] = 0ull;
        const RefNode N = ref_node(keys[first], g);
        const uint32_t i1 = min(last, p1);
        __syncwarp();
        ref_mark_particles(N, max(first, (uint32_t)p0) + lane, i1, 32u, px, py, pz, planes[threadIdx.x >> 5]);
        uint32_t word = 0;
#pragma unroll
        for (int z = 0; z < 8; ++z) {
            const unsigned long long v = mine[z * kVoxStride];
            const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(v >> 32));
            if (lane == 2u * z) word = lo;
            if (lane == 2u * z + 1u) word = hi;
        }
        uint32_t fresh = 0;
        if (lane < 16u && word) fresh = __popc(word & ~atomicOr(&masks[(size_t)b * 16u + lane], word));
        fresh = __reduce_add_sync(0xffffffffu, fresh);
        if (lane == 0u && fresh) atomicAdd(&counts[b], fresh);
    }
}

// generateVoxelIDs (particles.cu:192-321): compaction from the masks.  A warp
// lists the voxels of kNodes nodes in shared memory, 32 / kNodes lanes a node,
// and copies the list out in order.  Bound by the lanes' walks over their words'
// bits: eight lanes a node have the shortest, a lane a node takes the fewest
// instructions, which pays where nodes are many and sparse (the launch says
// from where); nodes too dense for its list then go in fours.  Few nodes (a warp
// each), and four with more voxels than the list holds, are written straight from
// their masks, lane l the voxel of bit l of each word.
constexpr uint32_t kIdList = 1280;
// nodes b0 .. b0 + count - 1, `total` voxels from `start` on
template <int kNodes>
__device__ __forceinline__ void ref_list_ids(uint32_t b0, uint32_t count, uint32_t start, uint32_t total,
                                             const uint32_t* __restrict__ keys, const uint32_t* __restrict__ masks,
                                             const uint32_t* __restrict__ node_voxels, const flip_grid& g, uint16_t* list,
                                             uint32_t* __restrict__ voxel_ids, int8_t* __restrict__ solids) {
    constexpr uint32_t kLanes = 32 / kNodes, kWords = kNodes == 32 ? 16 : 16 / kLanes;  // lanes a node, words a lane
    const uint32_t lane = threadIdx.x & 31u, b = b0 + lane / kLanes;
    const bool have = lane / kLanes < count;
    uint32_t m[kWords], at = 0;
    if (have) {
        const uint32_t* from = masks + (size_t)b * 16u + (lane % kLanes) * kWords;
        if (kWords % 4 == 0 && (reinterpret_cast<uintptr_t>(masks) & 15u) == 0u) {
#pragma unroll
            for (uint32_t k = 0; k + 4u <= kWords; k += 4u) {
                const uint4 q = *reinterpret_cast<const uint4*>(from + k);
                m[k] = q.x; m[k + 1] = q.y; m[k + 2] = q.z; m[k + 3] = q.w;
            }
        } else {  // (also a caller's pointer into a larger buffer)
#pragma unroll
            for (uint32_t k = 0; k < kWords; ++k) m[k] = from[k];
        }
        if (kNodes == 32 && lane) at = node_voxels[b - 1u] - start;
    }
    if (kNodes < 32) {
        uint32_t n = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWords; ++k) n += have ? __popc(m[k]) : 0u;
        at = warp_inclusive_scan(n) - n;
    }
    if (have) {
        const RefSolid sol = ref_solid(keys[b], g);
        uint16_t* to = list + at;
#pragma unroll
        for (uint32_t k = 0; k < kWords; ++k)
            for (uint32_t word = m[k]; word; word &= word - 1u) {
                const uint32_t id = 32u * (kWords * (lane % kLanes) + k) + (uint32_t)__ffs(word) - 1u;
                *to++ = (uint16_t)(id | (sol.at(id) << 15));  // bit 15: solid
            }
    }
    __syncwarp();
    for (uint32_t i = lane; i < total; i += 32u) {
        const uint32_t v = list[i];
        voxel_ids[start + i] = v & 511u;
        solids[start + i] = (int8_t)(v >> 15);
    }
    __syncwarp();  // the list is free
}
template <int kNodes>
__global__ void __launch_bounds__(32 * kVoxWarps) ref_voxel_ids_kernel(
    const uint32_t* __restrict__ keys, uint32_t nodes, const uint32_t* __restrict__ masks,
    const uint32_t* __restrict__ node_voxels, flip_grid g, uint32_t* __restrict__ voxel_ids, int8_t* __restrict__ solids) {
    __shared__ uint16_t lists[kVoxWarps][kNodes > 1 ? kIdList : 1];
    uint16_t* list = lists[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = (blockIdx.x * kVoxWarps + (threadIdx.x >> 5)) * kNodes;
    if (first >= nodes) return;
    const uint32_t last = min(first + kNodes, nodes);
    auto end_of = [&](uint32_t b) { return b ? node_voxels[b - 1u] : 0u; };  // of the nodes before b
    if constexpr (kNodes == 32) {
        const uint32_t start = end_of(first), total = end_of(last) - start;
        if (total <= kIdList) {
            ref_list_ids<kNodes>(first, last - first, start, total, keys, masks, node_voxels, g, list, voxel_ids, solids);
            return;
        }
    }
    for (uint32_t b0 = first; b0 < last; b0 += 4u) {
        const uint32_t count = min(4u, last - b0);
        if constexpr (kNodes > 1) {
            const uint32_t start = end_of(b0), total = end_of(b0 + count) - start;
            if (total <= kIdList) {
                ref_list_ids<4>(b0, count, start, total, keys, masks, node_voxels, g, list, voxel_ids, solids);
                continue;
            }
        }
        for (uint32_t b = b0; b < b0 + count; ++b) {
            const uint32_t m = lane < 16u ? masks[(size_t)b * 16u + lane] : 0u;
            uint32_t at = end_of(b);
            const RefSolid sol = ref_solid(keys[b], g);
            // the mask words that hold a voxel, in order
            for (uint32_t rest = __ballot_sync(0xffffffffu, m != 0u); rest; rest &= rest - 1u) {
                const int q = __ffs(rest) - 1;
                const uint32_t word = __shfl_sync(0xffffffffu, m, q);
                if ((word >> lane) & 1u) {
                    const uint32_t i = (uint32_t)q * 32u + lane, pos = at + __popc(word & ((1u << lane) - 1u));
                    voxel_ids[pos] = i;
                    solids[pos] = (int8_t)sol.at(i);
                }
                at += __popc(word);
            }
        }
    }
}

// ------------------------------------------------------------- P2G / G2P
__device__ __forceinline__ void ref_face_base(int dim, double hs, double& bx, double& by, double& bz) {
    if (dim == 0) { by += hs; bz += hs; }
    else if (dim == 1) { bx += hs; bz += hs; }
    else { by += hs; bx += hs; }
}
__device__ __forceinline__ double ref_weight(double d, double R) { return (d > R) ? 0.0 : 1.0 - d / R; }
// ref_weight of the distance whose square is s, with over2 = 1 / R^2:
// 1 - sqrt(t), t = s / R^2, 0 from t = 1 on.  The root is Newton's iteration
// from the FP32 reciprocal root y of t (relative error 2^-22): g = t y, one
// step g += g (1 - t y^2) / 2 (2^-43), and the remainder t - g^2 added back
// through y / 2 (below 2^-53), seven multiply-adds against sqrt()'s longer
// sequence.  A t below 1e-37 counts as such: the weight is 1 either way.
__device__ __forceinline__ double ref_tent(double s, double over2) {
    const double t = s * over2;
    if (t >= 1.0) return 0.0;
    const float yf = rsqrtf(fmaxf((float)t, 1e-37f));
    const double y = (double)yf, half = (double)(0.5f * yf);
    const double g = t * y, e = fma(-g, half, 0.5), g1 = fma(g, e, g);
    return 1.0 - fma(fma(-g1, g1, t), half, g1);
}

// one particle's weights and weighted velocities into the node's sums
__device__ __forceinline__ void ref_scatter(const RefLocal& L, const double (&v)[3], double scw, double hs, double R,
                                            double (*U)[512], double (*W)[512]) {
    for (int x = (int)(L.sx - 2u); (uint32_t)x < L.sx + 2u; ++x)
        for (int y = (int)(L.sy - 2u); (uint32_t)y < L.sy + 2u; ++y)
            for (int z = (int)(L.sz - 2u); (uint32_t)z < L.sz + 2u; ++z) {
                if (!((uint32_t)x < 8u && (uint32_t)y < 8u && (uint32_t)z < 8u)) continue;
                const int id = x + y * 8 + z * 64;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    double bx = x * scw, by = y * scw, bz = z * scw;
                    ref_face_base(d, hs, bx, by, bz);
                    double w = ref_weight(ref_dist(L.lx - bx, L.ly - by, L.lz - bz), R);
                    atomicAdd(&W[d][id], w);
                    atomicAdd(&U[d][id], __dmul_rn(w, v[d]));
                }
            }
}

// gatherParticleVelsToVoxels for X, Y and Z in one launch (particles.cu:379-488)
__global__ void __launch_bounds__(kNodeThreads) ref_p2g_kernel(
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes, uint64_t n,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const double* __restrict__ vx, const double* __restrict__ vy, const double* __restrict__ vz,
    const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids, const int8_t* __restrict__ solids,
    flip_grid g, double* __restrict__ ux, double* __restrict__ uy, double* __restrict__ uz) {
    __shared__ double U[3][512];
    __shared__ double W[3][512];
    __shared__ int8_t S[512];
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += kNodeThreads) {
        U[0][i] = U[1][i] = U[2][i] = 0.0;
        W[0][i] = W[1][i] = W[2][i] = 0.0;
        S[i] = 0;
    }
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) S[voxel_ids[k]] = solids[k];
    const uint32_t last = (b == nodes - 1) ? (uint32_t)n : starts[b + 1];
    const double scw = ref_scw(g), hs = scw / 2.0, R = 2.0 * scw;
    for (uint32_t idx = starts[b] + threadIdx.x; idx < last; idx += kNodeThreads) {
        RefLocal L = ref_particle_local(px, py, pz, keys, idx, g, scw);
        const double v[3] = {vx[idx], vy[idx], vz[idx]};
        ref_scatter(L, v, scw, hs, R, U, W);
    }
    __syncthreads();
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t id = voxel_ids[k];
        bool sol = S[id] != 0;
        ux[k] = (sol ? 0.0 : U[0][id]) / (W[0][id] + 0.0000001);
        uy[k] = (sol ? 0.0 : U[1][id]) / (W[1][id] + 0.0000001);
        uz[k] = (sol ? 0.0 : U[2][id]) / (W[2][id] + 0.0000001);
    }
}

// The same for dense nodes, without atomics: a thread owns one of the 4^3
// voxel cells a node's particles lie in and one velocity component.  The
// particles come into shared memory sorted by cell, 512 at a time, and the
// threads go through the stencil's offsets together, one offset a phase: in
// a phase no two threads of a component touch one voxel, so each adds its
// cell's sums with plain additions.  Offsets that no particle of the cell can
// reach are left out (k = -2 on the component's own axis is two voxels or
// more away, k = -2 on both others 2.1).  Particles outside those cells (on an
// upper face, or outside the box) go through the atomics of the other form.
// FP64 atomics in shared memory are compare-and-swap loops: 1,060 us for
// 524,264 particles in 1,665 nodes, 478 us this way (what bounds it now: the
// instructions around a weight, at 18 of 32 lanes, cells holding 8 +- 3).
constexpr int kP2gThreads = 192;  // three components x 64 cells
constexpr int kP2gRound = 512;
struct RefP2gSmem {
    double U[3][512], W[3][512];
    double l[3][kP2gRound], v[3][kP2gRound];  // sorted by cell
    uint32_t count[64], first[65];
    uint16_t odd[kP2gRound];
    uint32_t n_odd;
    int8_t S[512];
};
__global__ void __launch_bounds__(kP2gThreads, 4) ref_p2g_cells_kernel(
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes, uint64_t n,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const double* __restrict__ vx, const double* __restrict__ vy, const double* __restrict__ vz,
    const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids, const int8_t* __restrict__ solids,
    flip_grid g, double* __restrict__ ux, double* __restrict__ uy, double* __restrict__ uz) {
    extern __shared__ __align__(16) unsigned char p2g_smem[];
    RefP2gSmem& M = *reinterpret_cast<RefP2gSmem*>(p2g_smem);
    const uint32_t b = blockIdx.x, tid = threadIdx.x;
    for (int i = tid; i < 512; i += kP2gThreads) {
#pragma unroll
        for (int d = 0; d < 3; ++d) M.U[d][i] = M.W[d][i] = 0.0;
        M.S[i] = 0;
    }
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    const uint32_t begin = starts[b], end = (b == nodes - 1) ? (uint32_t)n : starts[b + 1];
    const RefNode N = ref_node(keys[begin], g);
    const double scw = N.scw, hs = scw / 2.0, R = N.R, over2 = 1.0 / (R * R);
    const int comp = (int)(tid >> 6), cell = (int)(tid & 63u), ca = cell & 3, cb = (cell >> 2) & 3, cc = cell >> 4;
    for (uint32_t r0 = begin; r0 < end; r0 += kP2gRound) {
        const uint32_t m = min((uint32_t)kP2gRound, end - r0);
        __syncthreads();
        if (tid < 64u) M.count[tid] = 0u;
        if (tid == 0) M.n_odd = 0u;
        __syncthreads();
        double l[3][3];
        uint32_t at[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t q = tid + kP2gThreads * (uint32_t)k;
            at[k] = 0xFFFFFFFFu;
            if (q < m) {
                l[k][0] = ref_node_local(N, 0, px[r0 + q]);
                l[k][1] = ref_node_local(N, 1, py[r0 + q]);
                l[k][2] = ref_node_local(N, 2, pz[r0 + q]);
                // (a velocity that is not finite spoils the whole stencil there, weight 0 or not)
                const double big = fmax(fabs(vx[r0 + q]), fmax(fabs(vy[r0 + q]), fabs(vz[r0 + q])));
                const bool finite = big < __longlong_as_double(0x7FF0000000000000ll) && !isnan(vx[r0 + q]) &&
                                    !isnan(vy[r0 + q]) && !isnan(vz[r0 + q]);
                const uint32_t x = sat_u32_d(floor(l[k][0] / scw)) - 2u, y = sat_u32_d(floor(l[k][1] / scw)) - 2u,
                               z = sat_u32_d(floor(l[k][2] / scw)) - 2u;
                if (finite && x < 4u && y < 4u && z < 4u) {
                    const uint32_t c = x + 4u * y + 16u * z;
                    at[k] = c | (atomicAdd(&M.count[c], 1u) << 6);
                } else {
                    M.odd[atomicAdd(&M.n_odd, 1u)] = (uint16_t)q;
                }
            }
        }
        __syncthreads();
        if (tid < 32u) {  // exclusive scan of 64 counts
            const uint32_t c0 = M.count[2u * tid], c1 = M.count[2u * tid + 1u];
            const uint32_t inc = warp_inclusive_scan(c0 + c1);
            M.first[2u * tid] = inc - c0 - c1;
            M.first[2u * tid + 1u] = inc - c1;
            if (tid == 31u) M.first[64] = inc;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (at[k] != 0xFFFFFFFFu) {
                const uint32_t j = M.first[at[k] & 63u] + (at[k] >> 6), q = r0 + tid + kP2gThreads * (uint32_t)k;
#pragma unroll
                for (int d = 0; d < 3; ++d) M.l[d][j] = l[k][d];
                M.v[0][j] = vx[q];
                M.v[1][j] = vy[q];
                M.v[2][j] = vz[q];
            }
        __syncthreads();
        const uint32_t j0 = M.first[cell], j1 = M.first[cell + 1];
        const double hx = comp == 0 ? 0.0 : hs, hy = comp == 1 ? 0.0 : hs, hz = comp == 2 ? 0.0 : hs;
        const double* V = M.v[comp];
        double *Uc = M.U[comp], *Wc = M.W[comp];
#pragma unroll 1
        for (int k = 0; k < 64; ++k) {
            const int kx = k >> 4, ky = (k >> 2) & 3, kz = k & 3;
            const int own = comp == 0 ? kx : (comp == 1 ? ky : kz), o1 = comp == 0 ? ky : kx, o2 = comp == 2 ? ky : kz;
            if (own == 0 || (o1 == 0 && o2 == 0)) continue;  // the same for the component's 64 threads
            // the reference's loops: x from s - 2, s = c + 2
            const int x = ca + kx, y = cb + ky, z = cc + kz;
            const double bx = x * scw + hx, by = y * scw + hy, bz = z * scw + hz;
            // four particles at a time: their chains of dependent FP64 operations overlap
            double aw = 0.0, au = 0.0;
            for (uint32_t j = j0; j < j1; j += 4u) {
                double w[4];
#pragma unroll
                for (uint32_t q = 0; q < 4u; ++q) {
                    const uint32_t i = min(j + q, j1 - 1u);
                    const double dx = M.l[0][i] - bx, dy = M.l[1][i] - by, dz = M.l[2][i] - bz;
                    w[q] = ref_tent(fma(dx, dx, fma(dy, dy, dz * dz)), over2);
                    if (j + q >= j1) w[q] = 0.0;
                }
                aw += (w[0] + w[1]) + (w[2] + w[3]);
#pragma unroll
                for (uint32_t q = 0; q < 4u; ++q) au = fma(w[q], V[min(j + q, j1 - 1u)], au);
            }
            const int id = x + 8 * y + 64 * z;
            Wc[id] += aw;
            Uc[id] += au;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + comp) : "memory");
        }
        __syncthreads();
        for (uint32_t i = tid; i < M.n_odd; i += kP2gThreads) {
            const uint32_t q = r0 + M.odd[i];
            RefLocal L = ref_particle_local(px, py, pz, keys, q, g, scw);
            const double v[3] = {vx[q], vy[q], vz[q]};
            ref_scatter(L, v, scw, hs, R, M.U, M.W);
        }
    }
    __syncthreads();
    for (uint32_t k = vs + tid; k < ve; k += kP2gThreads) M.S[voxel_ids[k]] = solids[k];
    __syncthreads();
    for (uint32_t k = vs + tid; k < ve; k += kP2gThreads) {
        const uint32_t id = voxel_ids[k];
        const bool sol = M.S[id] != 0;
        ux[k] = (sol ? 0.0 : M.U[0][id]) / (M.W[0][id] + 0.0000001);
        uy[k] = (sol ? 0.0 : M.U[1][id]) / (M.W[1][id] + 0.0000001);
        uz[k] = (sol ? 0.0 : M.U[2][id]) / (M.W[2][id] + 0.0000001);
    }
}

// gatherVoxelVelsToParticles for X, Y and Z (particles.cu:562-662).  FP64
// issue bound (a root and about 15 multiply-adds a weight); the stencil column
// k = -2 on a component's own axis weighs nothing and is left out.
__global__ void __launch_bounds__(kNodeThreads) ref_g2p_kernel(
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys, uint32_t nodes, uint64_t n,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids,
    const double* __restrict__ ux, const double* __restrict__ uy, const double* __restrict__ uz, flip_grid g,
    double* __restrict__ vx, double* __restrict__ vy, double* __restrict__ vz) {
    __shared__ double U[3][512];
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += kNodeThreads) U[0][i] = U[1][i] = U[2][i] = 0.0;
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t id = voxel_ids[k];
        U[0][id] = ux[k];
        U[1][id] = uy[k];
        U[2][id] = uz[k];
    }
    __syncthreads();
    const uint32_t first = starts[b], last = (b == nodes - 1) ? (uint32_t)n : starts[b + 1];
    const RefNode N = ref_node(keys[first], g);
    const double scw = N.scw, hs = scw / 2.0, R = N.R, over2 = 1.0 / (R * R);
    for (uint32_t idx = first + threadIdx.x; idx < last; idx += kNodeThreads) {
        const double lx = ref_node_local(N, 0, px[idx]), ly = ref_node_local(N, 1, py[idx]), lz = ref_node_local(N, 2, pz[idx]);
        const uint32_t sx = sat_u32_d(floor(lx / scw)), sy = sat_u32_d(floor(ly / scw)), sz = sat_u32_d(floor(lz / scw));
        double vel[3] = {0.0, 0.0, 0.0}, ws[3] = {0.0, 0.0, 0.0};
        // the reference's loops end at the tile's upper edge and do not begin
        // below its lower one
        const bool any = sx - 2u < 8u && sy - 2u < 8u && sz - 2u < 8u;
#pragma unroll 1
        for (int kx = 0; any && kx < 4; ++kx) {
            const uint32_t x = sx - 2u + (uint32_t)kx;
            if (x >= 8u) break;
            const double dx = lx - (int)x * scw, ex = lx - ((int)x * scw + hs);
#pragma unroll 1
            for (int ky = 0; ky < 4; ++ky) {
                const uint32_t y = sy - 2u + (uint32_t)ky;
                if (y >= 8u) break;
                const double dy = ly - (int)y * scw, ey = ly - ((int)y * scw + hs);
#pragma unroll
                for (int kz = 0; kz < 4; ++kz) {
                    const uint32_t z = sz - 2u + (uint32_t)kz;
                    if (z >= 8u) break;
                    const double dz = lz - (int)z * scw, ez = lz - ((int)z * scw + hs);
                    const double ez2 = ez * ez;
                    const int id = (int)(x + 8u * y + 64u * z);
                    auto take = [&](int d, bool skip, double s) {
                        const double u = U[d][id];
                        const double w = skip ? 0.0 : ref_tent(s, over2);
                        if (u != 0.0) {  // Q10
                            ws[d] += w;
                            vel[d] = fma(w, u, vel[d]);
                        }
                    };
                    take(0, kx == 0, fma(dx, dx, fma(ey, ey, ez2)));
                    take(1, ky == 0, fma(ex, ex, fma(dy, dy, ez2)));
                    take(2, kz == 0, fma(ex, ex, fma(ey, ey, dz * dz)));
                }
            }
        }
        vx[idx] = vel[0] / (ws[0] + 0.00000001);
        vy[idx] = vel[1] / (ws[1] + 0.00000001);
        vz[idx] = vel[2] / (ws[2] + 0.00000001);
    }
}

// advectParticlePositions for the three axes (particles.cu:664-669)
__global__ void ref_advect_kernel(uint64_t n, double dt, double* __restrict__ px, double* __restrict__ py,
                                  double* __restrict__ pz, const double* __restrict__ vx, const double* __restrict__ vy,
                                  const double* __restrict__ vz) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    px[i] = fma(dt, vx[i], px[i]);
    py[i] = fma(dt, vy[i], py[i]);
    pz[i] = fma(dt, vz[i], pz[i]);
}

// --------------------------------------------------------------- pressure
// applyGravityKernel / removeGravityKernel (voxelSolveFunctions.cu:160-175)
__global__ void ref_gravity_kernel(uint64_t nvox, const int8_t* __restrict__ solids, double* __restrict__ uy, double dt,
                                   int remove) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nvox || solids[i]) return;
    const double c = (double)(-9.8f);
    uy[i] = remove ? fma(-c, dt, uy[i]) : fma(c, dt, uy[i]);
}

__device__ void ref_apron_add(uint32_t nid, const uint32_t* node_voxels, const uint32_t* voxel_ids, const double* data,
                              double* S, int xo, int yo, int zo) {
    const uint32_t vs = nid ? node_voxels[nid - 1] : 0u, ve = node_voxels[nid];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += blockDim.x) {
        uint32_t id = voxel_ids[k];
        uint32_t sx = id % 8u, sy = (id % 64u) / 8u, sz = id / 64u;
        uint32_t tx = sx, ty = sy, tz = sz;
        int t = -1;
        if (xo < 0) { if (sx >= 8u + (uint32_t)xo) { tx = sx - 8u - (uint32_t)xo; t = tx + ty * 8 + tz * 64; } }
        else if (xo > 0) { if (sx < (uint32_t)xo) { tx = 8u - (uint32_t)xo + sx; t = tx + ty * 8 + tz * 64; } }
        else if (yo < 0) { if (sy >= 8u + (uint32_t)yo) { ty = sy - 8u - (uint32_t)yo; t = tx + ty * 8 + tz * 64; } }
        else if (yo > 0) { if (sy < (uint32_t)yo) { ty = 8u - (uint32_t)yo + sy; t = tx + ty * 8 + tz * 64; } }
        else if (zo < 0) { if (sz >= 8u + (uint32_t)zo) { tz = sz - 8u - (uint32_t)zo; t = tz + ty * 8 + tz * 64; } }  // Q6
        else if (zo > 0) { if (sz < (uint32_t)zo) { tz = 8u - (uint32_t)zo + sz; t = tx + ty * 8 + tz * 64; } }
        if (t >= 0) atomicAdd(&S[t], data[k]);
    }
}

// cudaCalcDivU for X, Y and Z (voxelSolveFunctions.cu:97-271): apron
// contributions of the x/y/z neighbours, then forward differences
__global__ void __launch_bounds__(kNodeThreads) ref_divergence_kernel(
    uint32_t nodes, const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids,
    const double* __restrict__ ux, const double* __restrict__ uy, const double* __restrict__ uz, flip_grid g,
    const uint32_t* __restrict__ ytable, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys,
    double* __restrict__ divU) {
    __shared__ double S[3][512];
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += kNodeThreads) S[0][i] = S[1][i] = S[2][i] = 0.0;
    __syncthreads();
    const double* data[3] = {ux, uy, uz};
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t id = voxel_ids[k];
        S[0][id] = ux[k];
        S[1][id] = uy[k];
        S[2][id] = uz[k];
    }
    __syncthreads();
    const uint32_t cur = keys[starts[b]];
    const uint32_t cx = cur % g.sizeX, cy = (cur % (g.sizeX * g.sizeY)) / g.sizeX, cz = cur / (g.sizeX * g.sizeY);
    const int xl = (int)(cx - 1u), xr = (int)(cx + 1u), yl = (int)(cy - 1u), yr = (int)(cy + 1u), zl = (int)(cz - 1u),
              zr = (int)(cz + 1u);
    const int T = 4;
    // y-row table lookups; a key on the upper face of the box aliases past the
    // last row (the reference reads out of bounds there), treated as "none"
    const uint32_t rows = g.sizeY * g.sizeZ;
    auto row = [&](uint32_t r) -> uint32_t { return r < rows ? ytable[r] : nodes; };
    const uint32_t nyl = yl >= 0 ? row((uint32_t)yl + cz * g.sizeY) : nodes;
    const uint32_t nyr = (uint32_t)yr < g.sizeY ? row((uint32_t)yr + cz * g.sizeY) : nodes;
    const uint32_t nzl = zl >= 0 ? row((uint32_t)zl * g.sizeY + cy) : nodes;
    const uint32_t nzr = (uint32_t)zr < g.sizeZ ? row((uint32_t)zr * g.sizeY + cy) : nodes;
    const bool hxl = xl >= 0 && b > 0 && keys[starts[b - 1]] == cur - 1u;
    const bool hxr = (uint32_t)xr < g.sizeX && b < nodes - 1 && keys[starts[b + 1]] == cur + 1u;
    for (int d = 0; d < 3; ++d) {
        if (hxl) ref_apron_add(b - 1, node_voxels, voxel_ids, data[d], S[d], -T, 0, 0);
        __syncthreads();
        if (hxr) ref_apron_add(b + 1, node_voxels, voxel_ids, data[d], S[d], T, 0, 0);
        __syncthreads();
        if (nyl < nodes) ref_apron_add(nyl, node_voxels, voxel_ids, data[d], S[d], 0, -T, 0);
        __syncthreads();
        if (nyr < nodes) ref_apron_add(nyr, node_voxels, voxel_ids, data[d], S[d], 0, T, 0);
        __syncthreads();
        if (nzl < nodes) ref_apron_add(nzl, node_voxels, voxel_ids, data[d], S[d], 0, 0, -T);
        __syncthreads();
        if (nzr < nodes) ref_apron_add(nzr, node_voxels, voxel_ids, data[d], S[d], 0, 0, T);
        __syncthreads();
    }
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t id = voxel_ids[k];
        double dx = (id % 8u < 7u) ? S[0][id + 1] - S[0][id] : 0.0;
        double dy = ((id % 64u) / 8u < 7u) ? S[1][id + 8] - S[1][id] : 0.0;
        double dz = (id / 64u < 7u) ? S[2][id + 64] - S[2][id] : 0.0;
        divU[k] = ((0.0 + dx) + dy) + dz;
    }
}

__device__ __forceinline__ bool ref_is_apron(uint32_t id) {
    uint32_t x = id % 8u, y = (id % 8u * 8u) / 8u, z = id / 64u;  // y as written: equals x
    return x < 1u || x >= 7u || y < 1u || y >= 7u || z < 1u || z >= 7u;
}
__device__ __forceinline__ bool ref_is_red(uint32_t id) {
    uint32_t x = id % 8u, y = (id % 64u) / 8u, z = id / 64u;
    return !((x + y + z) & 1u);
}

// `iters` red+black iterations of GSiteration (voxelSolveFunctions.cu:293-389)
// kept in shared memory: the reference's sweeps never read another node's
// voxels, so iterating in place is the same arithmetic as 2*iters launches.
__global__ void __launch_bounds__(kNodeThreads) ref_gs_kernel(
    uint32_t nodes, const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids,
    const int8_t* __restrict__ solids, const double* __restrict__ divU, double* __restrict__ p, double* __restrict__ res,
    double scale, double w, uint32_t iters) {
    __shared__ double D[512], P[512], Rr[512];
    __shared__ int8_t S[512];
    __shared__ uint16_t ids[512];
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += kNodeThreads) { D[i] = 0.0; P[i] = 0.0; Rr[i] = 0.0; S[i] = 0; }
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    const uint32_t cnt = ve - vs;
    for (uint32_t k = threadIdx.x; k < cnt; k += kNodeThreads) {
        uint32_t id = voxel_ids[vs + k];
        ids[k] = (uint16_t)id;
        D[id] = divU[vs + k];
        P[id] = p[vs + k];
        S[id] = solids[vs + k];
    }
    __syncthreads();
    for (uint32_t it = 0; it < iters; ++it) {
        for (int color = 1; color >= 0; --color) {
            for (uint32_t k = threadIdx.x; k < cnt; k += kNodeThreads) {
                uint32_t v = ids[k];
                Rr[v] = 0.0;  // the pass writes residual 0 for voxels it does not update
                if ((color == (int)ref_is_red(v)) && !S[v] && !ref_is_apron(v)) {
                    double Ad = 0.0, Anx = 0.0, Apx = 0.0, Any = 0.0, Apy = 0.0, Anz = 0.0, Apz = 0.0;
                    if (!S[v - 1]) { if (D[v - 1] != 0.0) Anx = -scale; Ad += scale; }
                    if (!S[v + 1]) { if (D[v + 1] != 0.0) Apx = -scale; Ad += scale; }
                    if (!S[v - 8]) { if (D[v - 8] != 0.0) Any = -scale; Ad += scale; }
                    if (!S[v + 8]) { if (D[v + 8] != 0.0) Apy = -scale; Ad += scale; }
                    if (!S[v - 64]) { if (D[v - 64] != 0.0) Anz = -scale; Ad += scale; }
                    if (!S[v + 64]) { if (D[v + 64] != 0.0) Apz = -scale; Ad += scale; }
                    double s = __dmul_rn(Anx, P[v - 1]);
                    s = fma(Apx, P[v + 1], s);
                    s = fma(Any, P[v - 8], s);
                    s = fma(Apy, P[v + 8], s);
                    s = fma(Anz, P[v - 64], s);
                    s = fma(Apz, P[v + 64], s);
                    double Adg = Ad + 0.000000001;
                    double t = __dsub_rn(__ddiv_rn(-D[v] - s, Adg), P[v]);
                    double pn = fma(w, t, P[v]);
                    P[v] = pn;
                    Rr[v] = __dadd_rn(fma(-Adg, pn, -D[v]), s);
                }
            }
            __syncthreads();
        }
    }
    for (uint32_t k = threadIdx.x; k < cnt; k += kNodeThreads) {
        uint32_t id = ids[k];
        p[vs + k] = P[id];
        res[vs + k] = Rr[id];
    }
}

// Many iterations of the same, for the chunks between two reads of the
// residual.  Bound by the latency of one dependent FP64 chain per color, so
// the chain is cut down: a thread keeps one red and one black voxel, the only
// ones that move (no apron, no solid), in registers with
//   p' = (1 - w) p + w (c - D / Adg), c = (scale / Adg) * sum of the coupled neighbours' p,
// the neighbours summed as a tree: 7 dependent operations instead of 12 and a
// division.  The residual that the reference reads is that of the last sweep,
// taken by its own formula.  160 nodes: 1.78 us per iteration by
// ref_gs_kernel, 0.35 us here.
// The apron test lets y = 0 and y = 7 move, where the index v -+ 8 names a
// voxel of the same color in the next plane, with y = 7 or 0.  No sweep reads
// one: a particle marks no voxel of the plane y = 0 (its stencil coordinate
// is at least 2, and the column two below it is never nearer than the radius),
// so a listed voxel there is a solid one, which neither moves nor is coupled,
// and one that is not listed has D = 0.  The order within a color is then free.
constexpr int kSorThreads = 160;  // 144 voxels of a color can move
__global__ void __launch_bounds__(kSorThreads) ref_gs_long_kernel(
    uint32_t nodes, const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids,
    const int8_t* __restrict__ solids, const double* __restrict__ divU, double* __restrict__ p, double* __restrict__ res,
    double scale, double w, uint32_t iters) {
    __shared__ double D[512], P[512], Rr[512];
    __shared__ int8_t S[512], in[512];
    const uint32_t b = blockIdx.x, tid = threadIdx.x;
    for (int i = tid; i < 512; i += kSorThreads) { D[i] = 0.0; P[i] = 0.0; Rr[i] = 0.0; S[i] = 0; in[i] = 0; }
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + tid; k < ve; k += kSorThreads) {
        const uint32_t id = voxel_ids[k];
        D[id] = divU[k];
        P[id] = p[k];
        S[id] = solids[k];
        in[id] = 1;
    }
    __syncthreads();
    // color 1 (red: even x + y + z) goes first
    const int step[6] = {-1, 1, -8, 8, -64, 64};
    int v[2];
    bool move[2], couple[2][6];
    double Adg[2], own[2], coef[2], base[2], pv[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int x3 = (int)tid % 3, y = ((int)tid / 3) & 7, z = 1 + (int)tid / 24;
        const int x = 1 + 2 * x3 + ((1 + y + z + c) & 1);  // c = 0: red, even parity
        v[c] = tid < 144u ? x + 8 * y + 64 * z : 73;
        move[c] = tid < 144u && in[v[c]] && !S[v[c]];
        double Ad = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int u = v[c] + step[k];
            couple[c][k] = !S[u] && D[u] != 0.0;
            if (!S[u]) Ad += scale;
        }
        Adg[c] = Ad + 0.000000001;
        coef[c] = w * (scale / Adg[c]);
        base[c] = w * (-D[v[c]] / Adg[c]);
        own[c] = 1.0 - w;
        pv[c] = P[v[c]];
    }
    for (uint32_t it = 0; it < iters; ++it) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (move[c]) {
                const int i = v[c];
                double n[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) n[k] = couple[c][k] ? P[i + step[k]] : 0.0;
                const double sum = ((n[0] + n[1]) + (n[2] + n[3])) + (n[4] + n[5]);
                const double pn = fma(coef[c], sum, fma(own[c], pv[c], base[c]));
                if (it + 1u == iters && c == 1) {  // the last sweep's residual (red's is written as 0)
                    double s = 0.0;
#pragma unroll
                    for (int k = 0; k < 6; ++k) s = fma(couple[c][k] ? -scale : 0.0, n[k], s);
                    Rr[i] = __dadd_rn(fma(-Adg[c], pn, -D[i]), s);
                }
                pv[c] = pn;
                P[i] = pn;
            }
            __syncthreads();
        }
    }
    for (uint32_t k = vs + tid; k < ve; k += kSorThreads) {
        const uint32_t id = voxel_ids[k];
        p[k] = P[id];
        res[k] = Rr[id];
    }
}

// pressureToAcceleration for X, Y and Z (voxelSolveFunctions.cu:415-479)
__global__ void __launch_bounds__(kNodeThreads) ref_velocity_update_kernel(
    uint32_t nodes, const uint32_t* __restrict__ node_voxels, const uint32_t* __restrict__ voxel_ids,
    const int8_t* __restrict__ solids, const double* __restrict__ p, double* __restrict__ ux, double* __restrict__ uy,
    double* __restrict__ uz, double scale) {
    __shared__ double P[512];
    __shared__ int8_t S[512];
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += kNodeThreads) { P[i] = 0.0; S[i] = 0; }
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t id = voxel_ids[k];
        P[id] = p[k];
        S[id] = solids[k];
    }
    __syncthreads();
    double* U[3] = {ux, uy, uz};
    const uint32_t stride[3] = {1u, 8u, 64u};
    for (uint32_t k = vs + threadIdx.x; k < ve; k += kNodeThreads) {
        uint32_t v = voxel_ids[k];
        if (S[v] || ref_is_apron(v)) continue;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            double dp = 0.0;
            if (!S[v - stride[d]]) dp = __dsub_rn(P[v], P[v - stride[d]]);
            U[d][k] = fma(-dp, scale, U[d][k]);
        }
    }
}

// getMaxFromArray (engine/cudaVec.cu:173-203) as the reference computes it:
// each 512-element block yields the pick of its elements 0 and 256.
__global__ void ref_getmax_kernel(uint64_t n, const double* __restrict__ a, double* __restrict__ out, int absolute) {
    uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t nb = n / 512 + 1;
    if (b >= nb) return;
    uint64_t i0 = b * 512, i1 = b * 512 + 256;
    double s0 = (i0 < n) ? a[i0] : 0.0, s1 = (i1 < n) ? a[i1] : 0.0;
    out[b] = absolute ? ((fabs(s0) > fabs(s1)) ? s0 : s1) : ((s0 > s1) ? s0 : s1);
}

// moveSolids (particles.cu:674-740): particles outside their tile or inside
// a solid voxel are re-seeded at a random point of the node's first solid
// voxel (the reference searches for a solid one, Q8), with the reference's
// launch shape (32 threads per node) so that each thread draws from the same
// curand subsequence.  The search is bounded by the node's own voxel list;
// the reference compares against the cumulative count and can read past it.
__global__ void __launch_bounds__(32) ref_move_solids_kernel(
    uint32_t nodes, uint64_t n, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ keys,
    double* __restrict__ px, double* __restrict__ py, double* __restrict__ pz, const uint32_t* __restrict__ node_voxels,
    const uint32_t* __restrict__ voxel_ids, const int8_t* __restrict__ solids, flip_grid g) {
    __shared__ int8_t S[512];
    __shared__ uint32_t proc[512];
    curandState rs;
    curand_init(1291293829ull, threadIdx.x + blockIdx.x * blockDim.x, 0ull, &rs);
    const uint32_t b = blockIdx.x;
    for (int i = threadIdx.x; i < 512; i += 32) { S[i] = 0; proc[i] = 512u; }
    __syncthreads();
    const uint32_t vs = b ? node_voxels[b - 1] : 0u, ve = node_voxels[b];
    for (uint32_t k = vs + threadIdx.x; k < ve; k += 32) { S[voxel_ids[k]] = solids[k]; proc[k - vs] = voxel_ids[k]; }
    __syncthreads();
    const uint32_t cnt = ve - vs;
    const uint32_t last = (b == nodes - 1) ? (uint32_t)n : starts[b + 1];
    const double scw = ref_scw(g);
    for (uint32_t idx = starts[b] + threadIdx.x; idx < last; idx += 32) {
        uint32_t qx, qy, qz;
        ref_decompose(keys[idx], g, qx, qy, qz);
        double lx = ref_local(px[idx], g.negX, qx, g.cellSize, scw);
        double ly = ref_local(py[idx], g.negY, qy, g.cellSize, scw);
        double lz = ref_local(pz[idx], g.negZ, qz, g.cellSize, scw);
        uint32_t sx = sat_u32_d(floor(lx / scw)), sy = sat_u32_d(floor(ly / scw)), sz = sat_u32_d(floor(lz / scw));
        if (sx >= 8u || sy >= 8u || sz >= 8u || S[sx + sy * 8u + sz * 64u]) {
            uint32_t i = 0;
            while (i < cnt && !S[proc[i]]) ++i;
            uint32_t nv = (i < 512u) ? proc[i] : 512u;
            int nx_ = (int)(nv % 8u), ny_ = (int)((nv % 64u) / 8u), nz_ = (int)(nv / 64u);
            double bx = fma((double)(nx_ - 2), scw, (double)fmaf((float)qx, g.cellSize, g.negX));
            double by = fma((double)(ny_ - 2), scw, (double)fmaf((float)qy, g.cellSize, g.negY));
            double bz = fma((double)(nz_ - 2), scw, (double)fmaf((float)qz, g.cellSize, g.negZ));
            px[idx] = fma((double)curand_uniform(&rs), scw, bx);
            py[idx] = fma((double)curand_uniform(&rs), scw, by);
            pz[idx] = fma((double)curand_uniform(&rs), scw, bz);
        }
    }
}

// reorderGridIndices<double> (radixSortKernels.cu:59-68): out[i] = in[perm[i]]
__global__ void ref_gather_f64_kernel(const uint32_t* __restrict__ perm, uint64_t n, const double* __restrict__ in,
                                      double* __restrict__ out) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        uint32_t s = perm[i];
        out[i] = __ldg(in + (s < n ? s : i));  // a valid permutation always has s < n
    }
}

// ------------------------------------------------------------ launchers
static inline unsigned nblk(uint64_t n, int t) { return (unsigned)((n + t - 1) / t); }

int ref_launch_keys(double* px, double* py, double* pz, uint64_t n, const flip_grid& g, uint32_t* keys, uint32_t* idx,
                    cudaStream_t s) {
    if (n) ref_keys_kernel<<<nblk(n, 256), 256, 0, s>>>(px, py, pz, n, g, keys, idx);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_ydim(const uint32_t* starts, const uint32_t* keys, uint32_t nodes, const flip_grid& g, uint32_t* table,
                    cudaStream_t s) {
    uint32_t rows = g.sizeY * g.sizeZ;
    if (rows) ref_ydim_fill_kernel<<<nblk(rows, 256), 256, 0, s>>>(table, rows, nodes);
    if (nodes) ref_ydim_rows_kernel<<<nblk(nodes, 256), 256, 0, s>>>(starts, keys, nodes, g, table);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
// Lanes a node, in us for 1, 8 and 32.  Below 8 particles a node a lane is
// enough once there are warps for every SM (4 particles: 32,000 nodes 22, 22 and
// 38, 63,000 25, 30 and 65, 257,000 50, 82 and 229; at 8, 262,000 124, 106 and
// 244).  Eight lanes wait less for the fullest node than a warp idles over the
// others', up to some 128 particles a node and where nodes fill the chip (16,000
// nodes of 8, 64, 128, 315 particles: 19 and 25, 35 and 37, 54 and 50, 126 and 99;
// 64,000: 35 and 66, 97 and 123, 160 and 181, 347 and 348); a warp a node keeps
// fewer, denser ones (4,096 nodes of 64, 315: 21 and 20, 50 and 35).
constexpr uint32_t kSparseNodes = 65536, kWideNodes = 16384;
constexpr uint64_t kSparsePer = 8, kWidePer = 128;
// The pass over the giants takes 3 to 5 us (32,768 particles: 19.7 with it, 15.8
// without); a warp by itself takes 25 us for each 1,024 particles of a node.
constexpr uint64_t kVoxGiantFrom = 32768;
int ref_launch_voxel_counts(const uint32_t* starts, const uint32_t* keys, uint32_t nodes, uint64_t n, const double* px,
                            const double* py, const double* pz, const flip_grid& g, uint32_t* counts, uint32_t* masks,
                            cudaStream_t s) {
    if (!nodes) return FLIP_OK;
    const size_t smem = sizeof(VoxWarp) * kVoxWarps;
    static_assert(sizeof(VoxWarp) * kVoxWarps <= 49152, "within the default shared memory");
    const bool giants = n > kVoxGiantFrom;
    const uint32_t giant = giants ? kVoxGiant : 0xFFFFFFFFu;
    const int lanes = n < kSparsePer * nodes ? (nodes >= kSparseNodes ? 1 : 8)
                                             : (nodes >= kWideNodes && n < kWidePer * nodes ? 8 : 32);
    const uint32_t per = 32u / (uint32_t)lanes * kVoxWarps, grid = (nodes + per - 1) / per;
    const auto kernel = lanes == 1 ? ref_voxel_counts_kernel<1> : (lanes == 8 ? ref_voxel_counts_kernel<8> : ref_voxel_counts_kernel<32>);
    kernel<<<grid, 32 * kVoxWarps, smem, s>>>(starts, keys, nodes, n, px, py, pz, g, giant, counts, masks);
    if (giants) {
        const uint64_t chunk = (uint64_t)kVoxGiant * kVoxWarps;
        ref_voxel_giants_kernel<<<(unsigned)((n + chunk - 1) / chunk), 32 * kVoxWarps, 0, s>>>(starts, keys, nodes, n, px, py,
                                                                                           pz, g, counts, masks);
    }
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
// Ids: a warp a node below 16,384 nodes, four nodes a warp (512 nodes 11.4 and 15.5
// us, 15,600 of 200 voxels 17.3 and 16.9, 32,000 of 75 20.9 and 16.6, 79,000 31 and 21,
// 258,000 109 and 57), and 32 from 524,288 on: with four and 32 a warp, nodes of some 27
// voxels, 165,000 31 and 50 us, 524,000 74 and 71, 2.6 million 359 and 256; of 60 and more
// (32 go in fours then) 258,000 57 and 72, 982,000 187 and 210, 4 million 715 and 773,
// where a warp a node takes 1,534.
constexpr uint32_t kFewNodes = 16384, kManyNodes = 1u << 19;
int ref_launch_voxel_ids(const uint32_t* keys, uint32_t nodes, const uint32_t* masks, const uint32_t* node_voxels,
                         const flip_grid& g, uint32_t* voxel_ids, int8_t* solids, cudaStream_t s) {
    if (!nodes) return FLIP_OK;
    const uint32_t each = nodes < kFewNodes ? 1u : (nodes < kManyNodes ? 4u : 32u);
    const uint32_t per = each * kVoxWarps, grid = (nodes + per - 1) / per;
    const auto kernel = each == 1u ? ref_voxel_ids_kernel<1> : (each == 4u ? ref_voxel_ids_kernel<4> : ref_voxel_ids_kernel<32>);
    kernel<<<grid, 32 * kVoxWarps, 0, s>>>(keys, nodes, masks, node_voxels, g, voxel_ids, solids);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
// Cells from this many particles a node on average: the two forms cross at 16
// to 24 (scatter and cells, 4,096 nodes of 8, 16, 32, 64 particles: 328 and 352, 390
// and 363, 463 and 379, 529 and 437 us; 27,000 of 8, 16, 24, 32: 1,829 and 2,179, 2,233
// and 2,259, 2,499 and 2,302, 2,687 and 2,337), with a few hundred nodes earlier.
constexpr uint64_t kP2gDense = 32;
int ref_launch_p2g(const uint32_t* starts, const uint32_t* keys, uint32_t nodes, uint64_t n, const double* px,
                   const double* py, const double* pz, const double* vx, const double* vy, const double* vz,
                   const uint32_t* node_voxels, const uint32_t* voxel_ids, const int8_t* solids, const flip_grid& g,
                   double* ux, double* uy, double* uz, cudaStream_t s) {
    if (!nodes) return FLIP_OK;
    if (n >= kP2gDense * nodes) {
        FLIP_CUDA_TRY(cudaFuncSetAttribute(ref_p2g_cells_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(RefP2gSmem)));
        ref_p2g_cells_kernel<<<nodes, kP2gThreads, sizeof(RefP2gSmem), s>>>(starts, keys, nodes, n, px, py, pz, vx, vy, vz,
                                                                           node_voxels, voxel_ids, solids, g, ux, uy, uz);
    } else {
        ref_p2g_kernel<<<nodes, kNodeThreads, 0, s>>>(starts, keys, nodes, n, px, py, pz, vx, vy, vz, node_voxels, voxel_ids,
                                                      solids, g, ux, uy, uz);
    }
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_g2p(const uint32_t* starts, const uint32_t* keys, uint32_t nodes, uint64_t n, const double* px,
                   const double* py, const double* pz, const uint32_t* node_voxels, const uint32_t* voxel_ids,
                   const double* ux, const double* uy, const double* uz, const flip_grid& g, double* vx, double* vy,
                   double* vz, cudaStream_t s) {
    if (nodes)
        ref_g2p_kernel<<<nodes, kNodeThreads, 0, s>>>(starts, keys, nodes, n, px, py, pz, node_voxels, voxel_ids, ux, uy, uz,
                                                      g, vx, vy, vz);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_advect(uint64_t n, double dt, double* px, double* py, double* pz, const double* vx, const double* vy,
                      const double* vz, cudaStream_t s) {
    if (n) ref_advect_kernel<<<nblk(n, 256), 256, 0, s>>>(n, dt, px, py, pz, vx, vy, vz);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_gravity(uint64_t nvox, const int8_t* solids, double* uy, double dt, int remove, cudaStream_t s) {
    if (nvox) ref_gravity_kernel<<<nblk(nvox, 512), 512, 0, s>>>(nvox, solids, uy, dt, remove);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_divergence(uint32_t nodes, const uint32_t* node_voxels, const uint32_t* voxel_ids, const double* ux,
                          const double* uy, const double* uz, const flip_grid& g, const uint32_t* ytable,
                          const uint32_t* starts, const uint32_t* keys, double* divU, cudaStream_t s) {
    if (nodes)
        ref_divergence_kernel<<<nodes, kNodeThreads, 0, s>>>(nodes, node_voxels, voxel_ids, ux, uy, uz, g, ytable, starts,
                                                             keys, divU);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
// The solve asks for 1 and 1,023 iterations in turn (fewer at its cap) and
// reads the residual after the single ones, which stay with the list form and
// its order of operations.  What the long chunks leave in p differs from the
// list form's by rounding.
constexpr uint32_t kSorLong = 512;
int ref_launch_gs(uint32_t nodes, const uint32_t* node_voxels, const uint32_t* voxel_ids, const int8_t* solids,
                  const double* divU, double* p, double* res, double scale, double w, uint32_t iters, cudaStream_t s) {
    if (nodes && iters >= kSorLong)
        ref_gs_long_kernel<<<nodes, kSorThreads, 0, s>>>(nodes, node_voxels, voxel_ids, solids, divU, p, res, scale, w, iters);
    else if (nodes && iters)
        ref_gs_kernel<<<nodes, kNodeThreads, 0, s>>>(nodes, node_voxels, voxel_ids, solids, divU, p, res, scale, w, iters);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_velocity_update(uint32_t nodes, const uint32_t* node_voxels, const uint32_t* voxel_ids,
                               const int8_t* solids, const double* p, double* ux, double* uy, double* uz, double scale,
                               cudaStream_t s) {
    if (nodes)
        ref_velocity_update_kernel<<<nodes, kNodeThreads, 0, s>>>(nodes, node_voxels, voxel_ids, solids, p, ux, uy, uz, scale);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
int ref_launch_getmax_level(uint64_t n, const double* a, double* out, int absolute, cudaStream_t s) {
    uint64_t nb = n / 512 + 1;
    ref_getmax_kernel<<<nblk(nb, 256), 256, 0, s>>>(n, a, out, absolute);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int ref_launch_move_solids(uint32_t nodes, uint64_t n, const uint32_t* starts, const uint32_t* keys, double* px,
                           double* py, double* pz, const uint32_t* node_voxels, const uint32_t* voxel_ids,
                           const int8_t* solids, const flip_grid& g, cudaStream_t s) {
    if (nodes) ref_move_solids_kernel<<<nodes, 32, 0, s>>>(nodes, n, starts, keys, px, py, pz, node_voxels, voxel_ids, solids, g);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int ref_gather_f64(const uint32_t* perm, uint64_t n, const double* in, double* out, cudaStream_t s) {
    if (n) ref_gather_f64_kernel<<<nblk(n, 256), 256, 0, s>>>(perm, n, in, out);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

}  // namespace flip

using namespace flip;

extern "C" int flip_ref_keys(double* px, double* py, double* pz, uint64_t n, const flip_grid* grid, uint32_t* keys,
                             uint32_t* idx, void* stream) {
    if (!grid || (n && (!px || !py || !pz || !keys))) return FLIP_ERR_ARG;
    return ref_launch_keys(px, py, pz, n, *grid, keys, idx, as_stream(stream));
}
extern "C" int flip_ref_ydim_rows(const uint32_t* starts, const uint32_t* sorted_keys, uint32_t nodes,
                                  const flip_grid* grid, uint32_t* table, void* stream) {
    if (!grid || !table) return FLIP_ERR_ARG;
    return ref_launch_ydim(starts, sorted_keys, nodes, *grid, table, as_stream(stream));
}
extern "C" int flip_ref_voxel_counts(const uint32_t* starts, const uint32_t* sorted_keys, uint32_t nodes, uint64_t n,
                                     const double* px, const double* py, const double* pz, const flip_grid* grid,
                                     uint32_t* counts, uint32_t* masks, void* stream) {
    if (!grid || (nodes && (!starts || !sorted_keys || !counts || !masks))) return FLIP_ERR_ARG;
    return ref_launch_voxel_counts(starts, sorted_keys, nodes, n, px, py, pz, *grid, counts, masks, as_stream(stream));
}
extern "C" int flip_ref_voxel_ids(const uint32_t* sorted_keys, uint32_t nodes, const uint32_t* masks,
                                  const uint32_t* node_voxels, const flip_grid* grid, uint32_t* voxel_ids, int8_t* solids,
                                  void* stream) {
    if (!grid) return FLIP_ERR_ARG;
    return ref_launch_voxel_ids(sorted_keys, nodes, masks, node_voxels, *grid, voxel_ids, solids, as_stream(stream));
}
extern "C" int flip_ref_p2g(const uint32_t* starts, const uint32_t* sorted_keys, uint32_t nodes, uint64_t n,
                            const double* px, const double* py, const double* pz, const double* vx, const double* vy,
                            const double* vz, const uint32_t* node_voxels, const uint32_t* voxel_ids,
                            const int8_t* solids, const flip_grid* grid, double* ux, double* uy, double* uz,
                            void* stream) {
    if (!grid) return FLIP_ERR_ARG;
    return ref_launch_p2g(starts, sorted_keys, nodes, n, px, py, pz, vx, vy, vz, node_voxels, voxel_ids, solids, *grid, ux,
                          uy, uz, as_stream(stream));
}
extern "C" int flip_ref_g2p(const uint32_t* starts, const uint32_t* sorted_keys, uint32_t nodes, uint64_t n,
                            const double* px, const double* py, const double* pz, const uint32_t* node_voxels,
                            const uint32_t* voxel_ids, const double* ux, const double* uy, const double* uz,
                            const flip_grid* grid, double* vx, double* vy, double* vz, void* stream) {
    if (!grid) return FLIP_ERR_ARG;
    return ref_launch_g2p(starts, sorted_keys, nodes, n, px, py, pz, node_voxels, voxel_ids, ux, uy, uz, *grid, vx, vy, vz,
                          as_stream(stream));
}

extern "C" size_t flip_ref_getmax_scratch_bytes(uint64_t n) { return 2 * sizeof(double) * (n / 512 + 2); }

extern "C" int flip_ref_getmax_f64(const double* data, uint64_t n, int absolute, void* scratch, size_t scratch_bytes,
                                   double* result, void* stream) {
    if (!data || !result || !scratch || scratch_bytes < flip_ref_getmax_scratch_bytes(n)) return FLIP_ERR_ARG;
    cudaStream_t s = as_stream(stream);
    double* b0 = (double*)scratch;
    double* b1 = b0 + (n / 512 + 2);
    int rc = ref_launch_getmax_level(n, data, b0, absolute, s);
    if (rc) return rc;
    for (uint64_t i = n / 512 + 1; i > 1; i = i / 512 + 1) {
        rc = ref_launch_getmax_level(i, b0, b1, absolute, s);
        if (rc) return rc;
        double* t = b0; b0 = b1; b1 = t;
    }
    FLIP_CUDA_TRY(cudaMemcpyAsync(result, b0, sizeof(double), cudaMemcpyDeviceToHost, s));
    FLIP_CUDA_TRY(cudaStreamSynchronize(s));
    return FLIP_OK;
}
