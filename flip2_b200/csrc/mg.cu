// mg.cu -- V-cycle kernels of the multilevel learned preconditioner (mg.cuh).
//
// Every level is tile-blocked like the solver's grid (slot = tile * 512 +
// (i & 7) + 8 (j & 7) + 64 (k & 7)).  Per level the hierarchy kernels
// (coarse types, cell codes) walk every slot; the two smoothing kernels walk
// the level's tile list and stage each tile with a 2-cell halo in shared
// memory (see "smoothing" below); the coarsest level also has a one-CTA
// Jacobi-PCG (training targets, and the comparison without the network).
// Non-fluid cells carry 0 in every vector, so the 7-point operator needs only
// the fluid bit and the non-solid neighbour count of the PCG cell code.
#include "common.cuh"
#include "mg.cuh"

namespace flip {

__device__ __forceinline__ uint32_t mg_slot(int i, int j, int k, const NatDims& D) {
    uint32_t t = (uint32_t)((i >> 3) + D.tx * ((j >> 3) + D.ty * (k >> 3)));
    return (t << 9) | (uint32_t)((i & 7) | ((j & 7) << 3) | ((k & 7) << 6));
}
__device__ __forceinline__ void mg_cell_of(uint32_t key, int tid, const NatDims& D, int& i, int& j, int& k) {
    i = 8 * (int)(key % D.tx) + (tid & 7);
    j = 8 * (int)((key / D.tx) % D.ty) + ((tid >> 3) & 7);
    k = 8 * (int)(key / (D.tx * D.ty)) + (tid >> 6);
}
__device__ __forceinline__ bool mg_in(int i, int j, int k, const NatDims& D) {
    return i >= 0 && j >= 0 && k >= 0 && i < D.nx && j < D.ny && k < D.nz;
}
__device__ __forceinline__ float mg_dinv(uint8_t c) {
    const uint32_t d = c & 7u;
    return d ? 1.0f / (float)d : 0.0f;
}
// sum over the fluid neighbours of (i, j, k) of val(slot)
template <class F>
__device__ __forceinline__ float mg_nb_sum(int i, int j, int k, const NatDims& D, const uint8_t* __restrict__ cell, F val) {
    const int oi[6] = {-1, 1, 0, 0, 0, 0}, oj[6] = {0, 0, -1, 1, 0, 0}, ok[6] = {0, 0, 0, 0, -1, 1};
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int a = i + oi[q], b = j + oj[q], c = k + ok[q];
        if (!mg_in(a, b, c, D)) continue;
        const uint32_t u = mg_slot(a, b, c, D);
        if (cell[u] & kCellFluid) s += val(u);
    }
    return s;
}
__device__ __forceinline__ bool mg_halted(const int* halt) { return halt && *halt; }

// ------------------------------------------------------------ hierarchy
// coarse type from the 8 children: air if any child is air, else fluid if any
// is fluid, else solid; cells past the level's extent are solid
__global__ void __launch_bounds__(512) mg_coarsen_kernel(MgLevel F, MgLevel C, const int* halt) {
    if (mg_halted(halt)) return;
    const uint32_t n = C.ntiles * 512u;
    for (uint32_t s = blockIdx.x * 512u + threadIdx.x; s < n; s += gridDim.x * 512u) {
        int I, J, K;
        mg_cell_of(s >> 9, (int)(s & 511u), C.D, I, J, K);
        uint8_t t = kSolid;
        if (I < C.ex && J < C.ey && K < C.ez) {
            bool air = false, fluid = false;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int i = 2 * I + (c & 1), j = 2 * J + ((c >> 1) & 1), k = 2 * K + (c >> 2);
                if (i >= F.ex || j >= F.ey || k >= F.ez) continue;  // solid
                const uint8_t ft = F.type[mg_slot(i, j, k, F.D)];
                air |= ft == kAir;
                fluid |= ft == kFluid;
            }
            t = air ? kAir : (fluid ? kFluid : kSolid);
        }
        C.type[s] = t;
    }
}
// PCG cell codes of a coarse level: fluid bit and the non-solid neighbour count
__global__ void __launch_bounds__(512) mg_codes_kernel(MgLevel C, const int* halt) {
    if (mg_halted(halt)) return;
    const uint32_t n = C.ntiles * 512u;
    const int oi[6] = {-1, 1, 0, 0, 0, 0}, oj[6] = {0, 0, -1, 1, 0, 0}, ok[6] = {0, 0, 0, 0, -1, 1};
    for (uint32_t s = blockIdx.x * 512u + threadIdx.x; s < n; s += gridDim.x * 512u) {
        uint8_t code = 0;
        if (C.type[s] == kFluid) {
            int i, j, k;
            mg_cell_of(s >> 9, (int)(s & 511u), C.D, i, j, k);
            uint32_t d = 0;
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const int a = i + oi[q], b = j + oj[q], c = k + ok[q];
                if (mg_in(a, b, c, C.D) && C.type[mg_slot(a, b, c, C.D)] != kSolid) ++d;
            }
            code = (uint8_t)(kCellFluid | d);
        }
        C.cell[s] = code;
    }
}

// ------------------------------------------------------------ smoothing
// The V-cycle's smoothing runs as two kernels per level.  Each CTA stages a
// box of its tile and a 2-cell halo in shared memory: 16 cells wide in x
// (x = -4 .. 11, so that every row is four 16-byte quads of the tile
// layout: x 4..7 of the left tile, the tile's two quads, x 0..3 of the right
// tile) and 12 in y and z (-2 .. 9).  The first sweep is evaluated where the
// second one (or the residual) reads it: the tile's 64 rows and the 32 rows
// of its y and z faces, two quads each (a thread a quad), and the cells
// x = -1 and x = 8 of the tile's rows.  The staged quads are those that this
// takes: 456 of the box's 576.
// Vectors are zero off the fluid cells, so a neighbour sum needs no tests.
// The sweeps work on v = D^-1 r, so that a cell costs its neighbours' sum and
// two or three multiply-adds; four fluid cells with six non-solid neighbours
// (nearly all) take 1/6 as a constant, the others 1/d from a shared table.
// Rows lie 24 floats apart: the 16-byte accesses of a quarter warp, two quads
// in each of four consecutive rows, then fall on distinct banks (16 apart, two
// of the rows share theirs, and the shared memory's bandwidth bounds the
// sweeps).
// These kernels are bound by instructions and shared memory, not by HBM (6% of
// its rate): staging all 576 quads with a code test per cell and sweeping all
// 400 quads of the 10 x 10 rows took 22 and 25 us (down, up) on 2,752 tiles,
// this 17 and 22 us.  Registers for a fifth CTA per SM cost more (10.9 against
// 10.5 ms for a step on 16,000 tiles), and so did holding the next tile's loads
// in registers while one is worked on (10.8 ms).
constexpr int kMgThreads = 256;
constexpr int kMgCtas = 4;                      // per SM (64 registers a thread)
constexpr int kBX = 24, kBY = 12, kBZ = 12;      // rows of 16 cells, padded: see above
constexpr int kBoxF = kBX * kBY * kBZ;
constexpr int kT1F = kBX * 10 * 10;             // the first sweep's box
constexpr int kStaged = 456;                    // quads staged
constexpr int kQPer = (kStaged + kMgThreads - 1) / kMgThreads;  // 2
constexpr uint32_t kAllSix = 0x86868686u;       // four fluid cells, diagonal 6

// Two FP64 sums over the grid of a level kernel: per-CTA sums into
// partials[q * gridDim.x + CTA], then the last CTA to arrive adds the
// partials in CTA order (deterministic for a given grid), resets the ticket
// and returns true with the totals in thread 0's out.
__device__ __forceinline__ bool mg_last_cta_sum2(double v0, double v1, double* partials, unsigned int* ticket,
                                                 double (&out)[2]) {
    __shared__ double sh[32];
    __shared__ bool s_last;
    const double v[2] = {v0, v1};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const double s = block_sum_f64<kMgThreads>(v[q], sh);
        if (threadIdx.x == 0) partials[q * gridDim.x + blockIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        double a = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += kMgThreads) a += ((volatile double*)partials)[q * gridDim.x + b];
        out[q] = block_sum_f64<kMgThreads>(a, sh);
    }
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

__device__ __forceinline__ void mg_inv_table(float* inv) {
    if (threadIdx.x < 8) inv[threadIdx.x] = threadIdx.x ? 1.0f / (float)threadIdx.x : 0.0f;
}
// row n of the 96 rows of the tile and its y and z faces: (y, z), one of them
// in 0 .. 7
__device__ __forceinline__ void mg_face_row(int n, int& y, int& z) {
    if (n < 64) { y = n & 7; z = n >> 3; }
    else if (n < 80) { y = n < 72 ? -1 : 8; z = n & 7; }
    else { y = n & 7; z = n < 88 ? -1 : 8; }
}
// A staged quad, as constants of the thread: where it lies in the box and,
// relative to the tile's first slot, in the grid.
struct MgQuad {
    int box;       // float index in the box, -1: none
    int local;     // slot within its tile
    int dx, dy, dz;  // the tile it lies in, relative to the CTA's
    int delta;     // slots from the tile's first slot to the quad's
};
__device__ __forceinline__ MgQuad mg_quad(int n, const NatDims& D) {
    MgQuad Q;
    Q.box = -1;
    Q.local = Q.dx = Q.dy = Q.dz = Q.delta = 0;
    if (n >= kStaged) return Q;
    int seg, y, z;
    if (n < 192) {  // x = -2, -1 and x = 8, 9: rows of the tile and its faces
        seg = n & 1 ? 3 : 0;
        mg_face_row(n >> 1, y, z);
    } else {        // the tile's own x range: those rows, the next ones out, the edges
        const int m = n - 192, r = m >> 1;
        seg = 1 + (m & 1);
        if (r < 96) mg_face_row(r, y, z);
        else if (r < 112) { y = r < 104 ? -2 : 9; z = r & 7; }
        else if (r < 128) { y = r & 7; z = r < 120 ? -2 : 9; }
        else { y = (r & 1) ? 8 : -1; z = (r & 2) ? 8 : -1; }
    }
    const int lx = seg == 0 ? 4 : (seg == 3 ? 0 : 4 * (seg - 1));
    Q.dx = seg == 0 ? -1 : (seg == 3 ? 1 : 0);
    Q.dy = y < 0 ? -1 : (y > 7 ? 1 : 0);
    Q.dz = z < 0 ? -1 : (z > 7 ? 1 : 0);
    Q.local = lx | ((y - 8 * Q.dy) << 3) | ((z - 8 * Q.dz) << 6);
    Q.delta = (Q.dx + D.tx * (Q.dy + D.ty * Q.dz)) * 512 + Q.local;
    Q.box = 4 * seg + kBX * ((y + 2) + kBY * (z + 2));
    return Q;
}
// a tile of the list: its key and its coordinates (inner: no neighbour lies
// outside the grid)
struct MgTile {
    uint32_t key;
    int tx, ty, tz;
    bool inner;
};
__device__ __forceinline__ MgTile mg_tile(const MgLevel& L, uint32_t n) {
    MgTile T;
    T.key = L.tiles[n];
    const uint32_t row = T.key / (uint32_t)L.D.tx;
    T.tx = (int)(T.key - row * (uint32_t)L.D.tx);
    T.tz = (int)(row / (uint32_t)L.D.ty);
    T.ty = (int)(row - (uint32_t)T.tz * (uint32_t)L.D.ty);
    T.inner = T.tx > 0 && T.ty > 0 && T.tz > 0 && T.tx < L.D.tx - 1 && T.ty < L.D.ty - 1 && T.tz < L.D.tz - 1;
    return T;
}
// whether the quad lies in the grid, and its first slot
__device__ __forceinline__ bool mg_quad_in(const MgQuad& Q, const MgTile& T, const NatDims& D) {
    return Q.box >= 0 && (T.inner || ((unsigned)(T.tx + Q.dx) < (unsigned)D.tx && (unsigned)(T.ty + Q.dy) < (unsigned)D.ty &&
                                      (unsigned)(T.tz + Q.dz) < (unsigned)D.tz));
}
__device__ __forceinline__ uint32_t mg_quad_slot(const MgQuad& Q, const MgTile& T) { return (uint32_t)((int)(T.key << 9) + Q.delta); }
__device__ __forceinline__ float f4(const float4& v, int m) { return m == 0 ? v.x : (m == 1 ? v.y : (m == 2 ? v.z : v.w)); }
__device__ __forceinline__ void f4set(float4& v, int m, float x) {
    if (m == 0) v.x = x; else if (m == 1) v.y = x; else if (m == 2) v.z = x; else v.w = x;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
// a * x on the fluid cells by D^-1, 0 elsewhere
__device__ __forceinline__ float4 mg_over_diag(uint32_t c4, const float4& x, float a, const float* inv) {
    if (c4 == kAllSix) {
        const float s = a * (1.0f / 6.0f);
        return make_float4(s * x.x, s * x.y, s * x.z, s * x.w);
    }
    float4 o;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const uint32_t c = (c4 >> (8 * m)) & 0xFFu;
        f4set(o, m, (c & kCellFluid) ? a * inv[c & 7u] * f4(x, m) : 0.0f);
    }
    return o;
}
// a sweep of a cell, u + w (v - D^-1 A u): with D^-1 A u = u - nb/d this is
// (1 - w) u + w v + w nb/d; a fluid cell between six solid ones has A = 0 (and
// v = 0) and keeps its u
__device__ __forceinline__ float mg_sweep_cell(uint32_t c, float u, float v, float nb, const float* inv) {
    const uint32_t d = c & 7u;
    return (c & kCellFluid) ? fmaf(d ? 1.0f - kMgOmega : 1.0f, u, fmaf(kMgOmega, v, kMgOmega * inv[d] * nb)) : 0.0f;
}
__device__ __forceinline__ float4 mg_sweep4(uint32_t c4, const float4& u, const float4& v, const float4& nb, const float* inv) {
    float4 o;
    if (c4 == kAllSix) {
        constexpr float a = 1.0f - kMgOmega, b = kMgOmega * (1.0f / 6.0f);
#pragma unroll
        for (int m = 0; m < 4; ++m) f4set(o, m, fmaf(a, f4(u, m), fmaf(kMgOmega, f4(v, m), b * f4(nb, m))));
        return o;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) f4set(o, m, mg_sweep_cell((c4 >> (8 * m)) & 0xFFu, f4(u, m), f4(v, m), f4(nb, m), inv));
    return o;
}
// x on the fluid cells, 0 elsewhere
__device__ __forceinline__ float4 mg_fluid(uint32_t c4, const float4& x) {
    if (c4 == kAllSix) return x;
    float4 o;
#pragma unroll
    for (int m = 0; m < 4; ++m) f4set(o, m, ((c4 >> (8 * m)) & kCellFluid) ? f4(x, m) : 0.0f);
    return o;
}
__device__ __forceinline__ float4 mg_add(const float4& a, const float4& b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ float4 mg_axpy(float a, const float4& x, const float4& y) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
// neighbour sums of the quad at float index b of a box of row stride SY and
// plane stride SZ, c its own values.  The tile's two quads of a row lie in
// neighbouring lanes (an even and an odd one) of a fully active warp, so
// their common x neighbours come by a shuffle; the outer one is read.
template <int SY, int SZ>
__device__ __forceinline__ float4 mg_quad_nb(const float* v, int b, int half, const float4& c) {
    const float got = __shfl_xor_sync(0xffffffffu, half ? c.x : c.w, 1);
    const float outer = v[b + (half ? 4 : -1)];
    const float l = half ? got : outer, r = half ? outer : got;
    const float4 ym = ld4(v + b - SY), yp = ld4(v + b + SY), zm = ld4(v + b - SZ), zp = ld4(v + b + SZ);
    float4 s;
    s.x = ((l + c.y) + (ym.x + yp.x)) + (zm.x + zp.x);
    s.y = ((c.x + c.z) + (ym.y + yp.y)) + (zm.y + zp.y);
    s.z = ((c.y + c.w) + (ym.z + yp.z)) + (zm.z + zp.z);
    s.w = ((c.z + r) + (ym.w + yp.w)) + (zm.w + zp.w);
    return s;
}
template <int SY, int SZ>
__device__ __forceinline__ float mg_cell_nb(const float* v, int b) {
    return ((v[b - 1] + v[b + 1]) + (v[b - SY] + v[b + SY])) + (v[b - SZ] + v[b + SZ]);
}
// The first sweep's places, as constants of the thread: threads 0 .. 191 a
// quad of the 96 rows, threads 192 .. 255 two of the cells x = -1, x = 8.
struct MgSweep1 {
    int box, t, half;     // the quad's float index in the box and in the sweep's box
    int cell[2], tcell[2];
};
__device__ __forceinline__ MgSweep1 mg_sweep1(int tid) {
    MgSweep1 P;
    int y, z;
    mg_face_row(tid < 192 ? tid >> 1 : 0, y, z);
    P.half = tid & 1;
    P.box = 4 * (1 + P.half) + kBX * ((y + 2) + kBY * (z + 2));
    P.t = 4 * (1 + P.half) + kBX * ((y + 1) + 10 * (z + 1));
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int row = tid & 63, x = k ? 8 : -1;
        P.cell[k] = (x + 4) + kBX * ((row & 7) + 2 + kBY * ((row >> 3) + 2));
        P.tcell[k] = (x + 4) + kBX * ((row & 7) + 1 + 10 * ((row >> 3) + 1));
    }
    return P;
}
// the tile's own quad of threads 0 .. 127
struct MgOwn {
    int half, ly, lz, box, t;
    uint32_t slot;
};
__device__ __forceinline__ MgOwn mg_own(int tid) {
    MgOwn P;
    const int row = (tid & 127) >> 1;
    P.half = tid & 1;
    P.ly = row & 7;
    P.lz = row >> 3;
    P.box = 4 * (1 + P.half) + kBX * ((P.ly + 2) + kBY * (P.lz + 2));
    P.t = 4 * (1 + P.half) + kBX * ((P.ly + 1) + 10 * (P.lz + 1));
    P.slot = (uint32_t)(4 * P.half + 8 * P.ly + 64 * P.lz);
    return P;
}
__device__ __forceinline__ uint32_t mg_code(const uint32_t* cb, int cell) { return (cb[cell >> 2] >> (8 * (cell & 3))) & 0xFFu; }

// pre-smoothing and restriction of level F into C.  With v = D^-1 r:
//   t1 = w v, t = t1 + w D^-1 (r - A t1) = (2 w - w^2) v + w^2 D^-1 sum v
//   (the sum over the neighbours; t is kept in F.t),
//   C.r[parent] = 1/2 sum over the 8 children of r - A t (fluid parents; the
//   parents of a tile are all written by it, and parents of tiles off the
//   list are never fluid)
template <bool SCALE = false>
__global__ void __launch_bounds__(kMgThreads, kMgCtas) mg_down_kernel(MgLevel F, MgLevel C, const int* halt, MgScale sc) {
    // SCALE (C the coarsest level): the sum of C.r^2 and the count over the
    // fluid parents this CTA writes, then *sc.inv_s as mg_scale_kernel sets it
    __shared__ double acc[SCALE ? 2 * 64 : 1];
    if (SCALE && threadIdx.x < 64) acc[2 * threadIdx.x] = acc[2 * threadIdx.x + 1] = 0.0;
    __shared__ uint32_t cb[kBoxF / 4];              // four codes per quad
    __shared__ __align__(16) float vb[kBoxF];       // v = D^-1 r
    __shared__ __align__(16) float tb[kT1F];        // t
    __shared__ float S[256];                        // x-pair sums of the residual
    __shared__ float inv[8];
    mg_inv_table(inv);
    const int tid = threadIdx.x;
    MgQuad Q[kQPer];
#pragma unroll
    for (int m = 0; m < kQPer; ++m) Q[m] = mg_quad(tid + m * kMgThreads, F.D);
    const MgSweep1 P = mg_sweep1(tid);
    const MgOwn O = mg_own(tid);
    pdl_wait();
    if (SCALE) pdl_trigger();
    if (mg_halted(halt)) return;
    const uint32_t n = *F.d_ntiles;
    uint32_t pc[kQPer];
    float4 pr[kQPer], ro;
    MgTile T{};
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto fetch = [&](uint32_t tt) {
        T = mg_tile(F, tt);
#pragma unroll
        for (int m = 0; m < kQPer; ++m) {
            pc[m] = 0u;
            pr[m] = zero4;
            if (mg_quad_in(Q[m], T, F.D)) {
                const uint32_t sl = mg_quad_slot(Q[m], T);
                pc[m] = *reinterpret_cast<const uint32_t*>(F.cell + sl);
                pr[m] = ld4(F.r + sl);
            }
        }
        if (tid < 128) ro = ld4(F.r + ((T.key << 9) | O.slot));
    };
    __syncthreads();  // the 1/d table
    for (uint32_t tt = blockIdx.x; tt < n; tt += gridDim.x) {
        fetch(tt);
        const uint32_t now = T.key;
        const int cx = 4 * T.tx, cy = 4 * T.ty, cz = 4 * T.tz;  // the tile's first parent
        const float4 r = ro;
#pragma unroll
        for (int m = 0; m < kQPer; ++m)
            if (Q[m].box >= 0) {
                cb[Q[m].box >> 2] = pc[m];
                st4(vb + Q[m].box, mg_over_diag(pc[m], pr[m], 1.0f, inv));
            }
        __syncthreads();
        constexpr float kA = 2.0f * kMgOmega - kMgOmega * kMgOmega, kB = kMgOmega * kMgOmega;
        if (tid < 192) {
            const uint32_t c4 = cb[P.box >> 2];
            const float4 v = ld4(vb + P.box);
            const float4 nb = mg_quad_nb<kBX, kBX * kBY>(vb, P.box, P.half, v);
            st4(tb + P.t, mg_axpy(kA, v, mg_over_diag(c4, nb, kB, inv)));
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t c = mg_code(cb, P.cell[k]);
                const float b = (c & kCellFluid) ? kB * inv[c & 7u] : 0.0f;
                tb[P.tcell[k]] = fmaf(kA, vb[P.cell[k]], b * mg_cell_nb<kBX, kBX * kBY>(vb, P.cell[k]));
            }
        }
        __syncthreads();
        if (tid < 128) {
            const uint32_t c4 = cb[O.box >> 2];
            const float4 tv = ld4(tb + O.t);
            const float4 nb = mg_quad_nb<kBX, kBX * 10>(tb, O.t, O.half, tv);
            float res[4];
            if (c4 == kAllSix) {
#pragma unroll
                for (int m = 0; m < 4; ++m) res[m] = f4(r, m) - (6.0f * f4(tv, m) - f4(nb, m));
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t c = (c4 >> (8 * m)) & 0xFFu;
                    res[m] = (c & kCellFluid) ? f4(r, m) - ((float)(c & 7u) * f4(tv, m) - f4(nb, m)) : 0.0f;
                }
            }
            st4(F.t + ((now << 9) | O.slot), tv);
            S[(2 * O.half) + 4 * (O.ly + 8 * O.lz)] = res[0] + res[1];
            S[(2 * O.half + 1) + 4 * (O.ly + 8 * O.lz)] = res[2] + res[3];
        }
        __syncthreads();
        if (tid >= 192) {  // parent (pi, pj, pk) of the tile's 4^3 parents
            const int q = tid - 192;
            const int pi = q & 3, pj = (q >> 2) & 3, pk = q >> 4;
            const int s0 = pi + 4 * (2 * pj + 8 * 2 * pk);
            const float sum = (S[s0] + S[s0 + 4]) + (S[s0 + 32] + S[s0 + 36]);
            const uint32_t p = mg_slot(cx + pi, cy + pj, cz + pk, C.D);
            const bool fl = (C.cell[p] & kCellFluid) != 0;
            const float v = fl ? 0.5f * sum : 0.0f;
            C.r[p] = v;
            if (SCALE && fl) {
                acc[2 * q] += (double)v * (double)v;
                acc[2 * q + 1] += 1.0;
            }
        }
        // the next tile's staging writes only vb and cb, which nothing reads
        // past the barrier above; its S comes two barriers later
    }
    if (SCALE) {
        __syncthreads();
        double out[2];
        const bool last = mg_last_cta_sum2(tid < 64 ? acc[2 * tid] : 0.0, tid < 64 ? acc[2 * tid + 1] : 0.0,
                                           sc.partials, sc.ticket, out);
        if (last && tid == 0) *sc.inv_s = out[0] > 0.0 ? (float)(1.0 / sqrt(out[0] / fmax(out[1], 1.0))) : 1.0f;
    }
}

// two damped Jacobi sweeps (mg_sweep_cell) from a start vector u, with v = D^-1 r;
// the second one's result is L.z.  MODE 0: u = L.t + C.z[parent] (prolongation
// of the coarse correction; post-smoothing; C.z is zero off the coarse fluid
// cells); MODE 1: u = zn + v (the coarsest level with the network output zn);
// MODE 2: u = w v (the coarsest level without the network); MODE 3: u = zn
// (the coarsest level after a CG solve into zn).  DOT (MODE 0 on level 0):
// FCG's dot products of the z it writes (MgDot), reduced by the last CTA.
template <int MODE, bool DOT = false>
__global__ void __launch_bounds__(kMgThreads, kMgCtas) mg_sweeps_kernel(MgLevel L, MgLevel C, const float* __restrict__ zn,
                                                                        const int* halt, MgDot dot) {
    __shared__ uint32_t cb[kBoxF / 4];
    __shared__ __align__(16) float vb[kBoxF];
    __shared__ __align__(16) float ub[kBoxF];
    __shared__ __align__(16) float tb[kT1F];
    __shared__ float inv[8];
    __shared__ double acc[DOT ? 2 * 128 : 1];  // r.z, z.q of each storing thread
    mg_inv_table(inv);
    const int tid = threadIdx.x;
    if (DOT && tid < 128) acc[2 * tid] = acc[2 * tid + 1] = 0.0;
    MgQuad Q[kQPer];
#pragma unroll
    for (int m = 0; m < kQPer; ++m) Q[m] = mg_quad(tid + m * kMgThreads, L.D);
    const MgSweep1 P = mg_sweep1(tid);
    const MgOwn O = mg_own(tid);
    pdl_wait();
    if (MODE != 0) pdl_trigger();
    if (mg_halted(halt)) return;
    const uint32_t n = *L.d_ntiles;
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint32_t pc[kQPer];
    MgTile T{};
    float4 pr[kQPer], pu[kQPer];
    float2 pe[kQPer];      // MODE 0: the two parents' corrections
    auto fetch = [&](uint32_t tt) {
        T = mg_tile(L, tt);
#pragma unroll
        for (int m = 0; m < kQPer; ++m) {
            pc[m] = 0u;
            pr[m] = pu[m] = zero4;
            pe[m] = make_float2(0.0f, 0.0f);
            if (mg_quad_in(Q[m], T, L.D)) {
                const uint32_t sl = mg_quad_slot(Q[m], T);
                pc[m] = *reinterpret_cast<const uint32_t*>(L.cell + sl);
                pr[m] = ld4(L.r + sl);
                if (MODE == 0) {
                    pu[m] = ld4(L.t + sl);
                    // parents of x, x+1 and of x+2, x+3: consecutive coarse cells
                    const int l = Q[m].local;
                    const uint32_t ps = mg_slot(4 * (T.tx + Q[m].dx) + ((l & 7) >> 1), 4 * (T.ty + Q[m].dy) + ((l >> 4) & 3),
                                                4 * (T.tz + Q[m].dz) + (l >> 7), C.D);
                    pe[m] = *reinterpret_cast<const float2*>(C.z + ps);
                } else if (MODE == 1 || MODE == 3) {
                    pu[m] = ld4(zn + sl);
                }
            }
        }
    };
    __syncthreads();  // the 1/d table
    for (uint32_t tt = blockIdx.x; tt < n; tt += gridDim.x) {
        fetch(tt);
        const uint32_t now = T.key;
#pragma unroll
        for (int m = 0; m < kQPer; ++m)
            if (Q[m].box >= 0) {
                const float4 v = mg_over_diag(pc[m], pr[m], 1.0f, inv);
                float4 u = pu[m];
                if (MODE == 0) u = mg_add(u, make_float4(pe[m].x, pe[m].x, pe[m].y, pe[m].y));
                if (MODE == 1) u = mg_add(u, v);
                if (MODE == 2) u = make_float4(kMgOmega * v.x, kMgOmega * v.y, kMgOmega * v.z, kMgOmega * v.w);
                cb[Q[m].box >> 2] = pc[m];
                st4(vb + Q[m].box, v);
                st4(ub + Q[m].box, mg_fluid(pc[m], u));
            }
        __syncthreads();
        float4 q4 = zero4, r4 = zero4;
        if (DOT && tid < 128) {
            q4 = ld4(dot.q + ((now << 9) | O.slot));
            r4 = ld4(L.r + ((now << 9) | O.slot));
        }
        if (tid < 192) {
            const uint32_t c4 = cb[P.box >> 2];
            const float4 u = ld4(ub + P.box), v = ld4(vb + P.box);
            const float4 nb = mg_quad_nb<kBX, kBX * kBY>(ub, P.box, P.half, u);
            st4(tb + P.t, mg_sweep4(c4, u, v, nb, inv));
        } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                tb[P.tcell[k]] = mg_sweep_cell(mg_code(cb, P.cell[k]), ub[P.cell[k]], vb[P.cell[k]],
                                               mg_cell_nb<kBX, kBX * kBY>(ub, P.cell[k]), inv);
            }
        }
        __syncthreads();
        if (tid < 128) {
            const uint32_t zs = (now << 9) | O.slot;
            const uint32_t c4 = cb[O.box >> 2];
            const float4 u = ld4(tb + O.t), v = ld4(vb + O.box);
            const float4 nb = mg_quad_nb<kBX, kBX * 10>(tb, O.t, O.half, u);
            const float4 z = mg_sweep4(c4, u, v, nb, inv);
            st4(L.z + zs, z);
            if (DOT) {
                double rz = 0.0, zq = 0.0;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    if (!((c4 >> (8 * m)) & kCellFluid)) continue;
                    rz += (double)f4(r4, m) * (double)f4(z, m);
                    zq += (double)f4(z, m) * (double)f4(q4, m);
                }
                acc[2 * tid] += rz;
                acc[2 * tid + 1] += zq;
            }
        }
        __syncthreads();  // vb and cb before the next tile's staging
    }
    if (DOT) {
        double out[2];
        const bool last = mg_last_cta_sum2(tid < 128 ? acc[2 * tid] : 0.0, tid < 128 ? acc[2 * tid + 1] : 0.0,
                                           dot.partials, &dot.st->ticket, out);
        if (last && tid == 0) {
            PcgState* st = dot.st;
            st->beta = dot.init ? 0.0 : (st->pq > 0.0 ? -out[1] / st->pq : 0.0);
            st->rz = out[0];
            st->rz_prev = out[0];
            st->zq = out[1];
            if (out[0] == 0.0 || !isfinite(out[0]) || !isfinite(out[1])) { st->done = 3; st->halt = 1; }
        }
    }
}

// 1 / rms(r) over the fluid cells of a level (one CTA)
__global__ void __launch_bounds__(1024) mg_scale_kernel(MgLevel L, float* inv_s, const int* halt) {
    pdl_wait();
    if (mg_halted(halt)) return;
    __shared__ double sh[32];
    const uint32_t n = *L.d_ntiles;
    double rr = 0.0, nf = 0.0;
    for (uint32_t v = threadIdx.x; v < n * 512u; v += 1024u) {
        const uint32_t s = (L.tiles[v >> 9] << 9) | (v & 511u);
        if (L.cell[s] & kCellFluid) {
            const double r = L.r[s];
            rr += r * r;
            nf += 1.0;
        }
    }
    rr = block_sum_f64<1024>(rr, sh);
    __syncthreads();
    nf = block_sum_f64<1024>(nf, sh);
    if (threadIdx.x == 0) *inv_s = rr > 0.0 ? (float)(1.0 / sqrt(rr / fmax(nf, 1.0))) : 1.0f;
}

// Jacobi-PCG on one level in one CTA (the coarsest level: at most 4096
// slots): x = A^-1 b to |r| <= tol |b| or max_iter iterations, FP32 vectors
// and FP64 dots.  r, p, q are scratch vectors of the level's size.  Used for
// the training targets of the coarsest solve.
__global__ void __launch_bounds__(1024) mg_cg_kernel(MgLevel L, const float* __restrict__ b, float* __restrict__ x,
                                                     float* __restrict__ r, float* __restrict__ p, float* __restrict__ q,
                                                     double tol, int max_iter, int* iters, const int* halt) {
    if (mg_halted(halt)) return;
    __shared__ double sh[32];
    __shared__ double bc;
    const uint32_t n = *L.d_ntiles * 512u;
    auto slot = [&](uint32_t v) { return (L.tiles[v >> 9] << 9) | (v & 511u); };
    auto bsum = [&](double v) {
        v = block_sum_f64<1024>(v, sh);
        if (threadIdx.x == 0) bc = v;
        __syncthreads();
        return bc;
    };
    double bb = 0.0, rz = 0.0;
    for (uint32_t v = threadIdx.x; v < n; v += 1024u) {
        const uint32_t s = slot(v);
        const uint8_t c = L.cell[s];
        const float bv = (c & kCellFluid) ? b[s] : 0.0f;
        x[s] = 0.0f;
        r[s] = bv;
        const float z = mg_dinv(c) * bv;
        p[s] = z;
        bb += (double)bv * bv;
        rz += (double)bv * z;
    }
    bb = bsum(bb);
    rz = bsum(rz);
    int it = 0;
    if (bb > 0.0) {
        for (it = 1; it <= max_iter; ++it) {
            double pq = 0.0;
            for (uint32_t v = threadIdx.x; v < n; v += 1024u) {
                const uint32_t s = slot(v);
                const uint8_t c = L.cell[s];
                float qv = 0.0f;
                if (c & kCellFluid) {
                    int i, j, k;
                    mg_cell_of(s >> 9, (int)(s & 511u), L.D, i, j, k);
                    const float nb = mg_nb_sum(i, j, k, L.D, L.cell, [&](uint32_t u) { return p[u]; });
                    qv = (float)(c & 7u) * p[s] - nb;
                }
                q[s] = qv;
                pq += (double)p[s] * qv;
            }
            pq = bsum(pq);
            if (!(pq > 0.0)) break;
            const float alpha = (float)(rz / pq);
            double rr = 0.0, rzn = 0.0;
            for (uint32_t v = threadIdx.x; v < n; v += 1024u) {
                const uint32_t s = slot(v);
                x[s] += alpha * p[s];
                const float rv = r[s] - alpha * q[s];
                r[s] = rv;
                rr += (double)rv * rv;
                rzn += (double)rv * (mg_dinv(L.cell[s]) * rv);
            }
            rr = bsum(rr);
            rzn = bsum(rzn);
            if (rr <= tol * tol * bb) break;
            const float beta = (float)(rzn / rz);
            rz = rzn;
            for (uint32_t v = threadIdx.x; v < n; v += 1024u) {
                const uint32_t s = slot(v);
                p[s] = mg_dinv(L.cell[s]) * r[s] + beta * p[s];
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0 && iters) *iters = it;
}

// ------------------------------------------------------------ host side
int mg_plan(int nx, int ny, int nz, float h, MgLevel* L, int max_levels) {
    int ex = nx, ey = ny, ez = nz, levels = 0;
    float hl = h;
    while (levels < max_levels) {
        MgLevel& l = L[levels];
        l = MgLevel{};
        l.ex = ex; l.ey = ey; l.ez = ez;
        l.D.nx = (ex + 7) & ~7; l.D.ny = (ey + 7) & ~7; l.D.nz = (ez + 7) & ~7;
        l.D.tx = l.D.nx / 8; l.D.ty = l.D.ny / 8; l.D.tz = l.D.nz / 8;
        l.D.ox = l.D.oy = l.D.oz = 0.0f;
        l.D.h = hl;
        l.D.inv_h = 1.0f / hl;
        l.ntiles = (uint32_t)(l.D.tx * l.D.ty * l.D.tz);
        ++levels;
        if (ex <= kMgCoarsest && ey <= kMgCoarsest && ez <= kMgCoarsest) break;
        ex = (ex + 1) / 2; ey = (ey + 1) / 2; ez = (ez + 1) / 2;
        hl *= 2.0f;
    }
    return levels;
}

// CTAs of the smoothing kernels: four per SM (grid0 on level 0) and no more
// than the level has tiles
static int mg_grid(const MgLevel& L, int grid0, int level) {
    if (level == 0) return grid0;
    return (int)(L.ntiles < 592u ? L.ntiles : 592u);
}

int mg_build(const MgHierarchy& H, const int* halt, cudaStream_t s) {
    for (int l = 1; l < H.levels; ++l) {
        const MgLevel& C = H.L[l];
        const int g = (int)(C.ntiles < 1184u ? C.ntiles : 1184u);
        mg_coarsen_kernel<<<g, 512, 0, s>>>(H.L[l - 1], C, halt);
        mg_codes_kernel<<<g, 512, 0, s>>>(C, halt);
        // tiles off the list are not written: their corrections read as zero
        FLIP_CUDA_TRY(cudaMemsetAsync(C.z, 0, (size_t)C.ntiles * 512u * sizeof(float), s));
        // the smoothing of an intermediate level walks its tiles with fluid
        // cells (flags in C.active); the coarsest keeps every tile
        if (l + 1 < H.levels) {
            const int rc = nat_launch_fluid_tiles(C.type, C.active, C.ntiles, const_cast<uint32_t*>(C.tiles),
                                                  const_cast<uint32_t*>(C.d_ntiles), (uint64_t)C.ntiles * 512u, s);
            if (rc != FLIP_OK) return rc;
        }
    }
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int mg_down(const MgHierarchy& H, const int* halt, int grid0, cudaStream_t s, bool scale) {
    if (scale && H.levels < 2) return FLIP_ERR_ARG;
    const MgScale ns{};
    for (int l = 0; l + 1 < H.levels; ++l) {
        const int g = mg_grid(H.L[l], grid0, l);
        if (scale && l + 2 == H.levels) {
            if (2 * g > kMgScalePartials) return FLIP_ERR_ARG;
            const MgScale sc{H.scale_partials, H.scale_ticket, H.inv_s};
            FLIP_CUDA_TRY(pdl_launch(mg_down_kernel<true>, g, kMgThreads, 0, s, H.L[l], H.L[l + 1], halt, sc));
        } else {
            FLIP_CUDA_TRY(pdl_launch(mg_down_kernel<false>, g, kMgThreads, 0, s, H.L[l], H.L[l + 1], halt, ns));
        }
    }
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int mg_coarsest(const MgHierarchy& H, const float* zn, const int* halt, cudaStream_t s, bool solved) {
    const int c = H.levels - 1;
    const MgLevel& L = H.L[c];
    const int g = mg_grid(L, 592, c);
    const float* z0 = zn;
    const MgDot nd{};
    if (zn && solved) FLIP_CUDA_TRY(pdl_launch(mg_sweeps_kernel<3>, g, kMgThreads, 0, s, L, L, z0, halt, nd));
    else if (zn) FLIP_CUDA_TRY(pdl_launch(mg_sweeps_kernel<1>, g, kMgThreads, 0, s, L, L, z0, halt, nd));
    else FLIP_CUDA_TRY(pdl_launch(mg_sweeps_kernel<2>, g, kMgThreads, 0, s, L, L, z0, halt, nd));
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int mg_up(const MgHierarchy& H, const int* halt, int grid0, cudaStream_t s, const MgDot* dot) {
    if (dot && (H.levels < 2 || 2 * grid0 > 4 * kPcgBlocks)) return FLIP_ERR_ARG;  // partials: 4 x kPcgBlocks
    const MgDot nd{};
    for (int l = H.levels - 2; l >= 0; --l) {
        const int g = mg_grid(H.L[l], grid0, l);
        if (l == 0 && dot)
            FLIP_CUDA_TRY(pdl_launch(mg_sweeps_kernel<0, true>, g, kMgThreads, 0, s, H.L[l], H.L[l + 1],
                                     (const float*)nullptr, halt, *dot));
        else
            FLIP_CUDA_TRY(pdl_launch(mg_sweeps_kernel<0>, g, kMgThreads, 0, s, H.L[l], H.L[l + 1], (const float*)nullptr,
                                     halt, nd));
    }
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int mg_cg(const MgLevel& L, const float* b, float* x, float* r, float* p, float* q, double tol, int max_iter, int* iters,
          cudaStream_t s, const int* halt) {
    mg_cg_kernel<<<1, 1024, 0, s>>>(L, b, x, r, p, q, tol, max_iter, iters, halt);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int mg_input_scale(const MgHierarchy& H, const int* halt, cudaStream_t s) {
    FLIP_CUDA_TRY(pdl_launch(mg_scale_kernel, 1, 1024, 0, s, H.L[H.levels - 1], H.inv_s, halt));
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

}  // namespace flip
