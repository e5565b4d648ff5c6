// pcg_resident.cu -- the whole Jacobi-PCG solve as one cooperative kernel
// (small boxes: one cluster) that keeps the solver's vectors on the chip.
//
// A CTA per SM owns a run of consecutive tiles for the whole solve.  p of its
// tiles always lives in shared memory; w = D^-1 r, t = D^-1 A p and xg (the
// FP32 increments of the solution) follow as far as there is room (w first,
// with kRegPasses x 4 tiles of it in registers where shared memory is
// short), the rest streams through L2.  There is one grid-wide exchange per
// iteration:
//   - q = A p, t = D^-1 q, and the sums p.q, w.q, q.t, r.z, r.r together;
//   - alpha = r.z / p.q, and the next r.z follows from the sums:
//     r'.z' = r.z - 2 alpha w.q + alpha^2 q.t.  It serves beta only: the r.z
//     and r.r that alpha and the stopping test use are summed from the
//     vector itself every iteration, so nothing accumulates (the prediction
//     differs from the sum by the rounding of w, 2^-24 per voxel);
//   - a face cell of another CTA's tile is followed locally: w' = w - alpha t
//     and p' = w' + beta p with the neighbour's t, the same operations on the
//     same values as its owner's.  A face between two tiles of one CTA is
//     read in place.
// What crosses between CTAs carries its own iteration number: a face cell's t
// is a word of 32 value and 32 tag bits in a mailbox, the five sums are ten
// such words in a packet.  A reader polls for the tag, so neither side needs
// a fence, and no line is polled by two CTAs.  The sums go in two hops, to the
// CTAs of the own group (a dozen) and then from group to group; all CTAs add
// the same packets in the same order, so the exchange is a barrier, a
// reduction and a broadcast at once.  (Packets from every CTA to every other,
// one hop, took 4.5 us on 148 CTAs: 740 scattered stores per CTA.)
#include <stddef.h>
#include "common.cuh"
#include "native.cuh"

namespace flip {

namespace {

constexpr int kThreads = 512;
constexpr int kGroups = 4;                 // tiles in flight: 128 threads a tile, four x-cells a thread
constexpr int kRegPasses = 10;             // tiles of a group whose w stays in registers (the large variant)
constexpr int kSums = 5;                   // p.q, w.q, q.t, r.z, r.r
constexpr int kMaxTiles = kResidentTiles;  // tiles per CTA (their p and codes fill the shared memory)
constexpr int kMaxFaces = 6 * kMaxTiles;
constexpr int kTileFloats = 512 + 64;      // p, and the cell codes of four cells in 16 bits
constexpr uint32_t kInner = 1u << 31;      // the face is read from another tile of this CTA
constexpr uint32_t kFar = 1u << 30;        // the face's values are in global memory (no room in the pool)
constexpr uint32_t kPoolMask = kFar - 1u;
constexpr uint32_t kSpin = 1u << 21;       // polls of a word before giving up (about two seconds)

struct Face {
    uint32_t src;   // first face slot of the neighbouring tile
    uint32_t in;    // mailbox word of the neighbour's face
    uint32_t pad;
    uint32_t t_f;   // own tile << 3 | face (0..5: -x, +x, -y, +y, -z, +z)
};
struct alignas(16) Fixed {
    uint32_t tab[kMaxTiles][8];  // per tile and face: pool offset | kInner / kFar; [6]: faces with mail (bits); [7]: their first mailbox word
    Face face[kMaxFaces];
    uint32_t key[kMaxTiles], coord[kMaxTiles];
    double red[kSums][kThreads / 32];
    double rr, rr_true, pq;  // kept for the state written back
    double rz;               // r.z of the last exchange
    float alpha, beta;       // the step that follows it
    uint32_t verdict;        // 0: a step, 1: convergence claimed, 2: breakdown
    float inv[8];
    uint32_t nface, lost;
};
constexpr int kSmemMax = 232448 - 1024;
constexpr int kPoolFloats = (kSmemMax - (int)sizeof(Fixed)) / 4;
static_assert(64 + kTileFloats * kMaxTiles <= kPoolFloats, "the tiles' p and codes fit the shared memory");
static_assert(sizeof(Fixed) % 16 == 0 && offsetof(Fixed, tab) % 16 == 0, "16-byte reads of the pool and of the table");

__device__ __forceinline__ float4 ld4cg(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
// y + a x
__device__ __forceinline__ float4 axpy4(const float4& x, const float4& y, float a) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
__device__ __forceinline__ void ld_relaxed_u64x2(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_relaxed_u64x2(unsigned long long* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
// the address of a word of this CTA's shared memory in CTA `rank` of the
// cluster; relaxed accesses to such words
__device__ __forceinline__ uint32_t cluster_addr(uint32_t smem, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster_u64x2(uint32_t p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_cluster_u64x2(uint32_t p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.cluster.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(p) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// small unsigned integer -> float without the conversion unit
__device__ __forceinline__ float small_float(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.0f; }

// sums of five values over a warp in 16 shuffles: lanes trade halves of the
// set of values instead of all of it, so that after the step over 16, 8 and
// 4 lanes each lane follows one value; the lane holding value k in v[0] is
// kLaneOf[k] (value 0 of lanes 0-3, 1 of 4-7, 2 of 8-15, 3 of 16-23, 4 of 24-31)
__device__ __forceinline__ double warp_sum5(const double (&v)[kSums], int lane) {
    const bool h = lane & 16, q = lane & 8, e = lane & 4;
    double a = h ? v[3] : v[0], b = h ? v[4] : v[1], c = h ? 0.0 : v[2];
    a += __shfl_xor_sync(0xffffffffu, h ? v[0] : v[3], 16);
    b += __shfl_xor_sync(0xffffffffu, h ? v[1] : v[4], 16);
    c += __shfl_xor_sync(0xffffffffu, h ? v[2] : 0.0, 16);
    // low half: a b | c, high half: a | b
    const double s0 = h ? (q ? a : b) : (q ? a : c), s1 = h ? 0.0 : b;
    const double r0 = __shfl_xor_sync(0xffffffffu, s0, 8), r1 = __shfl_xor_sync(0xffffffffu, h ? 0.0 : (q ? b : 0.0), 8);
    double x = h ? (q ? b : a) : (q ? c : a), y = (h || q) ? 0.0 : s1;
    x += r0;
    y += r1;
    // lanes 0-7 hold two values (x: 0, y: 1), the others one
    const bool two = !h && !q;
    const double s2 = two ? (e ? x : y) : x;
    const double r2 = __shfl_xor_sync(0xffffffffu, s2, 4);
    double z = two ? (e ? y : x) : x;
    z += r2;
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    return z;
}
// which value warp_sum5 leaves in a lane, and whether the lane is the first to hold it
__device__ __forceinline__ int sum5_of(int lane) { return lane < 4 ? 0 : (lane < 8 ? 1 : (lane < 16 ? 2 : (lane < 24 ? 3 : 4))); }
__device__ __forceinline__ bool sum5_first(int lane) { return lane == 0 || lane == 4 || lane == 8 || lane == 16 || lane == 24; }

// one CTA's view of the solve
struct Args {
    const uint32_t* tiles;
    const uint32_t* tcoord;
    NatDims D;
    double* x;
    float *xg, *r, *t;
    float* far;               // [tile of the list][face][p, w]: faces the pools have no room for
    unsigned long long* mail; // [2][tile of the list][face][64 cells]: tag << 32 | t
    uint32_t mail_half;       // words of one half
    const float* b;
    const uint8_t* cell;
    PcgState* st;
    unsigned long long* slots;  // packets, [2][hop][reader][two words of a sum][lane]
    uint32_t ctas;
    uint32_t* epoch;          // the last tag of the solve before
    uint32_t* err;
    int chunk, limit;
    ResidentHook hook;
};
__device__ __forceinline__ unsigned long long tagged(uint32_t tag, uint32_t v) { return ((unsigned long long)tag << 32) | v; }

// One reader's packets of one hop, a 128-byte line each
constexpr uint32_t kPacketWords = 16;
constexpr uint32_t kSlotWords = kPcgSlotWords;
static_assert(kSlotWords == 32 * kPacketWords, "a packet for every lane");

// The grid-wide exchange of five sums.  The CTAs form `groups` runs of equal
// size (up to one); hop 1 goes to every CTA of the own group, hop 2 from a
// member of each group to the members of the same rank elsewhere.  kLocal: the
// CTAs are one cluster, one group, and the packets go to the readers' shared
// memory.  That took an iteration on 48 tiles (12 CTAs) from 4.27 us with
// packets through L2 to 3.83, on 8 tiles from 4.04 to 3.62 (3.26 us on 48 tiles
// with the scalars taken once); 16 CTAs is the largest cluster, and with four
// tiles each it holds boxes of up to 64.
constexpr uint32_t kClusterMax = 16;
constexpr uint32_t kLocalWords = 2 * kClusterMax * 2 * kSums;  // [2][sender][two words of a sum]
// kHook: with the test hook (kernels of their own: the checks in the polling
// loops cost 0.5 us an iteration on 392 tiles).
template <bool kLocal, bool kHook>
struct Exchange {
    unsigned long long* slots;
    uint32_t local;   // kLocal: the packets' address in shared memory
    Fixed* S;
    uint32_t ctas;    // stride of the packets
    uint32_t tag;     // number of the exchange in flight; its low bit picks the half
    uint32_t n;       // CTAs taking part
    uint32_t groups, group, first, size, rank;  // group's first CTA, its size, the own rank in it
    uint32_t hook_which, hook_tag, hook_polls;  // kHook: in force from that tag on

    __device__ __forceinline__ bool in_vain(uint32_t which) const { return kHook && which == hook_which && tag >= hook_tag; }
    __device__ __forceinline__ uint32_t polls() const { return kHook ? hook_polls : kSpin; }
    __device__ __forceinline__ uint32_t group_first(uint32_t g) const { return g * n / groups; }
    __device__ __forceinline__ void init(uint32_t count) {
        n = count;
        groups = 1;
        if (n > 32u)
            while (groups * groups < n) ++groups;
        group = 0;
        while (group + 1u < groups && group_first(group + 1u) <= blockIdx.x) ++group;
        first = group_first(group);
        size = group_first(group + 1u) - first;
        rank = blockIdx.x - first;
    }
    __device__ __forceinline__ unsigned long long* packet(uint32_t hop, uint32_t reader, uint32_t lane) const {
        return slots + (((size_t)(tag & 1u) * 2u + hop) * ctas + reader) * kSlotWords + kPacketWords * lane;
    }
    __device__ __forceinline__ uint32_t local_packet(uint32_t sender) const {
        return local + ((tag & 1u) * kClusterMax + sender) * (16u * kSums);
    }
    __device__ __forceinline__ void push(uint32_t hop, uint32_t reader, uint32_t lane, const double (&v)[kSums]) const {
        unsigned long long* q = kLocal ? nullptr : packet(hop, reader, lane);
        const uint32_t l = kLocal ? cluster_addr(local_packet(lane), reader) : 0u;
#pragma unroll
        for (int k = 0; k < kSums; ++k) {
            const unsigned long long u = (unsigned long long)__double_as_longlong(v[k]);
            const unsigned long long lo = tagged(tag, (uint32_t)u), hi = tagged(tag, (uint32_t)(u >> 32));
            if (kLocal) st_cluster_u64x2(l + 16u * k, lo, hi);
            else st_relaxed_u64x2(q + 2 * k, lo, hi);
        }
    }
    // lane l of the first `count` takes packet l.  The whole warp polls until
    // every packet is there (the other lanes look at the last one): lanes that
    // leave the loop one by one cost microseconds (13.5 us a two-hop exchange
    // on 148 CTAs, 2.6 us this way).
    __device__ __forceinline__ bool poll(uint32_t hop, uint32_t lane, uint32_t count, double (&v)[kSums]) const {
        const unsigned long long* q = kLocal ? nullptr : packet(hop, blockIdx.x, min(lane, count - 1u));
        const uint32_t l = kLocal ? local_packet(min(lane, count - 1u)) : 0u;
        unsigned long long u[2 * kSums];
        uint32_t spin = 0;
        bool ok;
        do {
            ok = !in_vain(hop);
#pragma unroll
            for (int k = 0; k < kSums; ++k) {
                if (kLocal) ld_cluster_u64x2(l + 16u * k, u[2 * k], u[2 * k + 1]);
                else ld_relaxed_u64x2(q + 2 * k, u[2 * k], u[2 * k + 1]);
            }
#pragma unroll
            for (int k = 0; k < 2 * kSums; ++k) ok = ok && (uint32_t)(u[k] >> 32) == tag;
            ok = __all_sync(0xffffffffu, ok);
        } while (!ok && ++spin < polls());
#pragma unroll
        for (int k = 0; k < kSums; ++k)
            v[k] = lane < count ? __longlong_as_double((long long)((u[2 * k + 1] << 32) | (uint32_t)u[2 * k])) : 0.0;
        return ok;
    }
    // the sums of the lanes' values, in every lane
    __device__ __forceinline__ void lanes_sum(double (&v)[kSums], int lane) const {
        const double z = warp_sum5(v, lane);
        v[0] = __shfl_sync(0xffffffffu, z, 0);
        v[1] = __shfl_sync(0xffffffffu, z, 4);
        v[2] = __shfl_sync(0xffffffffu, z, 8);
        v[3] = __shfl_sync(0xffffffffu, z, 16);
        v[4] = __shfl_sync(0xffffffffu, z, 24);
    }
    // v: this thread's terms in, the grid's sums out; false when a packet
    // never came.  kFence: writes of every CTA before are visible after.
    // The first warp does the exchange, the others call idle() meanwhile.
    // fin(sums): by the first warp, before the others go on.
    template <bool kFence, class Idle, class Fin>
    __device__ __forceinline__ bool sum(double (&v)[kSums], Idle idle, Fin fin) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const double z = warp_sum5(v, lane);
        if (sum5_first(lane)) S->red[sum5_of(lane)][warp] = z;
        __syncthreads();
        ++tag;
        if (warp == 0) {
            // four lanes a value, four warps' sums a lane
            double a = 0.0;
            if (lane < 4 * kSums) {
                const double* q = &S->red[lane >> 2][4 * (lane & 3)];
                a = (q[0] + q[1]) + (q[2] + q[3]);
            }
            a += __shfl_xor_sync(0xffffffffu, a, 1);
            a += __shfl_xor_sync(0xffffffffu, a, 2);
#pragma unroll
            for (int k = 0; k < kSums; ++k) v[k] = __shfl_sync(0xffffffffu, a, 4 * k);
            if (kFence) __threadfence();
            if (lane < (int)size) push(0, first + lane, rank, v);
            __syncwarp();
            double w[kSums];
            bool ok = poll(0, lane, size, w);
            asm volatile("bar.arrive 1, 512;" ::: "memory");
            lanes_sum(w, lane);
            if (!kLocal && groups > 1 && ok) {  // a group that misses a packet has no sums to pass on
                if (kFence) __threadfence();
                if (lane < (int)groups) {
                    // a CTA of rank r hears from rank r modulo the group's size (in its own group: itself)
                    const uint32_t f2 = group_first(lane), s2 = group_first(lane + 1) - f2;
                    for (uint32_t r = rank; r < s2; r += size) push(1, f2 + r, group, w);
                }
                __syncwarp();
                ok = poll(1, lane, groups, w);
                lanes_sum(w, lane);
            }
            if (kFence) __threadfence();
            if (!ok) S->lost = 1;
            fin(w, lane);
        } else {
            asm volatile("bar.sync 1, 512;" ::: "memory");  // the packets of hop 1 are in
            idle();
        }
        __syncthreads();
        return S->lost == 0;
    }
};

// What phase 1 does with the vectors: a step (w, xg and p advance), a fresh
// direction (w was replaced: p' = w + beta p), or a correction of p by the
// change of w (w was replaced after p had advanced).
enum Phase { kStep, kFresh, kShift };

// where a CTA's vectors live: pool offsets, and how many tiles of each fit
struct Plan {
    uint32_t cnt, t0, nface;
    uint32_t face_p, face_w, n_face_w;  // face arrays of 64: p, w
    uint32_t off_w, n_w, off_t, off_x;
};

// The solve on one CTA's tiles.  kAll: w, t and xg in shared memory; else w
// in registers for kReg passes, then in shared memory as far as it fits, and
// t and xg in global memory.
template <int kReg, bool kAll, bool kLocal, bool kHook>
__device__ __forceinline__ void resident_solve(const Args& A, Fixed& S, float* pool, Exchange<kLocal, kHook> X, const Plan P) {
    const int tid = threadIdx.x, g = tid >> 7, u = tid & 127;
    const int row = u >> 1, half = u & 1, cy = row & 7, cz = row >> 3, cx = 4 * half;
    const uint32_t lo = (uint32_t)(cx + 8 * row), cnt = P.cnt;
    // scalars of the solve, the same in every thread of every CTA
    const double stop = A.st->tol2 * A.st->bb;
    const int max_iter = A.st->max_iter, true_every = A.st->true_every;
    float alpha = 0.0f, beta = (float)A.st->beta;
    int iter = A.st->iter, next_check = A.st->next_check, true_checks = A.st->true_checks, chunks = A.st->chunks;
    int done = 0, in_chunk = 0;
    bool flush = false, lost = false;
    auto slot = [&](uint32_t t) { return (S.key[t] << 9) | lo; };
    auto core_of = [&](uint32_t t) { return pool + 64 + kTileFloats * t + lo; };
    auto codes_of = [&](uint32_t t) { return reinterpret_cast<uint16_t*>(pool + 64 + kTileFloats * t + 512)[u]; };
    auto w_of = [&](uint32_t t) {
        const uint32_t k = t - 4u * kReg;
        return kAll || k < P.n_w ? pool + P.off_w + 512u * k + lo : A.r + slot(t);
    };
    auto t_of = [&](uint32_t t) { return kAll ? pool + P.off_t + 512u * t + lo : A.t + slot(t); };
    auto x_of = [&](uint32_t t) { return kAll ? pool + P.off_x + 512u * t + lo : A.xg + slot(t); };
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // F(t, w) for every tile of the thread's group
    float4 w[kReg ? kReg : 1];
    auto each = [&](auto F) {
        if (kReg) {
#pragma unroll
            for (int i = 0; i < kReg; ++i) {
                if (4u * i + g >= cnt) break;
                F(4u * i + g, w[i]);
            }
        }
#pragma unroll 1
        for (uint32_t t = 4u * kReg + g; t < cnt; t += 4u) {
            float4 w4 = ld4(w_of(t));
            F(t, w4);
        }
    };
    // the faces that the thread's cells touch, as bits
    const uint32_t touch = (half ? 2u : 1u) | (cy == 0 ? 4u : 0u) | (cy == 7 ? 8u : 0u) | (cz == 0 ? 16u : 0u) | (cz == 7 ? 32u : 0u);
    // codes and the vectors' first values
    for (uint32_t t = g; t < cnt; t += 4u) {
        const uint32_t c4 = *reinterpret_cast<const uint32_t*>(A.cell + slot(t));
        uint32_t n4 = 0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const uint32_t c = c4 >> (8 * m);
            n4 |= (((c >> 4) & 8u) | (c & 7u)) << (4 * m);
        }
        reinterpret_cast<uint16_t*>(pool + 64 + kTileFloats * t + 512)[u] = (uint16_t)n4;
        st4(core_of(t), zero4);
        if (kAll || (t >= 4u * kReg && t - 4u * kReg < P.n_w)) st4(w_of(t), ld4cg(A.r + slot(t)));
        if (kAll) st4(x_of(t), ld4cg(A.xg + slot(t)));
    }
    auto load_w = [&]() {  // w of the register passes from r
        if (kReg) {
#pragma unroll
            for (int i = 0; i < kReg; ++i) w[i] = 4u * i + g < cnt ? ld4cg(A.r + slot(4 * i + g)) : zero4;
        }
    };
    load_w();
    // sums over the neighbours of the thread's four cells of tile t: the
    // y, z rows as 16-byte reads (in the tile, in a neighbouring tile of this
    // CTA, or in a face array), the x neighbours from the lane beside and the
    // x faces
    auto around = [&](const uint4& ta, const uint4& tb, const float* core, const float4& p) {
        const float other = __shfl_xor_sync(0xffffffffu, half ? p.x : p.w, 1);
        const uint32_t vx = half ? ta.y : ta.x;
        const uint32_t ix = (vx & kPoolMask) + (uint32_t)row * ((vx & kInner) ? 8u : 1u);
        const uint32_t iym = (ta.z & kPoolMask) + (uint32_t)cx + (uint32_t)cz * ((ta.z & kInner) ? 64u : 8u);
        const uint32_t iyp = (ta.w & kPoolMask) + (uint32_t)cx + (uint32_t)cz * ((ta.w & kInner) ? 64u : 8u);
        const uint32_t izm = (tb.x & kPoolMask) + (uint32_t)(cx + 8 * cy), izp = (tb.y & kPoolMask) + (uint32_t)(cx + 8 * cy);
        float edge;
        float4 ym, yp, zm, zp;
        if (kAll || !((ta.x | ta.y | ta.z | ta.w | tb.x | tb.y) & kFar)) {
            edge = pool[ix];
            ym = ld4(cy > 0 ? core - 8 : pool + iym);
            yp = ld4(cy < 7 ? core + 8 : pool + iyp);
            zm = ld4(cz > 0 ? core - 64 : pool + izm);
            zp = ld4(cz < 7 ? core + 64 : pool + izp);
        } else {
            edge = ((vx & kFar) ? A.far : pool)[ix];
            ym = ld4(cy > 0 ? core - 8 : ((ta.z & kFar) ? A.far : pool) + iym);
            yp = ld4(cy < 7 ? core + 8 : ((ta.w & kFar) ? A.far : pool) + iyp);
            zm = ld4(cz > 0 ? core - 64 : ((tb.x & kFar) ? A.far : pool) + izm);
            zp = ld4(cz < 7 ? core + 64 : ((tb.y & kFar) ? A.far : pool) + izp);
        }
        const float left = half ? other : edge, right = half ? edge : other;
        float4 s;
        s.x = ((left + p.y) + (ym.x + yp.x)) + (zm.x + zp.x);
        s.y = ((p.x + p.z) + (ym.y + yp.y)) + (zm.y + zp.y);
        s.z = ((p.y + p.w) + (ym.z + yp.z)) + (zm.z + zp.z);
        s.w = ((p.z + right) + (ym.w + yp.w)) + (zm.w + zp.w);
        return s;
    };
    // a face's cells 4i .. 4i+3 in slots of its tile, from the face's first slot
    auto face_at = [&](const float* base, uint32_t f, uint32_t q) {
        if (f < 2) return make_float4(__ldcg(base + 8u * q), __ldcg(base + 8u * q + 8), __ldcg(base + 8u * q + 16), __ldcg(base + 8u * q + 24));
        return ld4cg(base + (f < 4 ? (q & 7u) + 64u * (q >> 3) : q));
    };
    // phase 1 on the faces of other CTAs' tiles: 16 threads a face, four cells each
    const uint32_t fq = 4u * (tid & 15u);
    auto mail_of = [&](uint32_t e) { return A.mail + (size_t)(X.tag & 1u) * A.mail_half + S.face[e].in + fq; };
    constexpr uint32_t kAllSix = 0xEEEEu;  // four fluid cells with six non-solid neighbours
    auto face_move = [&](uint32_t e, Phase ph, float4 v) {
        const uint32_t at = S.tab[S.face[e].t_f >> 3][S.face[e].t_f & 7u];
        float* fp = (!kAll && (at & kFar) ? A.far : pool) + (at & kPoolMask) + fq;
        float* fw = kAll || e < P.n_face_w ? pool + P.face_w + 64u * e + fq
                                   : A.far + 768u * (P.t0 + (S.face[e].t_f >> 3)) + 128u * (S.face[e].t_f & 7u) + 64u + fq;
        const float4 p = ld4(fp);
        if (ph == kShift) {
            const float4 o = ld4(fw);
            st4(fp, make_float4(p.x + (v.x - o.x), p.y + (v.y - o.y), p.z + (v.z - o.z), p.w + (v.w - o.w)));
        } else {
            if (ph == kStep) v = axpy4(v, ld4(fw), -alpha);
            st4(fp, axpy4(p, v, beta));
        }
        st4(fw, v);
    };
    __syncthreads();

    Phase ph = kFresh;
    unsigned long long m[4] = {0, 0, 0, 0}, mn[4];  // a face's mail, the next face's
    auto load_mail = [&](uint32_t e, unsigned long long (&v)[4]) {
        const unsigned long long* q = mail_of(e);
        ld_relaxed_u64x2(q, v[0], v[1]);
        ld_relaxed_u64x2(q + 2, v[2], v[3]);
    };
    auto fetch_mail = [&](uint32_t e, unsigned long long (&v)[4]) {  // until the warp's are there
        uint32_t spin = 0;
        while (!__all_sync(0xffffffffu, (uint32_t)(v[0] >> 32) == X.tag && (uint32_t)(v[1] >> 32) == X.tag &&
                                            (uint32_t)(v[2] >> 32) == X.tag && (uint32_t)(v[3] >> 32) == X.tag &&
                                            !X.in_vain(2))) {
            if (++spin >= X.polls()) { S.lost = 1; break; }
            load_mail(e, v);
        }
    };
    while (!done && !lost) {
        // ---- phase 1: the vectors advance by the last step's alpha and beta
        if (ph == kStep) {
            // loads run a tile and a face ahead of their use; two tiles where t
            // and xg come from L2 (an iteration on 6,498 tiles 20.2 -> 18.8 us;
            // w past the registers is then read as it is used)
            float4 tn, xn, wn, tm, xm;
            auto fetch = [&](uint32_t t) {
                if (t < cnt) {
                    tm = ld4(t_of(t));
                    xm = ld4(x_of(t));
                }
            };
            fetch(g);
            tn = tm; xn = xm;
            if (kAll) { if (g < cnt) wn = ld4(w_of(g)); }
            else fetch(g + 4u);
#pragma unroll 1
            // two faces a warp; the first warp has had the exchange to do
            for (uint32_t e0 = tid < 32 ? P.nface : 2u * ((tid >> 5) - 1u); e0 < P.nface; e0 += kThreads / 16 - 2) {
                const uint32_t e = e0 + ((tid >> 4) & 1u), en = e + kThreads / 16 - 2;
                load_mail(min(en, P.nface - 1u), mn);
                fetch_mail(min(e, P.nface - 1u), m);
                if (e < P.nface)
                    face_move(e, ph, make_float4(__uint_as_float((uint32_t)m[0]), __uint_as_float((uint32_t)m[1]),
                                                 __uint_as_float((uint32_t)m[2]), __uint_as_float((uint32_t)m[3])));
#pragma unroll
                for (int k = 0; k < 4; ++k) m[k] = mn[k];
            }
            auto advance = [&](uint32_t t, float4& w4) {
                const float4 t4 = tn, x4 = xn;
                if (kAll) {
                    fetch(t + 4u);
                    tn = tm; xn = xm;
                    if (t + 4u < cnt) wn = ld4(w_of(t + 4u));
                } else {
                    tn = tm; xn = xm;
                    fetch(t + 8u);
                }
                float* core = core_of(t);
                const float4 p = ld4(core);
                w4 = axpy4(t4, w4, -alpha);
                st4(x_of(t), axpy4(p, x4, alpha));
                st4(core, axpy4(p, w4, beta));
            };
            if (kReg) {
#pragma unroll
                for (int i = 0; i < kReg; ++i) {
                    if (4u * i + g >= cnt) break;
                    advance(4u * i + g, w[i]);
                }
            }
#pragma unroll 1
            for (uint32_t t = 4u * kReg + g; t < cnt; t += 4u) {
                float4 w4 = kAll ? wn : ld4(w_of(t));
                advance(t, w4);
                st4(w_of(t), w4);
            }
        } else {
            for (uint32_t e = tid >> 4; e < P.nface; e += kThreads / 16)
                face_move(e, ph, face_at(A.r + S.face[e].src, S.face[e].t_f & 7u, fq));
            each([&](uint32_t t, float4& w4) {
                if (flush) {  // after a true-residual check: xg into x on the fluid cells
                    const uint32_t s = slot(t), n4 = codes_of(t);
                    float* xp = x_of(t);
                    const float4 gq = ld4(xp);
                    const float* gv = &gq.x;
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if ((n4 >> (4 * m)) & 8u) A.x[s + m] += (double)gv[m];
                    st4(xp, zero4);
                }
                if (ph == kFresh) st4(core_of(t), axpy4(ld4(core_of(t)), w4, beta));
            });
            flush = false;
        }
        __syncthreads();
        if (S.lost) { lost = true; break; }
        // ---- phase 2: q = A p, t = D^-1 q and the five sums
        double sums[kSums] = {};
        double qq6 = 0.0, ww6 = 0.0;
        unsigned long long* const mail_out = A.mail + (size_t)((X.tag + 1u) & 1u) * A.mail_half;
        each([&](uint32_t t, float4& w4) {
            const float* core = core_of(t);
            const uint32_t n4 = codes_of(t);
            const uint4 ta = *reinterpret_cast<const uint4*>(&S.tab[t][0]);
            const uint4 tb = *reinterpret_cast<const uint4*>(&S.tab[t][4]);
            const float4 p = ld4(core);
            const float4 s = around(ta, tb, core, p);
            const float *pv = &p.x, *sv = &s.x, *wv = &w4.x;
            float4 t4;
            float* tv = &t4.x;
            if (__all_sync(0xffffffffu, n4 == kAllSix)) {
                // 6 for every diagonal: q.t, r.z and r.r from the sums of q^2 and w^2
                const float sixth = S.inv[6];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float q = fmaf(6.0f, pv[m], -sv[m]);
                    tv[m] = q * sixth;
                    const double qd = (double)q, wd = (double)wv[m];
                    sums[0] += (double)pv[m] * qd;
                    sums[1] += wd * qd;
                    qq6 += qd * qd;
                    ww6 += wd * wd;
                }
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t c = n4 >> (4 * m);
                    const float d = small_float(c & 7u);
                    const float q = (c & 8u) ? fmaf(d, pv[m], -sv[m]) : 0.0f;
                    tv[m] = q * S.inv[c & 7u];
                    const double qd = (double)q, wd = (double)wv[m], rd = (double)(d * wv[m]);
                    sums[0] += (double)pv[m] * qd;
                    sums[1] += wd * qd;
                    sums[2] += qd * (double)tv[m];
                    sums[3] += rd * wd;
                    sums[4] += rd * rd;
                }
            }
            st4(t_of(t), t4);
            // t of the cells on a face that another CTA's tile sees, into its mailbox
            const uint32_t need = tb.z & touch;
            if (need) {
                const uint32_t tag = X.tag + 1u;
                const unsigned long long m0 = tagged(tag, __float_as_uint(t4.x)), m1 = tagged(tag, __float_as_uint(t4.y)),
                                         m2 = tagged(tag, __float_as_uint(t4.z)), m3 = tagged(tag, __float_as_uint(t4.w));
                unsigned long long* q = mail_out + tb.w;
                if (need & 3u) st_relaxed_u64(q + 64 * half + row, half ? m3 : m0);
                if (need & 12u) {
                    st_relaxed_u64x2(q + (cy ? 192 : 128) + cx + 8 * cz, m0, m1);
                    st_relaxed_u64x2(q + (cy ? 192 : 128) + cx + 8 * cz + 2, m2, m3);
                }
                if (need & 48u) {
                    st_relaxed_u64x2(q + (cz ? 320 : 256) + cx + 8 * cy, m0, m1);
                    st_relaxed_u64x2(q + (cz ? 320 : 256) + cx + 8 * cy + 2, m2, m3);
                }
            }
        });
        sums[2] += (double)S.inv[6] * qq6;
        sums[3] += 6.0 * ww6;
        sums[4] += 36.0 * ww6;
        if (!X.template sum<false>(sums, [&]() {
                if (P.nface) load_mail(min(((uint32_t)tid >> 4) - 2u, P.nface - 1u), m);
            }, [&](const double (&w)[kSums], int lane) {
                // ---- scalars, once for the CTA (every thread dividing for itself
                // took 3.81 instead of 3.26 us an iteration on 48 tiles); a verdict of
                // 1: the residual before this step claims convergence.  Not before the
                // first one: what a start may claim, nat_launch_pcgw_init has settled,
                // and r.r = b.b <= tol^2 b.b also where both are infinite
                const double a = w[3] / w[0], over = 1.0 / w[3];
                const double b = fmax(fma(a, fma(a, w[2], -2.0 * w[1]), w[3]), 0.0) * over;
                if (lane == 0) {
                    S.pq = w[0];
                    S.rr = w[4];
                    S.rz = w[3];
                    S.alpha = (float)a;
                    S.beta = (float)b;
                    S.verdict = iter > 0 && w[4] <= stop ? 1u : (w[0] > 0.0 ? 0u : 2u);
                }
            })) { lost = true; break; }
        const bool pending = S.verdict == 1u;
        if (!pending) {
            if (S.verdict == 2u) { done = 3; break; }  // breakdown
            alpha = S.alpha;
            beta = S.beta;
            iter += 1;
            in_chunk += 1;
            ph = kStep;
        }
        const bool full = pending || in_chunk >= A.chunk;
        if (full) {
            ++chunks;
            in_chunk = 0;
        }
        if (!(pending || iter >= max_iter || chunks >= A.limit || (full && true_every > 0 && iter >= next_check))) continue;
        // ---- true residual b - A (x + xg) in FP64: replaces w, decides convergence
        each([&](uint32_t t, float4& w4) {
            float* xp = x_of(t);
            const float4 o = ld4(xp);
            const float4 v = pending ? o : axpy4(ld4(core_of(t)), o, alpha);
            st4(xp, v);
            st4(A.xg + slot(t), v);
            st4(A.r + slot(t), w4);  // the w that the residual replaces
        });
        double ts[kSums] = {};
        if (!X.template sum<true>(ts, [] {}, [](const double (&)[kSums], int) {})) { lost = true; break; }  // every CTA's xg is in place
#pragma unroll
        for (int k = 0; k < kSums; ++k) ts[k] = 0.0;
#pragma unroll 1
        for (uint32_t t = g; t < cnt; t += 4u) {
            const NatDims& D = A.D;
            const uint32_t key = S.key[t], tc = S.coord[t], s = slot(t), n4 = codes_of(t);
            const int bx = (int)(tc & 1023u), by = (int)((tc >> 10) & 1023u), bz = (int)(tc >> 20);
            // solution x + xg of one slot, of four consecutive ones; both are
            // zero off the fluid on every tile around the fluid
            auto sol = [&](uint32_t s) { return __ldcg(A.x + s) + (double)__ldcg(A.xg + s); };
            auto sol4 = [&](uint32_t s, double (&o)[4]) {
                const double2 a = __ldcg(reinterpret_cast<const double2*>(A.x + s));
                const double2 b = __ldcg(reinterpret_cast<const double2*>(A.x + s) + 1);
                const float4 q = ld4cg(A.xg + s);
                o[0] = a.x + (double)q.x; o[1] = a.y + (double)q.y; o[2] = b.x + (double)q.z; o[3] = b.y + (double)q.w;
            };
            double c[4], ym[4] = {}, yp[4] = {}, zm[4] = {}, zp[4] = {}, edge = 0.0;
            sol4(s, c);
            if (half == 0 && bx > 0) edge = sol(((key - 1u) << 9) + 7u + 8u * row);
            if (half == 1 && bx < D.tx - 1) edge = sol(((key + 1u) << 9) + 8u * row);
            if (cy > 0) sol4(s - 8, ym);
            else if (by > 0) sol4(((key - (uint32_t)D.tx) << 9) + 56u + cx + 64u * cz, ym);
            if (cy < 7) sol4(s + 8, yp);
            else if (by < D.ty - 1) sol4(((key + (uint32_t)D.tx) << 9) + cx + 64u * cz, yp);
            if (cz > 0) sol4(s - 64, zm);
            else if (bz > 0) sol4(((key - (uint32_t)(D.tx * D.ty)) << 9) + 448u + cx + 8u * cy, zm);
            if (cz < 7) sol4(s + 64, zp);
            else if (bz < D.tz - 1) sol4(((key + (uint32_t)(D.tx * D.ty)) << 9) + cx + 8u * cy, zp);
            const double other = __shfl_xor_sync(0xffffffffu, half ? c[0] : c[3], 1);
            const double left = half ? other : edge, right = half ? edge : other;
            const double xl[4] = {left, c[0], c[1], c[2]}, xr[4] = {c[1], c[2], c[3], right};
            const float4 b4 = ld4(A.b + s), w0 = ld4cg(A.r + s);
            float4 w4 = w0;
            const float* bq = &b4.x;
            float* wv = &w4.x;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const uint32_t n = n4 >> (4 * m);
                if (!(n & 8u)) continue;
                const double d = (double)(n & 7u);
                const double res = (double)bq[m] - (d * c[m] - (((xl[m] + xr[m]) + (ym[m] + yp[m])) + (zm[m] + zp[m])));
                ts[0] += res * res;
                const float ws = (n & 7u) ? (float)(res / d) : 0.0f;
                wv[m] = ws;
                ts[1] += d * (double)ws * (double)ws;
            }
            st4(A.r + s, w4);
            if (kAll || (t >= 4u * kReg && t - 4u * kReg < P.n_w)) st4(w_of(t), w4);
            if (pending) {
                float* core = core_of(t);
                const float4 p = ld4(core);
                st4(core, make_float4(p.x + (w4.x - w0.x), p.y + (w4.y - w0.y), p.z + (w4.z - w0.z), p.w + (w4.w - w0.w)));
            }
        }
        load_w();
        if (!X.template sum<true>(ts, [] {}, [&](const double (&w)[kSums], int lane) {
                if (lane == 0) {
                    S.rr = S.rr_true = w[0];
                    S.beta = (float)(w[1] / S.rz);
                    S.rz = w[1];
                }
            })) { lost = true; break; }
        true_checks += 1;
        next_check = iter + true_every;
        flush = true;
        ph = pending ? kShift : kFresh;
        if (!pending) beta = S.beta;
        if (S.rr_true <= stop) done = 1;
        else if (iter >= max_iter || chunks >= A.limit) done = 2;
    }
    // ---- what the solve leaves: x + xg, w (in place after a check)
    if (done == 3)
        each([&](uint32_t t, float4& w4) {
            st4(A.xg + slot(t), ld4(x_of(t)));
            st4(A.r + slot(t), w4);
        });
    if (lost && tid == 0) atomicOr(A.err, DEVERR_GRID_TIMEOUT);
    if (blockIdx.x == 0 && tid == 0) {
        PcgState* st = A.st;
        st->rz = S.rz;
        st->pq = S.pq;
        st->rr = S.rr;
        st->rr_true = S.rr_true;
        st->alpha = alpha;
        st->beta = beta;
        st->iter = iter;
        st->true_checks = true_checks;
        st->next_check = next_check;
        st->done = lost ? 5 : done;
        st->halt = 1;
        *A.epoch = X.tag + 4u;  // past any tag of a solve that gave up
    }
}

// kLocal: one cluster of at most kClusterMax CTAs, four tiles each
template <bool kLocal, bool kHook>
__global__ void __launch_bounds__(kThreads, 1) pcg_resident_kernel(const __grid_constant__ Args A, const uint32_t* __restrict__ d_ntiles) {
    extern __shared__ __align__(16) unsigned char smem[];
    Fixed& S = *reinterpret_cast<Fixed*>(smem);
    float* pool = reinterpret_cast<float*>(smem + sizeof(Fixed));
    const uint32_t nt = *d_ntiles;
    if (A.st->done || nt > (uint32_t)kMaxTiles * A.ctas) return;  // solved already, or more than the chip holds
    Exchange<kLocal, kHook> X;
    const uint32_t ctas = min(A.ctas, (nt + kGroups - 1u) / kGroups);
    if (blockIdx.x >= ctas) return;
    X.init(ctas);
    X.slots = A.slots;
    X.ctas = A.ctas;
    X.S = &S;
    X.tag = *A.epoch;
    if (kHook) {
        X.hook_which = blockIdx.x == ctas - 1u ? A.hook.which : 3u;
        X.hook_tag = X.tag + A.hook.exchange;
        X.hook_polls = A.hook.polls;
    }
    Plan P;
    P.t0 = (uint32_t)((uint64_t)nt * blockIdx.x / X.n);
    P.cnt = (uint32_t)((uint64_t)nt * (blockIdx.x + 1) / X.n) - P.t0;
    const int tid = threadIdx.x;
    const uint32_t cnt = P.cnt;
    // ---- the CTA's tiles and their faces
    for (uint32_t t = tid; t < cnt; t += kThreads) {
        S.key[t] = A.tiles[P.t0 + t];
        S.coord[t] = A.tcoord[P.t0 + t];
    }
    for (uint32_t t = tid; t < cnt; t += kThreads) {
        S.tab[t][6] = 0u;
        S.tab[t][7] = 64u * 6u * (P.t0 + t);
    }
    if (kLocal) {
        // the packets lie at the pool's end, which four tiles leave free; no
        // exchange carries the tag that they start with
        unsigned long long* w = reinterpret_cast<unsigned long long*>(pool + kPoolFloats / 4 * 4) - kLocalWords;
        for (uint32_t k = tid; k < kLocalWords; k += kThreads) w[k] = tagged(X.tag, 0u);
        X.local = (uint32_t)__cvta_generic_to_shared(w);
    }
    if (tid < 64) pool[tid] = 0.0f;  // the face of a wall or of a tile without fluid
    if (tid < 8) S.inv[tid] = tid ? __frcp_rn((float)tid) : 0.0f;
    if (tid == 0) {
        S.nface = 0;
        S.lost = 0;
        S.rr = A.st->rr;
        S.rr_true = A.st->rr_true;
        S.pq = 0.0;
        S.rz = A.st->rz;
    }
    __syncthreads();
    const uint32_t base = 64u + kTileFloats * cnt;
    const uint32_t room = ((uint32_t)kPoolFloats - base) / 64u;  // face arrays the pool holds
    const NatDims& D = A.D;
    for (uint32_t e = tid; e < 6u * cnt; e += kThreads) {
        const uint32_t t = e / 6u, f = e % 6u, a = f >> 1;
        const int c = (int)((S.coord[t] >> (10u * a)) & 1023u);
        const int T = a == 0 ? D.tx : (a == 1 ? D.ty : D.tz), step = a == 0 ? 1 : (a == 1 ? D.tx : D.tx * D.ty);
        uint32_t v = 0u;  // the zero face
        if ((f & 1u) ? c < T - 1 : c > 0) {
            const uint32_t want = S.key[t] + (uint32_t)((f & 1u) ? step : -step);
            uint32_t lo_t = 0, hi_t = nt;  // keys ascend
            if ((f & 1u) ? want <= S.key[cnt - 1] : want >= S.key[0]) {  // in this CTA's run, if anywhere
                hi_t = cnt;
                while (lo_t < hi_t) {
                    const uint32_t mid = (lo_t + hi_t) >> 1;
                    if (S.key[mid] < want) lo_t = mid + 1; else hi_t = mid;
                }
                // the neighbour's first face cell: its x, y or z = 7 for the low side
                if (S.key[lo_t] == want) v = kInner | (64u + kTileFloats * lo_t + ((f & 1u) ? 0u : (a == 0 ? 7u : (a == 1 ? 56u : 448u))));
            } else {
                while (lo_t < hi_t) {
                    const uint32_t mid = (lo_t + hi_t) >> 1;
                    if (A.tiles[mid] < want) lo_t = mid + 1; else hi_t = mid;
                }
                if (lo_t < nt && A.tiles[lo_t] == want) {
                    const uint32_t k = atomicAdd(&S.nface, 1u);
                    v = k < room ? base + 64u * k : kFar | (768u * (P.t0 + t) + 128u * f);
                    S.face[k] = Face{(want << 9) + ((f & 1u) ? 0u : (a == 0 ? 7u : (a == 1 ? 56u : 448u))),
                                     64u * (6u * lo_t + (f ^ 1u)), 0u, (t << 3) | f};
                    atomicOr(&S.tab[t][6], 1u << f);
                    float* z = (k < room ? pool : A.far) + (v & kPoolMask);
                    for (int m = 0; m < 64; m += 4) st4(z + m, make_float4(0.0f, 0.0f, 0.0f, 0.0f));
                }
            }
        }
        S.tab[t][f] = v;
    }
    __syncthreads();
    P.nface = S.nface;
    // Everything on the chip where the largest share of tiles has room for it with
    // three faces a tile towards other CTAs (21 tiles) and this CTA's own faces
    // have; else w in what the registers and the pool hold, then the faces' w.
    // The second condition is the CTA's own: both forms take the same exchanges,
    // publish the same face cells and leave the same xg and r for a check, so CTAs
    // of either form work together (21 tiles each in rows of 22: 50 of 148 keep
    // everything on the chip).
    const uint32_t most = (nt + X.n - 1u) / X.n;
    const uint32_t left = (uint32_t)kPoolFloats - base;
    if (kLocal) cluster_sync();  // every CTA's packets are ready
    if (kLocal || (64u + most * (uint32_t)(kTileFloats + 3 * 512 + 6 * 128 / 2) <= (uint32_t)kPoolFloats && P.nface * 128u + cnt * 1536u <= left)) {
        P.face_w = base + 64u * P.nface;
        P.off_w = P.face_w + 64u * P.nface;
        P.off_t = P.off_w + 512u * cnt;
        P.off_x = P.off_t + 512u * cnt;
        P.n_w = cnt;
        P.n_face_w = P.nface;
        resident_solve<0, true, kLocal, kHook>(A, S, pool, X, P);
    } else if (!kLocal) {
        const uint32_t faces = min(P.nface, room);
        P.off_w = base + 64u * faces;
        P.n_w = min(cnt - min(cnt, 4u * kRegPasses), (left - 64u * faces) / 512u);
        P.face_w = P.off_w + 512u * P.n_w;
        P.n_face_w = min(P.nface, (left - 64u * faces - 512u * P.n_w) / 64u);
        P.off_t = P.off_x = 0;
        resident_solve<kRegPasses, false, kLocal, kHook>(A, S, pool, X, P);
    }
    if (kLocal) cluster_sync();  // no CTA leaves while another may still write to it
}

static_assert(64 + kGroups * (kTileFloats + 3 * 512 + 6 * 128) + 2 * kLocalWords <= kPoolFloats, "four tiles and the packets");

// CTAs of the cluster that holds `ctas` of them: a power of two
uint32_t cluster_of(uint32_t ctas) {
    uint32_t n = 1;
    while (n < ctas) n *= 2;
    return n;
}
cudaLaunchConfig_t resident_config(uint32_t grid, cudaLaunchAttribute* attr, bool local, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemMax;
    cfg.stream = s;
    if (local) {
        attr->id = cudaLaunchAttributeClusterDimension;
        attr->val.clusterDim = {grid, 1, 1};
    } else {
        attr->id = cudaLaunchAttributeCooperative;
        attr->val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

// whether a box whose solve takes `ctas` CTAs runs as one cluster
int nat_pcg_cluster(uint32_t ctas, bool* fits) {
    *fits = false;
    if (ctas > kClusterMax) return FLIP_OK;
    const auto kernel = pcg_resident_kernel<true, false>;
    FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = resident_config(cluster_of(ctas), attr, true, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();  // no such cluster on this device
        return FLIP_OK;
    }
    *fits = clusters > 0;
    return FLIP_OK;
}

int nat_launch_pcg_resident(const uint32_t* tiles, const uint32_t* d_ntiles, const NatDims& D, PcgBuffers& B, int chunk,
                            int limit, uint32_t* err, cudaStream_t s) {
    const bool hook = B.hook.exchange != 0;
    const auto kernel = B.cluster ? (hook ? pcg_resident_kernel<true, true> : pcg_resident_kernel<true, false>)
                                  : (hook ? pcg_resident_kernel<false, true> : pcg_resident_kernel<false, false>);
    if (B.cluster && hook) FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = resident_config(B.cluster ? cluster_of(B.ctas) : B.ctas, attr, B.cluster, s);
    const Args A{tiles, B.tcoord, D, B.x, B.xg, B.r, B.q, B.far, B.mail, 64u * 6u * B.mail_tiles, B.b, B.cell, B.st, B.slots,
                 B.ctas, B.epoch, err, chunk, limit, B.hook};
    FLIP_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, A, d_ntiles));
    return FLIP_OK;
}

}  // namespace flip
