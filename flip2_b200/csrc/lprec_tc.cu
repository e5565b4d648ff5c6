// lprec_tc.cu -- tensor-core forward of the learned preconditioner's
// 16 -> 16 channel layers (dilated 3^3 convolutions, BF16 in, FP32
// accumulation in tensor memory, ReLU, BF16 out) as an implicit GEMM on the
// sm_100a UMMA unit (tcgen05.mma, kind::f16).
//
// One CTA works on one 8^3 tile of the active list at a time:
//   1. stage the tile's input box (8 + 2 dil)^3 voxels x 16 channels in
//      shared memory as two 8-channel planes, 16 B per voxel and plane, in
//      x-fastest order; voxels outside the box or in inactive tiles read 0;
//   2. one thread issues, for each z-slice of the tile and each of the 27
//      taps, one M=64 x N=16 x K=16 MMA: A = the 64 voxels (8 x, 8 y) of the
//      slice shifted by the tap, read straight from the box (rows 16 B apart,
//      8-row groups one box row apart, the two channel planes one plane
//      apart: the K-major no-swizzle canonical layout), B = the tap's 16 x 16
//      weights; the 27 products accumulate into one TMEM accumulator per
//      z-slice (8 slices x 16 columns);
//   3. the MMAs commit to an mbarrier; every warp waits on it (bounded), reads
//      its accumulators with tcgen05.ld, applies ReLU and stores BF16.
// An M=64 accumulator keeps row m in TMEM lane (m % 16) + 32 (m / 16) and
// column n at column n.  Waits are bounded: on a timeout the kernel sets an
// error flag, waits (bounded) for its MMAs, frees its TMEM and returns.
#include <cuda_bf16.h>
#include "common.cuh"
#include "lprec.cuh"

namespace flip {

namespace {
constexpr int kTcCols = 128;      // 8 z-slices x 16 FP32 columns
constexpr uint32_t kTcSpinLimit = 1u << 24;
constexpr uint32_t kInstrDesc = (1u << 4)           // D: FP32
                                | (1u << 7)         // A: BF16
                                | (1u << 10)        // B: BF16
                                | ((16u >> 3) << 17)  // N = 16
                                | ((64u >> 4) << 24);  // M = 64

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major, no swizzle: rows 16 B apart, 8-row groups sbo bytes apart, the two
// 16-byte K halves lbo bytes apart; descriptor version 1 (sm100)
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ void mma_f16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait; false on timeout
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (uint32_t it = 0; it < kTcSpinLimit; ++it)
        if (mbar_try_wait(mbar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tile_origin_tc(uint32_t key, const NatDims& D, int& ox, int& oy, int& oz) {
    ox = 8 * (int)(key % D.tx);
    oy = 8 * (int)((key / D.tx) % D.ty);
    oz = 8 * (int)(key / (D.tx * D.ty));
}
}  // namespace

// 16 bytes from global to shared memory, zeros where !ok (src is not read then)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// first slot of neighbour nb (x, y, z offsets nb % 3 - 1, nb / 3 % 3 - 1,
// nb / 9 - 1) of tile key, kNoTile outside the grid or where no activations are
constexpr uint32_t kNoTile = 0xFFFFFFFFu;
__device__ __forceinline__ uint32_t tile_neighbour(const LpGrid& G, uint32_t key, int nb) {
    const int tx = (int)(key % G.D.tx) + nb % 3 - 1, ty = (int)((key / G.D.tx) % G.D.ty) + (nb / 3) % 3 - 1,
              tz = (int)(key / (G.D.tx * G.D.ty)) + nb / 9 - 1;
    if ((unsigned)tx >= (unsigned)G.D.tx || (unsigned)ty >= (unsigned)G.D.ty || (unsigned)tz >= (unsigned)G.D.tz) return kNoTile;
    const uint32_t t = (uint32_t)(tx + G.D.tx * (ty + G.D.ty * tz));
    return G.tile_active[t] ? t << 9 : kNoTile;
}
// cell (px, py, pz) relative to a tile (-8 .. 15 an axis): the neighbour it
// lies in and its slot there
__device__ __forceinline__ int rel_neighbour(int px, int py, int pz) {
    return ((px >> 3) + 1) + 3 * ((py >> 3) + 1) + 9 * ((pz >> 3) + 1);
}
__device__ __forceinline__ uint32_t rel_local(int px, int py, int pz) {
    return (uint32_t)((px & 7) | ((py & 7) << 3) | ((pz & 7) << 6));
}
__device__ __forceinline__ uint4 bf16x8(const float4& a, const float4& b) {
    uint4 o;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
    h[0] = __floats2bfloat162_rn(a.x, a.y);
    h[1] = __floats2bfloat162_rn(a.z, a.w);
    h[2] = __floats2bfloat162_rn(b.x, b.y);
    h[3] = __floats2bfloat162_rn(b.z, b.w);
    return o;
}

// CTAs that share a tile's z-slices, where there are more CTAs than tiles.  A
// tile by itself takes a CTA some 20 us, most of it MMAs one after the other: a
// training step on one tile went from 419 to 332 us, on 64 from 462 to 403.  Whole
// tiles have a form of their own: with the slices' bounds in registers a step on
// 4,096 tiles took 2.5% longer.
__device__ __forceinline__ uint32_t tile_parts(uint32_t n) { return 4u * n <= gridDim.x ? 4u : (2u * n <= gridDim.x ? 2u : 1u); }

// shared-memory footprint of one CTA for dilation DIL.  The planes lie 64
// bytes more than their size apart, so that a voxel's two stores fall on
// different banks.  The dilation-4 box leaves room for one CTA per SM, which
// then has twice the threads.
template <int DIL>
struct TcSmem {
    static constexpr int B = 8 + 2 * DIL;                 // box edge
    static constexpr int kPlane = B * B * B * 16 + 64;    // bytes of one 8-channel plane
    static constexpr int kBox = 2 * kPlane;
    static constexpr int kW = 27 * 512;                   // 27 taps x (16 co x 16 ci) BF16
    static constexpr int kBytes = kBox + kW + 64;
    static constexpr int kThreads = DIL == 4 ? 512 : 256;
};

// GRAD = false: out = relu(conv(in)).  GRAD = true, the layer's input
// gradient: gin[v][ci] = relu'(ain[v][ci]) sum_tap sum_co W[tap][ci][co]
// in[v - dil off(tap)][co] with in = the output gradient (FP32, rounded to BF16
// in the box) -- the same GEMM with the taps' offsets mirrored and each tap's
// weights transposed.
// Bound by the latency of a tile's steps (stage, MMAs, read back): the box's
// loads are therefore all in flight at once (cp.async; eight float4 a thread
// for the FP32 box), and a table of the tile's 27 neighbours, made while the
// previous tile's MMAs run, takes the lookups out of them.  128^3, 4,096 tiles,
// dilation 2 and 4: forward 118 and 462 -> 100 and 243 us; the input gradient
// 131 and 305 us, against 583 us with each voxel's 27 neighbours gathered into a
// K-major A, 128 voxels at a time.
// mid_tc_tiles: the tiles (SPLIT: parts of tiles) of a CTA.
template <int DIL, bool GRAD, bool SPLIT>
__device__ __forceinline__ void mid_tc_tiles(const LpGrid& G, const void* __restrict__ in_, const __nv_bfloat16* __restrict__ ain,
                                             void* __restrict__ out_, int* __restrict__ err, uint32_t n, uint32_t tmem,
                                             unsigned char* smem, int& s_abort, uint32_t (&s_nb)[2][27]) {
    using S = TcSmem<DIL>;
    constexpr int B = S::B, kThr = S::kThreads;
    unsigned char* box = smem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t parts = SPLIT ? tile_parts(n) : 1u, all = n * parts;
    const int nz = 8 / (int)parts;
    const uint32_t box_s = smem_u32(box), w_s = box_s + S::kBox, mbar_s = w_s + S::kW;
    uint32_t phase = 0;
    bool pending_mma = false;
    int cur = 0;
    for (uint32_t t = blockIdx.x; t < all; t += gridDim.x, cur ^= 1) {
        const uint32_t key = G.act_tiles[t / parts];
        const int z0 = (int)(t % parts) * nz, z1 = z0 + nz;  // this CTA's slices
        int ox, oy, oz;
        tile_origin_tc(key, G.D, ox, oy, oz);
        // 1. input box (of the slices: z0 .. z1 + 2 DIL), two 16-byte chunks per voxel
        auto source = [&](int e, uint32_t& sl) {  // its voxel's slot; whether there is one
            const int v = e >> 1;
            const int px = v % B - DIL, py = (v / B) % B - DIL, pz = v / (B * B) - DIL;
            const uint32_t base = s_nb[cur][rel_neighbour(px, py, pz)];
            const bool ok = base != kNoTile && ox + px < G.D.nx && oy + py < G.D.ny && oz + pz < G.D.nz;
            sl = ok ? base | rel_local(px, py, pz) : 0u;
            return ok;
        };
        const int first = 2 * B * B * z0, last = 2 * B * B * (z1 + 2 * DIL);
        if (GRAD) {
            const float* in = static_cast<const float*>(in_);
            for (int e0 = first + tid; e0 < last; e0 += 4 * kThr) {
                float4 g[4][2];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int e = e0 + m * kThr;
                    uint32_t sl;
                    g[m][0] = g[m][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (e < last && source(e, sl)) {
                        const float4* p = reinterpret_cast<const float4*>(in + (size_t)sl * 16 + (e & 1) * 8);
                        g[m][0] = p[0];
                        g[m][1] = p[1];
                    }
                }
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int e = e0 + m * kThr;
                    if (e < last)
                        *reinterpret_cast<uint4*>(box + (e & 1) * S::kPlane + (e >> 1) * 16) = bf16x8(g[m][0], g[m][1]);
                }
            }
        } else {
            const __nv_bfloat16* in = static_cast<const __nv_bfloat16*>(in_);
            for (int e = first + tid; e < last; e += kThr) {
                uint32_t sl;
                const bool ok = source(e, sl);
                cp_async16(box_s + (uint32_t)((e & 1) * S::kPlane + (e >> 1) * 16), in + (size_t)sl * 16 + (e & 1) * 8, ok);
            }
            cp_async_commit();
            cp_async_wait<0>();
        }
        // make the writes visible to the tensor core's async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        // 2. 8 slices x 27 taps of M=64 N=16 K=16
        if (tid == 0) {
            for (int z = z0; z < z1; ++z) {
                if (DIL == 4) {
                    // a descriptor holds its address in units of 16 B, and the
                    // taps' offsets are constants: an addition each
                    const uint64_t bd = umma_desc(w_s, 256, 128);
                    const uint64_t ad = umma_desc(box_s + (uint32_t)(z * B * B * 16), S::kPlane, B * 16);
#pragma unroll
                    for (int tap = 0; tap < 27; ++tap) {
                        const int at = GRAD ? 26 - tap : tap;  // mirrored
                        const int aoff = ((DIL * (at / 9)) * B + DIL * ((at / 3) % 3)) * B + DIL * (at % 3);
                        mma_f16(tmem + (uint32_t)(z * 16), ad + (uint64_t)aoff, bd + (uint64_t)(32 * tap), kInstrDesc,
                                tap > 0 ? 1u : 0u);
                    }
                } else {
                    // three CTAs share an SM's tensor core: issued as fast as
                    // above, each one's chains into one accumulator hold up the
                    // others' (202 us at dilation 2, against 100)
                    for (int tap = 0; tap < 27; ++tap) {
                        constexpr int kStep = GRAD ? -DIL : DIL;
                        const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
                        const int bz = z + DIL + kStep * dz, by0 = DIL + kStep * dy, bx0 = DIL + kStep * dx;
                        const uint32_t aoff = (uint32_t)(((bz * B + by0) * B + bx0) * 16);
                        const uint64_t ad = umma_desc(box_s + aoff, S::kPlane, B * 16);
                        const uint64_t bd = umma_desc(w_s + tap * 512, 256, 128);
                        mma_f16(tmem + (uint32_t)(z * 16), ad, bd, kInstrDesc, tap > 0 ? 1u : 0u);
                    }
                }
            }
            mma_commit(mbar_s);
        }
        pending_mma = true;
        if (warp == 1 && lane < 27 && t + gridDim.x < all)
            s_nb[cur ^ 1][lane] = tile_neighbour(G, G.act_tiles[(t + gridDim.x) / parts], lane);
        // 3. epilogue: warp w reads sub-partition w % 4 of every (warps / 4)-th slice
        const bool ok = mbar_wait(mbar_s, phase);
        if (!ok) {
            if (lane == 0) atomicExch(&s_abort, 1);
        }
        __syncthreads();
        if (s_abort) break;
        pending_mma = false;
        phase ^= 1u;
        tc_fence_after();
        const int q = warp & 3;
        for (int zz = z0 + (warp >> 2); zz < z1; zz += kThr / 128) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(zz * 16), v);
            if (lane < 16) {
                const int m = lane + 16 * q;  // row of the slice: x = m % 8, y = m / 8
                const uint32_t sl = (key << 9) | (uint32_t)((m & 7) | ((m >> 3) << 3) | (zz << 6));
                if (GRAD) {
                    const uint4* ap = reinterpret_cast<const uint4*>(ain + (size_t)sl * 16);
                    const uint4 q0 = ap[0], q1 = ap[1];
                    const __nv_bfloat16* a0 = reinterpret_cast<const __nv_bfloat16*>(&q0);
                    const __nv_bfloat16* a1 = reinterpret_cast<const __nv_bfloat16*>(&q1);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        v[c] = __bfloat162float(a0[c]) > 0.0f ? v[c] : 0.0f;
                        v[8 + c] = __bfloat162float(a1[c]) > 0.0f ? v[8 + c] : 0.0f;
                    }
                    float4* dst = reinterpret_cast<float4*>(static_cast<float*>(out_) + (size_t)sl * 16);
#pragma unroll
                    for (int k = 0; k < 4; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                } else {
                    uint4 o0, o1;
                    __nv_bfloat162* h0 = reinterpret_cast<__nv_bfloat162*>(&o0);
                    __nv_bfloat162* h1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        h0[k] = __floats2bfloat162_rn(fmaxf(v[2 * k], 0.0f), fmaxf(v[2 * k + 1], 0.0f));
                        h1[k] = __floats2bfloat162_rn(fmaxf(v[8 + 2 * k], 0.0f), fmaxf(v[8 + 2 * k + 1], 0.0f));
                    }
                    uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(out_) + (size_t)sl * 16);
                    dst[0] = o0;
                    dst[1] = o1;
                }
            }
        }
        tc_fence_before();
        __syncthreads();  // TMEM and the box are free for the next tile
        tc_fence_after();
    }
    if (s_abort) {
        if (tid == 0) atomicOr(err, 1);
        // bounded wait for the MMAs of the abandoned tile before freeing TMEM
        if (pending_mma) mbar_wait(mbar_s, phase);
        __syncthreads();
    }
}

template <int DIL, bool GRAD>
__global__ void __launch_bounds__(TcSmem<DIL>::kThreads)
    lp_mid_tc_kernel(LpGrid G, const __nv_bfloat16* __restrict__ wb, const void* __restrict__ in,
                     const __nv_bfloat16* __restrict__ ain, void* __restrict__ out, int* __restrict__ err) {
    using S = TcSmem<DIL>;
    constexpr int kThr = S::kThreads;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* wsm = smem + S::kBox;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + S::kBox + S::kW);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + S::kBox + S::kW + 16);
    __shared__ int s_abort;
    __shared__ uint32_t s_nb[2][27];  // this tile's neighbours and the next one's
    if (G.halt && *G.halt) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // weights: global [tap][ci][co] -> per tap a K-major B: rows = co, K = ci
    // (GRAD: rows = ci, K = co)
    for (int e = tid; e < 27 * 256; e += kThr) {
        const int tap = e >> 8, ci = (e >> 4) & 15, co = e & 15;
        const int row = GRAD ? ci : co, k = GRAD ? co : ci;
        *reinterpret_cast<__nv_bfloat16*>(wsm + tap * 512 + (k >> 3) * 256 + row * 16 + (k & 7) * 2) = wb[e];
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const uint32_t n = *G.d_nact, parts = tile_parts(n);
    if (warp == 1 && lane < 27 && blockIdx.x < n * parts)
        s_nb[0][lane] = tile_neighbour(G, G.act_tiles[blockIdx.x / parts], lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    if (parts == 1u) mid_tc_tiles<DIL, GRAD, false>(G, in, ain, out, err, n, tmem, smem, s_abort, s_nb);
    else mid_tc_tiles<DIL, GRAD, true>(G, in, ain, out, err, n, tmem, smem, s_abort, s_nb);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols) : "memory");
}

template <int DIL, bool GRAD>
static int launch_mid_tc(const LpGrid& G, const __nv_bfloat16* wb, const void* in, const __nv_bfloat16* ain, void* out,
                         int* err, int sms, cudaStream_t st) {
    using S = TcSmem<DIL>;
    const auto kernel = lp_mid_tc_kernel<DIL, GRAD>;
    static bool attr_set = false;  // per process; the attribute is per function
    if (!attr_set) {
        FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes));
        // all of the unified L1 as shared memory, so several CTAs fit per SM
        FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        attr_set = true;
    }
    // CTAs per SM from the shared-memory budget (each CTA also holds 1 KB of
    // static and 1 KB of reserved shared memory); at most 4 x 128 TMEM columns
    int dev = 0, smem_sm = 0;
    FLIP_CUDA_TRY(cudaGetDevice(&dev));
    FLIP_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    int per_sm = smem_sm / (S::kBytes + 2048);
    per_sm = per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm);
    kernel<<<sms * per_sm, S::kThreads, S::kBytes, st>>>(G, wb, in, ain, out, err);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

// ------------------------------------------------------------ small grids
// The 16 -> 16 layers on a small grid whose every tile is active (the
// coarsest level of the multilevel preconditioner, at most 4,096 voxels):
// one CTA per 128 consecutive voxels of the tile list.  The CTA gathers, for
// each of the 27 taps, its voxels' 16 input channels into an A operand of
// 128 rows (K-major, no swizzle: rows 16 B apart, 8-row groups 128 B apart,
// the two 8-channel halves 2 KB apart), so that one thread issues 27 MMAs of
// M=128 x N=16 x K=16 into one TMEM accumulator (row m in lane m).  Warps 0-3
// read their 32 lanes back, apply ReLU and store BF16.  Waits are bounded as
// in the per-tile kernel above.
namespace {
constexpr int kSmTcThreads = 256;
constexpr int kSmTcRows = 128;
constexpr int kSmTcA = 27 * kSmTcRows * 32;  // 27 taps x 128 rows x 16 BF16
constexpr int kSmTcW = 27 * 512;
constexpr int kSmTcBytes = kSmTcA + kSmTcW + 64;
constexpr uint32_t kInstrDescM128 = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
}  // namespace

__global__ void __launch_bounds__(kSmTcThreads) lp_small_mid_tc_kernel(LpGrid G, const __nv_bfloat16* __restrict__ wb, int dil,
                                                                       const __nv_bfloat16* __restrict__ in,
                                                                       __nv_bfloat16* __restrict__ out, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* asm_ = smem;
    unsigned char* wsm = smem + kSmTcA;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + kSmTcA + kSmTcW);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kSmTcA + kSmTcW + 16);
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t v0 = blockIdx.x * kSmTcRows;
    // weights: global [tap][ci][co] -> per tap [ci/8][co][ci%8]; 27 per thread,
    // loaded in batches of nine before they are stored
#pragma unroll
    for (int m0 = 0; m0 < 27; m0 += 9) {
        __nv_bfloat16 w[9];
#pragma unroll
        for (int j = 0; j < 9; ++j) w[j] = wb[tid + (m0 + j) * kSmTcThreads];
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const int e = tid + (m0 + j) * kSmTcThreads;
            const int tap = e >> 8, ci = (e >> 4) & 15, co = e & 15;
            *reinterpret_cast<__nv_bfloat16*>(wsm + tap * 512 + (ci >> 3) * 256 + co * 16 + (ci & 7) * 2) = w[j];
        }
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    // A: for each tap, row r = voxel v0 + r, half h = channels 8h .. 8h+7.
    // A thread keeps one (row, half) and walks the 27 taps: its voxel is
    // worked out once (the tile list is the problem's, not the previous
    // kernel's), and all its copies are in flight together.
    const int h = tid & 1, r = tid >> 1;  // 256 threads = 128 rows x 2 halves
    const uint32_t nvox = *G.d_nact * 512u;
    const uint32_t vx = v0 + (uint32_t)r;
    const bool have = vx < nvox;
    const uint32_t key = have ? G.act_tiles[vx >> 9] : 0u;
    int ci, cj, ck;
    tile_origin_tc(key, G.D, ci, cj, ck);
    ci += (int)(vx & 7u);
    cj += (int)((vx >> 3) & 7u);
    ck += (int)((vx >> 6) & 7u);
    pdl_wait();
    pdl_trigger();
    if (G.halt && *G.halt) return;
    if (v0 >= nvox) return;
    {
        const uint32_t dst = smem_u32(asm_) + (uint32_t)(h * (kSmTcRows * 16) + r * 16);
#pragma unroll
        for (int tap = 0; tap < 27; ++tap) {
            const int dz = tap / 9 - 1, dy = (tap / 3) % 3 - 1, dx = tap % 3 - 1;
            const int gx = ci + dil * dx, gy = cj + dil * dy, gz = ck + dil * dz;
            const bool ok = have && gx >= 0 && gy >= 0 && gz >= 0 && gx < G.D.nx && gy < G.D.ny && gz < G.D.nz;
            const uint32_t tt = (uint32_t)((gx >> 3) + G.D.tx * ((gy >> 3) + G.D.ty * (gz >> 3)));
            const uint32_t sl = ok ? (tt << 9) | rel_local(gx, gy, gz) : 0u;
            cp_async16(dst + (uint32_t)(tap * (kSmTcRows * 32)), in + (size_t)sl * 16 + h * 8, ok);
        }
        cp_async_commit();
        cp_async_wait<0>();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(32)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the generic-proxy stores above become visible to the tensor core's async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t a_s = smem_u32(asm_), w_s = smem_u32(wsm), mbar_s = smem_u32(mbar);
    if (tid == 0) {
        for (int tap = 0; tap < 27; ++tap) {
            const uint64_t ad = umma_desc(a_s + (uint32_t)(tap * kSmTcRows * 32), kSmTcRows * 16, 128);
            const uint64_t bd = umma_desc(w_s + (uint32_t)(tap * 512), 256, 128);
            mma_f16(tmem, ad, bd, kInstrDescM128, tap > 0 ? 1u : 0u);
        }
        mma_commit(mbar_s);
    }
    // one decision for the whole CTA: the TMEM reads below are warp-collective
    if (!mbar_wait(mbar_s, 0)) atomicExch(&s_abort, 1);
    __syncthreads();
    const bool ok = s_abort == 0;
    tc_fence_after();
    if (ok && warp < 4) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16), v);
        const uint32_t vx = v0 + (uint32_t)(32 * warp + lane);
        if (vx < nvox) {
            const uint32_t sl = (G.act_tiles[vx >> 9] << 9) | (vx & 511u);
            uint4 o0, o1;
            __nv_bfloat162* h0 = reinterpret_cast<__nv_bfloat162*>(&o0);
            __nv_bfloat162* h1 = reinterpret_cast<__nv_bfloat162*>(&o1);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                h0[k] = __floats2bfloat162_rn(fmaxf(v[2 * k], 0.0f), fmaxf(v[2 * k + 1], 0.0f));
                h1[k] = __floats2bfloat162_rn(fmaxf(v[8 + 2 * k], 0.0f), fmaxf(v[8 + 2 * k + 1], 0.0f));
            }
            uint4* dst = reinterpret_cast<uint4*>(out + (size_t)sl * 16);
            dst[0] = o0;
            dst[1] = o1;
        }
    }
    if (!ok) {
        if (tid == 0) atomicOr(err, 1);
        mbar_wait(mbar_s, 0);  // bounded: the MMAs before TMEM is freed
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32) : "memory");
}

// ------------------------------------------------------------ backward
// The input gradient of the 16 -> 16 layers is lp_mid_tc_kernel<DIL, true>.
//
// Weight gradient (wgrad), every layer: dW[tap][ci][co] = sum_v In[v + dil
// off(tap)][ci] Gout[v][co], a GEMM whose reduction runs over the voxels.  A
// persistent grid, a CTA per SM, takes the listed tiles in turn and stages a
// tile's input box, as the forward kernel does, in rows of x for each (z, y, 8-channel
// half), the rows of y and y + dil next to each other.  K = 16 voxels are the
// rows y and y + dil of a z-slice (8 voxels each, 16 B apart), and M = 64 rows
// are eight consecutive box rows of 8 channels: the taps dy = -1, 0, 1 of one
// (dz, dx) with their halves, read straight from the box as an MN-major A,
// and two more that come to nothing.  So a K-step is nine MMAs, one per (dz,
// dx), each into its own accumulator.  Gout at the tile's own voxels is an
// MN-major B (voxels along K, co along N): its BF16 rounding in columns 0-15 and
// the BF16 rounding of the remainder in columns 16-31, so that the products
// keep about 16 bits of Gout (and of the input layer's r/s, split the same way
// into two rows).  The accumulators collect all of a CTA's tiles; at the end
// warps 0-3 add them into dW with FP32 atomics.
//
// What bounds it at dilation 4 is the box's way from L2 (8 times the tile),
// below that its 288 MMAs a tile, some 65 cycles each.  Up to dilation 2 two
// boxes fit, and the next tile's copies (cp.async) run beside the MMAs.  128^3,
// 4,096 tiles: 16 -> 16 layers 275 and 285 us (dilation 2 and 4), 16 -> 1 218 us,
// 3 -> 16 205 us.  Gathering all 27 neighbours of each voxel into one A operand
// took 610 us (both dilations), 480 and 560 us with a wait for the MMAs before the
// next gather, and 460, 420 and 270 us with three stages of copies ahead of
// them: 27 reads of a voxel from L2 instead of 3.4 or 8.
// Waits are bounded as in the forward kernels.
namespace {
constexpr int kBwThreads = 512;

// the BF16 rounding of what bf16x8 dropped
__device__ __forceinline__ uint4 bf16x8_rest(const float4& a, const float4& b, const uint4& hi) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&hi);
    const float2 h0 = __bfloat1622float2(h[0]), h1 = __bfloat1622float2(h[1]), h2 = __bfloat1622float2(h[2]),
                 h3 = __bfloat1622float2(h[3]);
    return bf16x8(make_float4(a.x - h0.x, a.y - h0.y, a.z - h1.x, a.w - h1.y),
                  make_float4(b.x - h2.x, b.y - h2.y, b.z - h3.x, b.w - h3.y));
}
}  // namespace

// Weight-gradient layouts per layer (WG): the box rows, the accumulators'
// M rows and B's columns.
//   WG 1 (16 -> 16): two halves a row, M rows (dy, half, ci % 8); B = Gout
//                    [slot][16] as a high and a low part, N = 32; dW = their sum.
//   WG 2 (16 -> 1):  rows as WG 1; B = s gz [slot] with its high part in
//                    column 0 and its low part in column 1, N = 16;
//                    dW = column 0 + column 1.  Voxels: the output list.
//   WG 0 (3 -> 16):  one row of [r/s high, fluid, solid, r/s low, 0, 0, 0, 0] as
//                    lp_in_rows_kernel lays them out, M rows (dy, channel); B as
//                    WG 1; dW[.][0] = channel 0 + channel 3.
template <int WG, int DIL>
struct WgShape {
    static constexpr int B = 8 + 2 * DIL;
    static constexpr int kHalves = WG == 0 ? 1 : 2;
    static constexpr int kRow = B * 16 + (DIL == 4 ? 64 : 0);  // bytes of a box row (a voxel's halves on different banks)
    static constexpr int kBox = B * B * kHalves * kRow;
    static constexpr int kN = WG == 2 ? 16 : 32;
    static constexpr int kPart = 512 * 16;                     // bytes of eight of B's columns
    // B follows the box: the rows past a block of y that the MMAs read end in it
    static constexpr int kStage = kBox + (kN / 8) * kPart;
    static constexpr int kStages = 2 * kStage <= 220 * 1024 ? 2 : 1;
    static constexpr int kBytes = kStages * kStage + 64;
    static constexpr uint32_t kCols = WG == 2 ? 256 : 512;     // 9 accumulators of kN columns
    // FP32 += BF16 x BF16, A and B MN-major, N, M=64
    static constexpr uint32_t kInstr = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                       ((uint32_t)(kN >> 3) << 17) | ((64u >> 4) << 24);
    static_assert(kBytes <= 226 * 1024, "a stage has to fit");
    // box row of (z, y) in box coordinates
    __device__ static constexpr int row(int bz, int by) { return (bz * B + (by % DIL) * (B / DIL) + by / DIL) * kHalves; }
};

// the input layer's A rows, 16 bytes per slot of the active tiles
__global__ void __launch_bounds__(512) lp_in_rows_kernel(LpGrid G, const float* __restrict__ d_inv_s, uint4* __restrict__ rows) {
    const float inv_s = *d_inv_s;
    const uint32_t n = *G.d_nact;
    for (uint32_t t = blockIdx.x; t < n; t += gridDim.x) {
        const uint32_t u = (G.act_tiles[t] << 9) | threadIdx.x;
        const uint8_t ty = G.type[u];
        const float x = (ty == kFluid && G.r) ? G.r[u] * inv_s : 0.0f;
        const __nv_bfloat16 xh = __float2bfloat16_rn(x);
        uint4 v;
        __nv_bfloat162* hv = reinterpret_cast<__nv_bfloat162*>(&v);
        hv[0] = __halves2bfloat162(xh, __float2bfloat16_rn(ty == kFluid ? 1.0f : 0.0f));
        hv[1] = __floats2bfloat162_rn(ty == kSolid ? 1.0f : 0.0f, x - __bfloat162float(xh));
        hv[2] = hv[3] = __floats2bfloat162_rn(0.0f, 0.0f);
        rows[u] = v;
    }
}

// SPLIT: a tile's K-steps shared as tile_parts() says (a kernel of its own:
// with both forms in one, whole tiles of the input layer took 42 instead of 37 us
// on 343 tiles)
template <int WG, int DIL, bool SPLIT>
__global__ void __launch_bounds__(kBwThreads) lp_tc_wgrad_kernel(LpGrid G, const float* __restrict__ gout,
                                                                 const __nv_bfloat16* __restrict__ ain,
                                                                 const float* __restrict__ d_inv_s, float sign,
                                                                 const uint32_t* __restrict__ tiles,
                                                                 const uint32_t* __restrict__ d_n, float* __restrict__ dw,
                                                                 int* __restrict__ err) {
    using S = WgShape<WG, DIL>;
    constexpr int B = S::B, H = S::kHalves, kStages = S::kStages;
    extern __shared__ __align__(1024) unsigned char smem[];  // stages of the box, then B: [part][co half][512 v][8 co]
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + kStages * S::kStage);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + kStages * S::kStage + 32);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t n = *d_n, parts = SPLIT ? tile_parts(n) : 1u, all = n * parts;
    if (blockIdx.x >= all) return;
    const int nz = 8 / (int)parts;
    const float scale = WG == 2 ? sign / *d_inv_s : 1.0f;
    if (WG == 2)  // the columns that stay empty
        for (int e = tid; e < kStages * 2 * 512; e += kBwThreads)
            *reinterpret_cast<uint4*>(smem + (e >> 10) * S::kStage + S::kBox + (e & 1023) * 16) = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar + s)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(S::kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t smem_s = smem_u32(smem), mbar_s = smem_u32(mbar);

    // lane nb < 27 of every warp holds the first slot of the tile's neighbour
    // nb (a shuffle looks one up); the next tile's, and the key of the one
    // after it, are loaded a tile ahead
    auto key_at = [&](uint32_t t) { return tiles[(t < all ? t : all - 1u) / parts]; };
    auto around = [&](uint32_t k) { return lane < 27 ? tile_neighbour(G, k, lane) : kNoTile; };
    uint32_t key = key_at(blockIdx.x), key1 = key_at(blockIdx.x + gridDim.x), nb = around(key);
    auto gather = [&](uint32_t t, int stage) {  // the tile key, or part of it, of place t; moves on to the next one
        unsigned char* st = smem + stage * S::kStage;
        // Gout at the tile's voxels: loads now, stores after the box's copies
        float4 g[2][2];
        float gz = 0.0f;
        if (WG == 2) {
            gz = gout[(key << 9) | (uint32_t)tid];
        } else {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int e = tid + m * kBwThreads;
                const float4* p = reinterpret_cast<const float4*>(gout + (size_t)((key << 9) | (uint32_t)(e >> 1)) * 16 + (e & 1) * 8);
                g[m][0] = p[0];
                g[m][1] = p[1];
            }
        }
        const uint32_t nb1 = around(key1), key2 = key_at(t + 2u * gridDim.x);
        int ox, oy, oz;
        tile_origin_tc(key, G.D, ox, oy, oz);
        const uint32_t st_s = smem_s + (uint32_t)(stage * S::kStage);
        const int z0 = (int)(t % parts) * nz;  // the box's planes that its slices take
        const int first = H * B * B * z0, last = H * B * B * (z0 + nz + 2 * DIL);
#pragma unroll 4
        for (int w0 = first + tid - lane; w0 < last; w0 += kBwThreads) {  // the same for the whole warp
            const int e = w0 + lane < last ? w0 + lane : last - 1;
            const int h = e % H, v = e / H;
            const int bx = v % B, by = (v / B) % B, bz = v / (B * B);
            const int px = bx - DIL, py = by - DIL, pz = bz - DIL;
            const uint32_t base = __shfl_sync(0xffffffffu, nb, rel_neighbour(px, py, pz));
            const bool ok = base != kNoTile && ox + px < G.D.nx && oy + py < G.D.ny && oz + pz < G.D.nz;
            const uint32_t sl = ok ? base | rel_local(px, py, pz) : 0u;
            if (w0 + lane < last)
                cp_async16(st_s + (uint32_t)((S::row(bz, by) + h) * S::kRow + bx * 16), ain + (size_t)sl * (8 * H) + h * 8, ok);
        }
        cp_async_commit();
        unsigned char* b = st + S::kBox;
        if (WG == 2) {
            const float x = gz * scale;
            const __nv_bfloat16 hi = __float2bfloat16_rn(x);
            __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(b + tid * 16);
            row[0] = hi;
            row[1] = __float2bfloat16_rn(x - __bfloat162float(hi));
        } else {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int e = tid + m * kBwThreads;
                const uint4 hi = bf16x8(g[m][0], g[m][1]);
                unsigned char* row = b + (e & 1) * S::kPart + (e >> 1) * 16;
                *reinterpret_cast<uint4*>(row) = hi;
                *reinterpret_cast<uint4*>(row + 2 * S::kPart) = bf16x8_rest(g[m][0], g[m][1], hi);
            }
        }
        key = key1;
        key1 = key2;
        nb = nb1;
    };
    gather(blockIdx.x, 0);
    uint32_t i = 0;  // tiles whose MMAs are on their way
    bool failed = false;
    // whether the MMAs of this CTA's k-th tile are done
    auto wait_tile = [&](uint32_t k) {
        return mbar_wait(mbar_s + 8u * (k % kStages), (k / kStages) & 1u);
    };
    for (uint32_t t = blockIdx.x; t < all; t += gridDim.x) {
        cp_async_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // one decision for the whole CTA
        if (__syncthreads_or(failed)) break;
        if (tid == 0) {
            const uint32_t a_s = smem_s + (i % kStages) * S::kStage, b_s = a_s + S::kBox;
            const int k0 = 4 * (int)(t % parts) * nz;
            for (int ks = k0; ks < k0 + 4 * nz; ++ks) {
                // rows y and y + DIL of slice z
                const int z = ks >> 2, y = ((ks & 3) / DIL) * 2 * DIL + (ks & 3) % DIL;
                const uint64_t bd = umma_desc(b_s + (uint32_t)((64 * z + 8 * y) * 16), DIL * 128, S::kPart);
                // a descriptor holds its address in units of 16 B, and the
                // offsets of the nine (dz, dx) are constants: an addition each
                const uint64_t ad = umma_desc(a_s + (uint32_t)(S::row(z, y) * S::kRow), H * S::kRow, S::kRow);
                const uint32_t add = (i > 0 || ks > k0) ? 1u : 0u;
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    mma_f16(tmem + (uint32_t)(S::kN * j), ad + (uint64_t)((S::row(DIL * (j / 3), 0) * S::kRow) / 16 + DIL * (j % 3)), bd,
                            S::kInstr, add);
            }
            mma_commit(mbar_s + 8u * (i % kStages));
        }
        ++i;
        if (t + gridDim.x < all) {
            // the stage is that of the tile kStages before: its MMAs have to be done
            if (i >= (uint32_t)kStages && !wait_tile(i - kStages)) failed = true;
            if (!__any_sync(0xffffffffu, failed)) gather(t + gridDim.x, (int)(i % kStages));
        }
    }
    cp_async_wait<0>();
    // the last commit covers every MMA before it (bounded: also before TMEM is freed)
    if (!wait_tile(i - 1)) failed = true;
    const bool abort = __syncthreads_or(failed) != 0;
    if (abort && tid == 0) atomicOr(err, 1);
    if (!abort && warp < 4) {
        tc_fence_after();
        for (int j = 0; j < 9; ++j) {
            float acc[16];
            tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(S::kN * j), acc);
            if (S::kN == 32) {
                float rest[16];
                tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(S::kN * j + 16), rest);
#pragma unroll
                for (int co = 0; co < 16; ++co) acc[co] += rest[co];
            }
            const int m = lane + 16 * warp;  // this lane's row of the accumulator, its box row g
            const int g = m / 8, dy = g / H;
            if (lane < 16 && dy < 3) {
                const int tap = 9 * (j / 3) + 3 * dy + j % 3;
                if (WG == 0) {
                    // r/s high (0) and low (3) both feed channel 0
                    const int ch = m & 7;
                    float* d = dw + (tap * 3 + (ch == 3 ? 0 : ch)) * 16;
                    if (ch <= 3) {
#pragma unroll
                        for (int co = 0; co < 16; ++co)
                            if (acc[co] != 0.0f) atomicAdd(d + co, acc[co]);
                    }
                } else {
                    const int cin = 8 * (g & 1) + (m & 7);
                    if (WG == 2) {
                        const float v = acc[0] + acc[1];
                        if (v != 0.0f) atomicAdd(dw + tap * 16 + cin, v);
                    } else {
                        float* d = dw + (tap * 16 + cin) * 16;
#pragma unroll
                        for (int co = 0; co < 16; ++co)
                            if (acc[co] != 0.0f) atomicAdd(d + co, acc[co]);
                    }
                }
            }
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kCols) : "memory");
}

template <int WG, int DIL, bool SPLIT>
static int launch_wgrad_form(const LpGrid& G, const float* gout, const __nv_bfloat16* ain, const float* d_inv_s, float sign,
                            const uint32_t* tiles, const uint32_t* d_n, float* dw, int* err, int sms, cudaStream_t st) {
    using S = WgShape<WG, DIL>;
    const auto kernel = lp_tc_wgrad_kernel<WG, DIL, SPLIT>;
    static bool attr_set = false;  // per process; the attribute is per function
    if (!attr_set) {
        FLIP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes));
        attr_set = true;
    }
    kernel<<<sms, kBwThreads, S::kBytes, st>>>(G, gout, ain, d_inv_s, sign, tiles, d_n, dw, err);
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}
// shared tiles where a box has no more of them than half the CTAs
template <int WG, int DIL>
static int launch_wgrad_tc(const LpGrid& G, const float* gout, const __nv_bfloat16* ain, const float* d_inv_s, float sign,
                           const uint32_t* tiles, const uint32_t* d_n, float* dw, int* err, int sms, cudaStream_t st) {
    const auto launch = 2ll * G.D.tx * G.D.ty * G.D.tz <= sms ? launch_wgrad_form<WG, DIL, true> : launch_wgrad_form<WG, DIL, false>;
    return launch(G, gout, ain, d_inv_s, sign, tiles, d_n, dw, err, sms, st);
}
int lp_in_wgrad_tc(const LpGrid& G, int dil, const float* gout, const float* d_inv_s, void* rows, float* dw, int* err, int sms,
                   cudaStream_t st) {
    if (dil != 1) return FLIP_ERR_ARG;
    lp_in_rows_kernel<<<4 * sms, 512, 0, st>>>(G, d_inv_s, static_cast<uint4*>(rows));
    return launch_wgrad_tc<0, 1>(G, gout, static_cast<const __nv_bfloat16*>(rows), d_inv_s, 1.0f, G.act_tiles, G.d_nact, dw, err,
                                 sms, st);
}
int lp_mid_wgrad_tc(const LpGrid& G, int dil, const float* gout, const __nv_bfloat16* ain, float* dw, int* err, int sms,
                    cudaStream_t st) {
    switch (dil) {
    case 2: return launch_wgrad_tc<1, 2>(G, gout, ain, nullptr, 1.0f, G.act_tiles, G.d_nact, dw, err, sms, st);
    case 4: return launch_wgrad_tc<1, 4>(G, gout, ain, nullptr, 1.0f, G.act_tiles, G.d_nact, dw, err, sms, st);
    default: return FLIP_ERR_ARG;
    }
}
int lp_out_wgrad_tc(const LpGrid& G, int dil, const float* gz, const __nv_bfloat16* ain, const float* d_inv_s, float sign,
                    float* dw, int* err, int sms, cudaStream_t st) {
    if (dil != 1) return FLIP_ERR_ARG;
    return launch_wgrad_tc<2, 1>(G, gz, ain, d_inv_s, sign, G.out_tiles, G.d_nout, dw, err, sms, st);
}

int lp_small_mid_forward_tc(const LpGrid& G, const __nv_bfloat16* wb, int dil, const __nv_bfloat16* in, __nv_bfloat16* out,
                            int* err, uint32_t ntiles, cudaStream_t st) {
    static bool attr_set = false;  // per process; the attribute is per function
    if (!attr_set) {
        FLIP_CUDA_TRY(cudaFuncSetAttribute(lp_small_mid_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmTcBytes));
        attr_set = true;
    }
    const int grid = (int)((ntiles * 512u + kSmTcRows - 1) / kSmTcRows);
    FLIP_CUDA_TRY(pdl_launch(lp_small_mid_tc_kernel, grid, kSmTcThreads, kSmTcBytes, st, G, wb, dil, in, out, err));
    FLIP_CUDA_TRY(cudaGetLastError());
    return FLIP_OK;
}

int lp_mid_forward_tc(const LpGrid& G, const __nv_bfloat16* wb, int dil, const __nv_bfloat16* in, __nv_bfloat16* out,
                      int* err, int sms, cudaStream_t st) {
    switch (dil) {
    case 1: return launch_mid_tc<1, false>(G, wb, in, nullptr, out, err, sms, st);
    case 2: return launch_mid_tc<2, false>(G, wb, in, nullptr, out, err, sms, st);
    case 4: return launch_mid_tc<4, false>(G, wb, in, nullptr, out, err, sms, st);
    default: return FLIP_ERR_ARG;
    }
}
int lp_mid_dgrad_tc(const LpGrid& G, const __nv_bfloat16* wb, int dil, const float* gout, const __nv_bfloat16* ain,
                    float* gin, int* err, int sms, cudaStream_t st) {
    switch (dil) {
    case 2: return launch_mid_tc<2, true>(G, wb, gout, ain, gin, err, sms, st);
    case 4: return launch_mid_tc<4, true>(G, wb, gout, ain, gin, err, sms, st);
    default: return FLIP_ERR_ARG;
    }
}

}  // namespace flip
