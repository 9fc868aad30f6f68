// pg_unet.cu -- the learned pressure guess: a 3-level 3D conv U-Net with 16
// base channels, BF16 weights and activations, FP32 accumulation on the
// tensor cores (mma.sync m16n8k16), trained on the device by its own
// forward and backward kernels.  No reference counterpart (panopaea has no
// learned component).
//
// Network (channels-last tensors [voxel][channel], level l = dims >> l):
//   X0 = (b / rms(b), n_open / 6, 0 x 14)
//   L0 16->16, L1 16->16 (skip0), P0 = avgpool(L1)
//   L2 16->32, L3 32->32 (skip1), P1 = avgpool(L3)
//   L4 32->64, L5 64->64
//   C1 = [up(L5) | L3] (96), L6 96->32, L7 32->32
//   C0 = [up(L7) | L1] (48), L8 48->16, L9 16->16
//   q = L9 . wh (FP32), 0 on solid cells; guess = q * rms(b) * out_scale / dt
// Every conv is 3x3x3, zero padded, followed by ReLU.
//
// Kernels:
//   tc::k_conv_tc  implicit-GEMM conv on tcgen05.mma (below)
//   k_conv   the same on mma.sync: M = voxels of a CTA tile, N = C_out,
//            K = 27 taps x C_in.  The input brick (tile + 1-voxel halo, one
//            16-channel chunk at a time) is staged in shared memory with a
//            48-byte voxel stride (conflict-free ldmatrix rows); B fragments
//            come pre-permuted from global memory (L1-resident weights).  The
//            backward-data pass is the same kernel with the transposed,
//            tap-mirrored weights and a ReLU-gate epilogue.
//   k_wgrad  dW[tap] = X(shifted)^T dZ for all 27 taps at once: tiles of X
//            (with halo) and dZ staged in shared memory and fed to the
//            tensor cores with ldmatrix.trans; per-CTA partials summed in
//            fixed order (deterministic).
//   small elementwise kernels: input, pooling, upsample+concat and their
//            backward forms, the output layer + loss, Adam, weight layouts.

#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "pg_internal.cuh"
#include "pg_solve.cuh"
#include "pg_tma.cuh"

namespace pg {
template <class T> int launch_laplacian(const pg_grid* g, T* out, const T* p, double dt);
}

namespace pg {
namespace unet {

typedef __nv_bfloat16 bf16;

constexpr int kL = 10;
constexpr int kCin[kL] = {16, 16, 16, 32, 32, 64, 96, 32, 48, 16};
constexpr int kCout[kL] = {16, 16, 32, 32, 64, 64, 32, 32, 16, 16};
constexpr int kLevel[kL] = {0, 0, 1, 1, 2, 2, 1, 1, 0, 0};
constexpr int kSkip[kL] = {0, 0, 0, 0, 0, 0, 3, 0, 1, 0};  // decoder layers 6, 8: the layer concatenated

inline i64 param_offset(int k) {
    i64 o = 0;
    for (int j = 0; j < k; ++j) o += 27LL * kCin[j] * kCout[j];
    return o;
}
inline i64 num_params() { return param_offset(kL) + 16; }

// ---------------------------------------------------------------------------
// Tensor-core primitives (inline PTX).

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x2_t(uint32_t& r0, uint32_t& r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}
// D += A (16x16, row) * B (16x8, col), bf16 inputs, f32 accumulators.
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    uint32_t u;
    memcpy(&u, &h, 4);
    return u;
}

// ---------------------------------------------------------------------------
// Implicit-GEMM 3x3x3 convolution.

enum { EPI_RELU = 0, EPI_NONE = 1, EPI_GATE = 2 };
constexpr int kConvThreads = 256;
constexpr int kRowBytes = 48;  // one brick voxel, one 16-channel chunk: 32 B + 16 B pad

struct ConvGeom {
    int D, H, W;
    int TX, TY, TZ;
    int BX, BY;  // brick extent (tile + 2) in x and y
    int tiles_x, tiles_y;
};

// out[v][co] = epi(sum_tap sum_ci in[v + off(tap)][ci] * w[tap][ci][co]).
// wf: fragments [tap][CIN/16][COUT/8][lane] of the B operand.
template <int CIN, int COUT, int MT>
__global__ void __launch_bounds__(kConvThreads) k_conv(const bf16* __restrict__ in, const uint2* __restrict__ wf,
                                                       bf16* __restrict__ out, const bf16* __restrict__ gate,
                                                       ConvGeom G, int epi) {
    extern __shared__ __align__(16) unsigned char brick[];
    constexpr int NT = COUT / 8, KC = CIN / 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int t = blockIdx.x;
    const int tx0 = (t % G.tiles_x) * G.TX;
    t /= G.tiles_x;
    const int ty0 = (t % G.tiles_y) * G.TY;
    const int tz0 = (t / G.tiles_y) * G.TZ;
    const int nbrick = G.BX * G.BY * (G.TZ + 2);
    const uint32_t sbase = smem_addr(brick);

    // ldmatrix row address of this lane for each m-tile: voxel (lane & 15)
    // of the tile, channel half (lane >> 4) of the 16-channel chunk.
    uint32_t arow[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int v = (warp * MT + mt) * 16 + (lane & 15);
        const int x = v % G.TX, y = (v / G.TX) % G.TY, z = v / (G.TX * G.TY);
        arow[mt] = sbase + ((z * G.BY + y) * G.BX + x) * kRowBytes + (lane >> 4) * 16;
    }
    float acc[MT][NT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[mt][nt][j] = 0.f;

    for (int kc = 0; kc < KC; ++kc) {
        if (kc) __syncthreads();
        for (int i = threadIdx.x; i < nbrick * 2; i += kConvThreads) {
            const int bv = i >> 1, hf = i & 1;
            const int bx = bv % G.BX, r = bv / G.BX;
            const int by = r % G.BY, bz = r / G.BY;
            const int gx = tx0 + bx - 1, gy = ty0 + by - 1, gz = tz0 + bz - 1;
            uint4 val = make_uint4(0u, 0u, 0u, 0u);
            if ((unsigned)gx < (unsigned)G.W && (unsigned)gy < (unsigned)G.H && (unsigned)gz < (unsigned)G.D)
                val = __ldg(reinterpret_cast<const uint4*>(in + (((size_t)gz * G.H + gy) * G.W + gx) * CIN + kc * 16 +
                                                           hf * 8));
            *reinterpret_cast<uint4*>(brick + bv * kRowBytes + hf * 16) = val;
        }
        __syncthreads();
#pragma unroll 1
        for (int tap = 0; tap < 27; ++tap) {
            const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
            const uint32_t toff = (uint32_t)(((dz * G.BY + dy) * G.BX + dx) * kRowBytes);
            uint32_t a[MT][4];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) ldsm_x4(a[mt], arow[mt] + toff);
            const uint2* wp = wf + ((size_t)(tap * KC + kc) * NT) * 32 + lane;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 b = __ldg(wp + nt * 32);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) mma_bf16(acc[mt][nt], a[mt], b.x, b.y);
            }
        }
    }

#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int v = (warp * MT + mt) * 16 + (lane >> 2) + hf * 8;
            const int x = tx0 + v % G.TX, y = ty0 + (v / G.TX) % G.TY, z = tz0 + v / (G.TX * G.TY);
            if (x >= G.W || y >= G.H || z >= G.D) continue;
            const size_t o = (((size_t)z * G.H + y) * G.W + x) * COUT + (lane & 3) * 2;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float v0 = acc[mt][nt][hf * 2], v1 = acc[mt][nt][hf * 2 + 1];
                if (epi == EPI_RELU) {
                    v0 = v0 > 0.f ? v0 : 0.f;
                    v1 = v1 > 0.f ? v1 : 0.f;
                } else if (epi == EPI_GATE) {
                    const __nv_bfloat162 gv = *reinterpret_cast<const __nv_bfloat162*>(gate + o + nt * 8);
                    if (!(__bfloat162float(gv.x) > 0.f)) v0 = 0.f;
                    if (!(__bfloat162float(gv.y) > 0.f)) v1 = 0.f;
                }
                *reinterpret_cast<__nv_bfloat162*>(out + o + nt * 8) = __floats2bfloat162_rn(v0, v1);
            }
        }
}

// ---------------------------------------------------------------------------
// The same convolution on the fifth-generation tensor cores: tcgen05.mma
// (kind::f16, BF16 operands, FP32 accumulators in tensor memory), issued by
// the elected lane of a warp of its own, operands described in shared memory.
//
// GEMM per tile: M = 128 output voxels (an 8 x 16 x-y tile of one z plane),
// N = C_out, K = 27 taps x C_in; TZ consecutive z planes per tile, each with
// its own 128 x N accumulator in tensor memory.  The input brick (tile plus
// a one-voxel halo, TZ + 2 planes) is staged per 16-channel chunk as
// [bz][by][bx] x 32 bytes in the 32-byte swizzle (the halves of a voxel change
// places where bit 7 of its address is set), by one TMA load that also fills
// in the zeros outside the grid.  In that layout the A operand of every tap
// is a K-major operand inside the brick -- 8 consecutive x voxels, 8-row
// groups one brick row (BX x 32 B) apart -- so a tap is only a different
// start address: no im2col copy.  The weights of a chunk arrive pre-laid-out
// as [tap][8-channel half][n][8] (B operand, K-major, no swizzle: n rows 16 B
// apart, 8-row groups 128 B apart, halves N x 16 B apart).
//
// A CTA walks over tiles and keeps the tensor cores fed: three stages of
// bricks and two sets of accumulators, so that while the MMAs of one (tile,
// chunk) run, the bricks of the next two are on their way and eight warps
// write out the tile before.  A ninth warp issues the MMAs: it is held up
// while the tensor cores' queue is full, for about as long as they compute.
// The weights stay in shared memory where all of a layer's fit beside the
// bricks, else a chunk's travel with its brick.  An MMA of N = 48 takes 42
// cycles where its 4 KB A operand alone takes 32 to read; a 16 -> 16 tile is
// 54 of them, 33 us of a layer at 128^3, which takes 42 (48 -> 16: 131).  One
// CTA per tile, loading, multiplying and storing in turn, took 83 (182); with
// this walk but the bricks loaded by the eight warps (9 loads and stores of 16
// bytes per thread, 1200 to 2300 cycles of every 3800) 58 (141).
namespace tc {

constexpr int TX = 8, TY = 16, BX = TX + 2, BY = TY + 2;
constexpr int kVox = 32;  // bytes of a voxel's 16 channels
constexpr int kWorkers = 256, kThreads = kWorkers + 32;  // copy and write out; issue the MMAs

// Shared-memory matrix descriptor, no swizzle (start, leading- and
// stride-dimension byte offsets in 16-byte units; descriptor version 1), and
// the 32-byte swizzle's bits to add (patterns start at multiples of 256 B).
constexpr uint64_t kSwizzle32 = 6ull << 61;
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 1 in one lane of the (converged) warp.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p;
}
// Called by a whole warp, issued by its elected lane: with every operand
// uniform over the warp an MMA takes a few instructions to issue; from a
// divergent thread each operand's way into the uniform registers made it 93
// cycles, more than the tensor cores need for N <= 96.
__device__ __forceinline__ void mma(uint32_t leader, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                    uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(leader)
        : "memory");
}
// One arrival on bar once every tcgen05.mma the elected lane issued has completed.
__device__ __forceinline__ void commit(uint32_t leader, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
        "r"(leader)
        : "memory");
}
// Zero 16 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void st16_zero(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
        "r"(0u)
        : "memory");
}

// 16 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Contiguous copy by the bulk-copy engine, completing on bar.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void st_shared(uint32_t at, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Small output channel counts merge the three z taps into one MMA: an input
// brick plane bs feeds output planes bs, bs - 1 and bs - 2 through the taps
// dz = 0, 1, 2 with the same A operand, so their weights are stacked along N
// (N' = 3 N) and the planes' accumulators are laid out in reverse order
// (plane t at column (TZ + 1 - t) N): one MMA per input plane and (dx, dy)
// writes the three planes' columns.  Planes -2, -1, TZ, TZ + 1 take the edge
// products that no output needs.  Half the A-operand reads of the 27-tap
// loop, for the layers whose MMA is bound by that shared-memory traffic.
__host__ __device__ constexpr bool merge_dz(int n) { return n <= 32; }

template <int CIN, int COUT, int TZ_> struct Cfg {
    static constexpr bool kMerge = merge_dz(COUT);
    static constexpr int KC = CIN / 16;
    static constexpr int TZ = TZ_;
    static constexpr int BZ = TZ + 2;
    static constexpr int kBrick = BX * BY * BZ * kVox;    // one 16-channel chunk
    static constexpr int kWTap = 2 * COUT * 16;           // one tap of one chunk
    static constexpr int kWTap9 = 3 * kWTap;              // merged: the three z taps of one (dx, dy)
    static constexpr int kWChunk = 27 * kWTap;
    // Stages: three where they fit; all of the weights beside them or, where
    // those don't fit even with two, a chunk with each brick.
    static constexpr int kBrickOff = 256, kFree = 227 * 1024 - kBrickOff - 256;
    static constexpr bool kResident = 2 * kBrick + KC * kWChunk <= kFree;
    static constexpr int NS = (kResident ? 3 * kBrick + KC * kWChunk : 3 * (kBrick + kWChunk)) <= kFree ? 3 : 2;
    static constexpr int kWOff = kBrickOff + NS * kBrick;
    static constexpr size_t kSmem = kWOff + (size_t)(kResident ? KC : NS) * kWChunk;
    static constexpr int kAccCols = kMerge ? (TZ + 4) * COUT : TZ * COUT;
    static constexpr int kCols = kAccCols <= 32 ? 64 : (kAccCols <= 64 ? 128 : (kAccCols <= 128 ? 256 : 512));  // two sets
    static_assert(kAccCols <= 256, "two sets of accumulators must fit in tensor memory");
    static_assert(kSmem + 256 <= 227 * 1024, "bricks and weights must fit in shared memory");
    static_assert(kBrick % 256 == 0 && kWChunk % 128 == 0, "operand alignment");
    // tensor-memory column of output plane t's accumulator
    __host__ __device__ static constexpr int col(int t) { return kMerge ? (TZ + 1 - t) * COUT : t * COUT; }
};

struct Geom {
    int D, H, W;
    int tiles_x, tiles_y, tiles;
};

// vox: the input's map.  wtc: [chunk][tap][half][n][8] BF16 (see above).
// CA > 0: the input is the concatenation [up's voxel at half the coordinates
// (CA channels) | vox] that k_upcat would write.  err: set when a wait for the tensor cores gave
// up (the result is then not to be trusted).
template <int CIN, int COUT, int TZ_, int CA>
__global__ void __launch_bounds__(kThreads)
    k_conv_tc(const __grid_constant__ CUtensorMap vox, const bf16* __restrict__ up, const bf16* __restrict__ wtc,
              bf16* __restrict__ out, const bf16* __restrict__ gate, Geom G, int epi, int* err) {
    typedef Cfg<CIN, COUT, TZ_> C;
    constexpr int KC = C::KC, TZ = C::TZ;
    constexpr uint32_t kIdesc = idesc_bf16(128, COUT);
    extern __shared__ __align__(128) unsigned char tc_smem_raw[];
    unsigned char* const base = tc_smem_raw + ((256u - (smem_u32(tc_smem_raw) & 255u)) & 255u);
    constexpr int NS = C::NS;
    uint64_t* const full = (uint64_t*)base;  // per stage, items in turn: the warps are ready for the item's MMAs
    uint64_t* const cfull = full + NS;       // what is copied for it (brick, weights) is in shared memory
    uint64_t* const bar = cfull + NS;        // its MMAs are done
    uint32_t* const tslot = (uint32_t*)(base + 128);
    const uint32_t bricks = smem_u32(base + C::kBrickOff), wsm = smem_u32(base + C::kWOff);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, half = warp >> 2;  // this warp's TMEM lanes 32 q .. +31, and every second accumulator
    if (warp == 0) tmem_alloc(tslot, C::kCols);
    if (tid == 0) {
        for (int k = 0; k < NS; ++k) {
            mbar_init(full + k, kWorkers / 32);
            mbar_init(cfull + k, 1);
            mbar_init(bar + k, 1);
        }
        mbar_fence_init();
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t tlane = tmem + ((uint32_t)(q * 32) << 16);
    constexpr int kUnits = TZ * COUT / 16;  // 128 x 16 pieces of a tile's accumulators
    if (C::kMerge && warp < kWorkers / 32) {  // every merged MMA accumulates: start the accumulators at zero
        for (int u = half; u < 2 * kUnits; u += 2) {
            const int v = u % kUnits;
            st16_zero(tlane + (uint32_t)((u / kUnits) * (C::kCols / 2) + C::col(v / (COUT / 16)) + v % (COUT / 16) * 16));
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    auto origin = [&](int tile, int& x0, int& y0, int& z0) {
        const int r = tile / G.tiles_x;
        x0 = (tile - r * G.tiles_x) * TX;
        z0 = r / G.tiles_y;
        y0 = (r - z0 * G.tiles_y) * TY;
        z0 *= TZ;
    };
    // item i: chunk i % KC of the CTA's tile i / KC
    const int items = ((G.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * KC;
    auto tile_of = [&](int i) { return (int)blockIdx.x + i / KC * (int)gridDim.x; };
    // What item i needs copied, started by one thread.
    auto brick_copied = [&](int i) { return CA == 0 || i % KC * 16 >= CA; };
    auto weights_copied = [&](int i) { return !C::kResident || i < KC; };
    auto copy = [&](int i) {
        const int kc = i % KC, s = i % NS;
        if (!brick_copied(i) && !weights_copied(i)) {
            mbar_arrive(cfull + s);
            return;
        }
        mbar_expect_tx(cfull + s, (brick_copied(i) ? C::kBrick : 0) + (weights_copied(i) ? C::kWChunk : 0));
        if (brick_copied(i)) {
            int x0, y0, z0;
            origin(tile_of(i), x0, y0, z0);
            tma_load_4d(bricks + (uint32_t)(s * C::kBrick), &vox, cfull + s, kc * 16 - CA, x0 - 1, y0 - 1, z0 - 1);
        }
        if (weights_copied(i))
            bulk_load(wsm + (uint32_t)((C::kResident ? kc : s) * C::kWChunk),
                      reinterpret_cast<const unsigned char*>(wtc) + (size_t)kc * C::kWChunk, C::kWChunk, cfull + s);
    };
    // A brick of the upsampled channels: every voxel of `up` that its parents
    // cover is loaded once, 16 bytes per lane, and stored to its children.
    constexpr int UX = BX / 2 + 1, UY = BY / 2 + 1, UZ = C::BZ / 2 + 1, kUp = 2 * UX * UY * UZ;
    constexpr int NU = CA > 0 ? (kUp + kWorkers - 1) / kWorkers : 1;
    uint4 piece[NU];
    auto fetch_up = [&](int i) {
        int x0, y0, z0;
        origin(tile_of(i), x0, y0, z0);
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int j = tid + k * kWorkers, v = j >> 1;
            const int X = x0 / 2 - 1 + v % UX, Y = y0 / 2 - 1 + v / UX % UY, Z = z0 / 2 - 1 + v / (UX * UY);
            piece[k] = make_uint4(0u, 0u, 0u, 0u);
            if (j < kUp && (unsigned)X < (unsigned)(G.W / 2) && (unsigned)Y < (unsigned)(G.H / 2) &&
                (unsigned)Z < (unsigned)(G.D / 2))
                piece[k] = __ldg(reinterpret_cast<const uint4*>(
                    up + (((i64)Z * (G.H / 2) + Y) * (G.W / 2) + X) * CA + i % KC * 16 + (j & 1) * 8));
        }
    };
    auto fill_up = [&](int i) {
        const uint32_t brick = bricks + (uint32_t)(i % NS * C::kBrick);
#pragma unroll
        for (int k = 0; k < NU; ++k) {
            const int j = tid + k * kWorkers, v = j >> 1;
            const int bx = 2 * (v % UX) - 1, by = 2 * (v / UX % UY) - 1, bz = 2 * (v / (UX * UY)) - 1;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int x = bx + (c & 1), y = by + (c >> 1 & 1), z = bz + (c >> 2);
                const uint32_t at = brick + (uint32_t)(((z * BY + y) * BX + x) * kVox);
                if (j < kUp && (unsigned)x < BX && (unsigned)y < BY && (unsigned)z < C::BZ)
                    st_shared(at + (((uint32_t)j ^ at >> 7) & 1u) * 16, piece[k]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // stored brick -> tensor-core reads
    };
    auto multiply = [&](uint32_t leader, int i) {
        const int kc = i % KC;
        const uint32_t acc = tmem + (uint32_t)((i / KC & 1) * (C::kCols / 2));
        // (start addresses count in 16 bytes)
        const uint64_t a0 = sdesc(bricks + (uint32_t)(i % NS * C::kBrick), 16, BX * kVox) | kSwizzle32;
        const uint64_t b0 =
            sdesc(wsm + (uint32_t)((C::kResident ? kc : i % NS) * C::kWChunk), (C::kMerge ? 3 : 1) * COUT * 16, 128);
        if (C::kMerge) {
            constexpr uint32_t kIdesc3 = idesc_bf16(128, 3 * COUT);
#pragma unroll
            for (int tap9 = 0; tap9 < 9; ++tap9) {
                const int dy = tap9 / 3, dx = tap9 % 3;
#pragma unroll
                for (int pz = 0; pz < C::BZ; ++pz)
                    mma(leader, acc + (uint32_t)C::col(pz), a0 + (uint64_t)(((pz * BY + dy) * BX + dx) * (kVox / 16)),
                        b0 + (uint64_t)(tap9 * C::kWTap9 / 16), kIdesc3, 1u);
            }
        } else {
#pragma unroll
            for (int tap = 0; tap < 27; ++tap) {
                const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
#pragma unroll
                for (int tz = 0; tz < TZ; ++tz)
                    mma(leader, acc + (uint32_t)(tz * COUT), a0 + (uint64_t)((((tz + dz) * BY + dy) * BX + dx) * (kVox / 16)),
                        b0 + (uint64_t)(tap * C::kWTap / 16), kIdesc, (kc > 0 || tap > 0) ? 1u : 0u);
            }
        }
        commit(leader, bar + i % NS);
    };
    // The accumulators of the tile that ended with item i, written out (and zeroed).
    auto finish = [&](int i) {
        int x0, y0, z0;
        origin(tile_of(i), x0, y0, z0);
        const uint32_t acc = tlane + (uint32_t)((i / KC & 1) * (C::kCols / 2));
        const int m = q * 32 + lane;
        const int x = x0 + (m & 7), y = y0 + (m >> 3);
#pragma unroll 1
        for (int u = half; u < kUnits; u += 2) {
            const int tz = u / (COUT / 16), cg = u % (COUT / 16), z = z0 + tz;
            const bool in_grid = x < G.W && y < G.H && z < G.D;
            const size_t o = (((size_t)z * G.H + y) * G.W + x) * COUT + cg * 16;
            uint4 gv[2] = {};
            if (epi == EPI_GATE && in_grid) {
                gv[0] = *reinterpret_cast<const uint4*>(gate + o);
                gv[1] = *reinterpret_cast<const uint4*>(gate + o + 8);
            }
            const uint32_t at = acc + (uint32_t)(C::col(tz) + cg * 16);
            float v[16];
            ld16(at, v);
            if (C::kMerge) st16_zero(at);
            if (!in_grid) continue;
            if (epi == EPI_RELU) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = v[j] > 0.f ? v[j] : 0.f;
            } else if (epi == EPI_GATE) {
                const uint32_t gw[8] = {gv[0].x, gv[0].y, gv[0].z, gv[0].w, gv[1].x, gv[1].y, gv[1].z, gv[1].w};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    __nv_bfloat162 pr;
                    memcpy(&pr, &gw[j], 4);
                    if (!(__bfloat162float(pr.x) > 0.f)) v[2 * j] = 0.f;
                    if (!(__bfloat162float(pr.y) > 0.f)) v[2 * j + 1] = 0.f;
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
                *reinterpret_cast<uint4*>(out + o + 8 * j) =
                    make_uint4(pack_bf16(v[8 * j], v[8 * j + 1]), pack_bf16(v[8 * j + 2], v[8 * j + 3]),
                               pack_bf16(v[8 * j + 4], v[8 * j + 5]), pack_bf16(v[8 * j + 6], v[8 * j + 7]));
        }
        if (C::kMerge) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    };
    // A wait that gives up ends the warp's work and flags the result; the
    // others' waits then complete or give up as well.
    if (warp < kWorkers / 32) {
        auto done = [&](int i) {  // item i's MMAs (uniform per warp)
            const bool w = lane != 0 || mbar_wait(bar + i % NS, (unsigned)(i / NS) & 1u);
            const bool ok = __all_sync(0xffffffffu, w);
            fence_after();
            return ok;
        };
        bool ok = true;
        int last = -1;  // the last item whose copies were started
        auto load = [&](int i) {  // item i into its stage; then the pieces of the next
            if (i < items) {
                if (tid == 0) copy(i);
                if (CA > 0 && !brick_copied(i)) fill_up(i);
                last = i;
            }
            if (CA > 0 && i + 1 < items && !brick_copied(i + 1)) fetch_up(i + 1);
        };
        if (CA > 0) fetch_up(0);
        for (int i = 0; i < NS - 1; ++i) load(i);
        for (int i = 0; i < items; ++i) {
            fence_before();  // (accumulators read and zeroed)
            __syncwarp();
            if (lane == 0) mbar_arrive(full + i % NS);
            if (i > 0 && !(ok = done(i - 1))) break;  // the item before has read its operands
            load(i + NS - 1);
            if (i > 0 && i % KC == 0) finish(i - 1);
        }
        if (ok && (ok = done(items - 1))) finish(items - 1);
        if (!ok && lane == 0) {
            atomicExch(err, 1);
            if (tid == 0)  // (bounded) for the copies in flight
                for (int i = max(0, last - NS + 1); i <= last; ++i)
                    mbar_wait(cfull + i % NS, (unsigned)(i / NS) & 1u);
        }
    } else {
        const uint32_t leader = elect_one();
        for (int i = 0; i < items; ++i) {
            const unsigned parity = (unsigned)(i / NS) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(full + i % NS, parity) && mbar_wait(cfull + i % NS, parity))) {
                // flag it and wait (bounded) for the last committed group
                if (leader) {
                    atomicExch(err, 1);
                    if (i > 0) mbar_wait(bar + (i - 1) % NS, (unsigned)((i - 1) / NS) & 1u);
                }
                break;
            }
            fence_after();
            multiply(leader, i);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        tmem_dealloc(tmem, C::kCols);
    }
}

// Weights of the tensor-core path: wtc[chunk][tap][half][n][8] with the
// K index k = 16 chunk + 8 half + j an input channel of the convolution and
// n an output channel; forward W[tap][k][n], backward-data (transposed,
// tap-mirrored) W[26 - tap][n][k] of the forward layer.
// With merge_dz(N) the three z taps of one (dx, dy) are stacked along N:
// wtc[chunk][dy 3 + dx][half][dz N + n][8].
// blockIdx.y: layer, forward then backward-data (one launch: 19 of 3 us each
// were launch latency).
struct PrepArgs {
    const float* W[2 * kL];
    bf16* wtc[2 * kL];  // null: no such layout
    int cin[kL], cout[kL];
};
__global__ void k_wprep_tc(PrepArgs A) {
    const int layer = blockIdx.y >> 1, transposed = blockIdx.y & 1, cin = A.cin[layer], cout = A.cout[layer];
    const float* __restrict__ W = A.W[blockIdx.y];
    bf16* __restrict__ wtc = A.wtc[blockIdx.y];
    if (!wtc) return;
    const int K = transposed ? cout : cin, N = transposed ? cin : cout;
    const bool merged = merge_dz(N);
    const int n_all = 27 * K * N;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_all; i += gridDim.x * blockDim.x) {
        const int j = i & 7;
        int r = i >> 3;
        int n, hf, tap, kc;
        if (merged) {
            const int nn = r % (3 * N);
            r /= 3 * N;
            hf = r & 1;
            r >>= 1;
            const int tap9 = r % 9;
            kc = r / 9;
            n = nn % N;
            tap = (nn / N) * 9 + tap9;
        } else {
            n = r % N;
            r /= N;
            hf = r & 1;
            r >>= 1;
            tap = r % 27;
            kc = r / 27;
        }
        const int k = kc * 16 + hf * 8 + j;
        const float v = transposed ? W[((size_t)(26 - tap) * cin + n) * cout + k] : W[((size_t)tap * cin + k) * cout + n];
        wtc[i] = __float2bfloat16_rn(v);
    }
}

}  // namespace tc

// ---------------------------------------------------------------------------
// Weight gradient: part[s][tap][ci][co] = sum over CTA s's voxels v of
// X[v + off(tap)][ci] * dZ[v][co].
//
// A CTA owns 16 input and CO output channels and the nine taps of one dz
// (blockIdx.y), and a contiguous range of 8 x 16 x 2 voxel tiles.  It stages
// a tile's X with a one-voxel halo in x and y and its dZ in shared memory
// once for the nine taps, the next tile's copies in flight meanwhile.  Six
// warps: one per dx and half of the output channels; a K step of the MMA is
// the 8 x 2 (x, z) voxels of one row y.  Walking up the rows, the X fragment
// of row Y meets the dZ fragments of rows Y + 1, Y, Y - 1 (the taps
// dy = -1, 0, 1), of which two are still in registers, so one ldmatrix of
// each operand feeds 3 CO / 16 MMAs: the kernel is bound by the warp-level
// MMAs, not by shared memory.  The sums of a tap stay in registers over the
// whole range; the partials are folded in a fixed order by k_wgrad_sum.
// One CTA per tap, each staging both
// operands again, took 455 us (16 -> 16) and 1097 us (48 -> 16) at 96^3; now
// 64 and 195 us (190 TFLOP/s), with 3.2 TB/s of staging out of L2.  Nine
// warps for all three dz of a tile staged once (fewer bytes, but three times
// as many ranges for the same warps) took 57 and 150 us; its shorter sums
// move the gradient of a 48 -> 16 layer by 2.2e-5 of its norm, beyond what
// two orders of one FP32 sum should differ by.
constexpr int kWgThreads = 192;
constexpr int kWgX = 8, kWgY = 16, kWgZ = 2;  // tile (voxels)
constexpr int kWgBX = kWgX + 2, kWgBY = kWgY + 2;
constexpr int kWgBrick = kWgBX * kWgBY * kWgZ, kWgTile = kWgX * kWgY * kWgZ;
constexpr int kWgXS = 16 * 2 + 16;  // bytes per staged X voxel (the pad keeps ldmatrix rows off each other's banks)
__host__ __device__ constexpr int wg_zs(int co) { return co * 2 + 16; }
__host__ __device__ constexpr int wg_stage(int co) { return kWgBrick * kWgXS + kWgTile * wg_zs(co); }
__host__ __device__ constexpr int wg_co(int cout) { return cout < 32 ? cout : 32; }  // output channels of a CTA
// Resident CTAs per SM: three where a layer has few channel blocks; two for
// the wide layers (more than 32 input channels), whose partials are largest.
constexpr int kWgCtasPerSm = 3;
constexpr int wg_ctas_per_sm(int cin) { return cin > 32 ? 2 : kWgCtasPerSm; }

struct WgGeom {
    int D, H, W;
    int cin, cout;
    int ca;  // > 0: the first ca input channels come from `up`, at half the coordinates (X has the others)
    int tiles_x, tiles_y, tiles;
};

__device__ __forceinline__ void cp16_or_zero(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

template <int CO>
__global__ void __launch_bounds__(kWgThreads, kWgCtasPerSm)
    k_wgrad(const bf16* __restrict__ X, const bf16* __restrict__ up, const bf16* __restrict__ dZ,
            float* __restrict__ part, WgGeom G) {
    constexpr int ZV = CO / 8, NT = CO / 16, ZS = wg_zs(CO);  // 16-byte vectors per dZ voxel; n-tiles of a warp
    static_assert(NT == 1 || NT == 2, "a warp owns one or two n-tiles");
    extern __shared__ __align__(16) unsigned char wg_smem_raw[];
    const uint32_t base = smem_addr(wg_smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dx = warp % 3, nh = warp / 3;
    const int dz = blockIdx.y % 3, chunk = blockIdx.y / 3;
    const int ci0 = chunk % (G.cin / 16) * 16, co0 = chunk / (G.cin / 16) * CO;
    const int t_lo = (int)((i64)G.tiles * blockIdx.x / gridDim.x);
    const int t_hi = (int)((i64)G.tiles * (blockIdx.x + 1) / gridDim.x);
    // this lane's ldmatrix rows: X voxel (lane & 7, z lane >> 4), channel half
    // (lane >> 3) & 1; dZ voxel (lane & 7, z (lane >> 3) & 1), n-tile lane >> 4
    // (one n-tile: the upper lanes' addresses are not used)
    const uint32_t a_row = (((lane >> 4) * kWgBY) * kWgBX + (lane & 7) + dx) * kWgXS + ((lane >> 3) & 1) * 16;
    const uint32_t b_row = kWgBrick * kWgXS + ((((lane >> 3) & 1) * kWgY) * kWgX + (lane & 7)) * ZS +
                           (nh * NT + (NT == 2 ? lane >> 4 : 0)) * 16;
    auto origin = [&](int tile, int& x0, int& y0, int& z0) {
        const int r = tile / G.tiles_x;
        x0 = (tile - r * G.tiles_x) * kWgX;
        z0 = r / G.tiles_y;
        y0 = (r - z0 * G.tiles_y) * kWgY;
        z0 *= kWgZ;
    };
    auto stage = [&](int tile, int slot) {
        int x0, y0, z0;
        origin(tile, x0, y0, z0);
        const uint32_t xb = base + slot * wg_stage(CO), zb = xb + kWgBrick * kWgXS;
        for (int i = threadIdx.x; i < kWgBrick * 2; i += kWgThreads) {
            const int hf = i & 1, v = i >> 1;
            const int bx = v % kWgBX, q = v / kWgBX, by = q % kWgBY, bz = q / kWgBY;
            const int gx = x0 + bx - 1, gy = y0 + by - 1, gz = z0 + bz + dz - 1;
            const bool in = (unsigned)gx < (unsigned)G.W && (unsigned)gy < (unsigned)G.H && (unsigned)gz < (unsigned)G.D;
            const bf16* src = X;
            if (in && ci0 < G.ca)
                src = up + (((size_t)(gz >> 1) * (G.H >> 1) + (gy >> 1)) * (G.W >> 1) + (gx >> 1)) * G.ca + ci0 + hf * 8;
            else if (in)
                src = X + (((size_t)gz * G.H + gy) * G.W + gx) * (G.cin - G.ca) + ci0 - G.ca + hf * 8;
            cp16_or_zero(xb + v * kWgXS + hf * 16, src, in);
        }
        for (int i = threadIdx.x; i < kWgTile * ZV; i += kWgThreads) {
            const int p = i % ZV, v = i / ZV;
            const int gx = x0 + v % kWgX, q = v / kWgX, gy = y0 + q % kWgY, gz = z0 + q / kWgY;
            const bool in = gx < G.W && gy < G.H && gz < G.D;
            const size_t o = in ? (((size_t)gz * G.H + gy) * G.W + gx) * G.cout + co0 + p * 8 : 0;
            cp16_or_zero(zb + v * ZS + p * 16, dZ + o, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[3][NT][4];
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[t][n][j] = 0.f;

    if (t_lo < t_hi) stage(t_lo, 0);
    for (int tile = t_lo; tile < t_hi; ++tile) {
        const int slot = (tile - t_lo) & 1;
        if (tile + 1 < t_hi) {
            stage(tile + 1, slot ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        int x0, y0, z0;
        origin(tile, x0, y0, z0);
        const uint32_t ab = base + slot * wg_stage(CO) + a_row, bb = base + slot * wg_stage(CO) + b_row;
        const int rows = min(kWgY, G.H - y0);  // dZ rows of the tile inside the grid
        uint32_t b[3][NT][2];                  // dZ fragments of the last three rows, row r in b[r % 3]
        // X row y0 - 1 + by against dZ rows by - 1 - dy; cur = by % 3
        auto step = [&](int by, int cur, bool top, bool mid, bool low) {
            uint32_t a[4];
            ldsm_x4_t(a, ab + by * (kWgBX * kWgXS));
            if (top) {
                if (NT == 2) {
                    uint32_t f[4];
                    ldsm_x4_t(f, bb + by * (kWgX * ZS));
                    b[cur][0][0] = f[0];
                    b[cur][0][1] = f[1];
                    b[cur][NT - 1][0] = f[2];
                    b[cur][NT - 1][1] = f[3];
                } else {
                    ldsm_x2_t(b[cur][0][0], b[cur][0][1], bb + by * (kWgX * ZS));
                }
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_bf16(acc[0][n], a, b[cur][n][0], b[cur][n][1]);
            }
            const int p1 = (cur + 2) % 3, p2 = (cur + 1) % 3;
            if (mid) {
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_bf16(acc[1][n], a, b[p1][n][0], b[p1][n][1]);
            }
            if (low) {
#pragma unroll
                for (int n = 0; n < NT; ++n) mma_bf16(acc[2][n], a, b[p2][n][0], b[p2][n][1]);
            }
        };
        if (rows == kWgY) {  // no branch between the rows: the loads of later rows move up
#pragma unroll
            for (int by = 0; by < kWgY + 2; ++by) step(by, by % 3, by < kWgY, by >= 1 && by <= kWgY, by >= 2);
        } else {
#pragma unroll 1
            for (int by = 0; by < rows + 2; by += 3) {
                step(by, 0, by < rows, by >= 1 && by <= rows, by >= 2);
                if (by + 1 < rows + 2) step(by + 1, 1, by + 1 < rows, by + 1 <= rows, by >= 1);
                if (by + 2 < rows + 2) step(by + 2, 2, by + 2 < rows, by + 2 <= rows, true);
            }
        }
        __syncthreads();  // this slot may be staged again
    }
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int tap = dz * 9 + t * 3 + dx;
        float* out = part + (((size_t)blockIdx.x * 27 + tap) * G.cin + ci0) * G.cout + co0;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int co = (nh * NT + n) * 8 + 2 * tq;
            *reinterpret_cast<float2*>(out + g * G.cout + co) = make_float2(acc[t][n][0], acc[t][n][1]);
            *reinterpret_cast<float2*>(out + (g + 8) * G.cout + co) = make_float2(acc[t][n][2], acc[t][n][3]);
        }
    }
}

// grad[i] += sum_s part[s][i]: eight interleaved runs of s, each in order,
// then the eight in order (32 outputs per block, so the reads are whole
// 128-byte lines and S / 8 loads follow one another instead of S).
// All layers in one launch (ten of 7 us each were launch latency).
struct WgSumArgs {
    const float* part[kL];
    float* grad[kL];
    int S[kL], n[kL], block0[kL];  // block0: a layer's first block
};
__global__ void __launch_bounds__(256) k_wgrad_sum(WgSumArgs A) {
    __shared__ float sm[8][32];
    const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
    int layer = kL - 1;
    while (blockIdx.x < (unsigned)A.block0[layer]) --layer;
    const float* __restrict__ part = A.part[layer];
    float* __restrict__ grad = A.grad[layer];
    const int S = A.S[layer], n = A.n[layer];
    const int i = (blockIdx.x - A.block0[layer]) * 32 + lane;  // n is a multiple of 32
    float s = 0.f;
#pragma unroll 4
    for (int k = seg; k < S; k += 8) s += __ldg(part + (size_t)k * n + i);
    sm[seg][lane] = s;
    __syncthreads();
    if (seg) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) s += sm[k][lane];
    grad[i] += s;
}

// ---------------------------------------------------------------------------
// Weight layouts: forward B fragments and the transposed, tap-mirrored ones
// of the backward-data pass (W'[tap][co][ci] = W[26 - tap][ci][co]).
__global__ void k_wprep(const float* __restrict__ W, int cin, int cout, uint2* __restrict__ wf,
                        uint2* __restrict__ wt) {
    const int KC = cin / 16, NT = cout / 8, KCt = cout / 16, NTt = cin / 8;
    const int nf = 27 * KC * NT * 32, ntr = wt ? 27 * KCt * NTt * 32 : 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + ntr; i += gridDim.x * blockDim.x) {
        const bool fwd = i < nf;
        const int j = fwd ? i : i - nf;
        const int lane = j & 31, g = lane >> 2, tq = lane & 3;
        int r = j >> 5;
        const int nt = r % (fwd ? NT : NTt);
        r /= fwd ? NT : NTt;
        const int kc = r % (fwd ? KC : KCt), tap = r / (fwd ? KC : KCt);
        if (fwd) {
            const int co = nt * 8 + g, ci = kc * 16 + 2 * tq;
            const float* base = W + (size_t)tap * cin * cout + co;
            wf[j] = make_uint2(pack_bf16(base[ci * cout], base[(ci + 1) * cout]),
                               pack_bf16(base[(ci + 8) * cout], base[(ci + 9) * cout]));
        } else {
            const int ci = nt * 8 + g, co = kc * 16 + 2 * tq;
            const float* base = W + ((size_t)(26 - tap) * cin + ci) * cout + co;
            wt[j] = make_uint2(pack_bf16(base[0], base[1]), pack_bf16(base[8], base[9]));
        }
    }
}

// ---------------------------------------------------------------------------
// Input normalisation.

constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 512;

__global__ void __launch_bounds__(kRedThreads) k_sumsq(const float* __restrict__ b, i64 n, double* __restrict__ part) {
    __shared__ double sm[kRedThreads];
    double s = 0.0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const double v = b[i];
        s += v * v;
    }
    s = block_sum<kRedThreads>(s, sm);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// The sum of a stride-spaced column of partials, by one warp (a thread alone
// takes 60 cycles per addition: 33 us for 512).
__device__ __forceinline__ double warp_fold(const double* __restrict__ part, int n, int stride) {
    double s = 0.0;
    for (int i = threadIdx.x & 31; i < n; i += 32) s += part[(size_t)i * stride];
    return warp_sum(s);
}

// scal = {s, 1/s, s * out_scale, dt / (s * out_scale)}
__global__ void k_scalars(const double* __restrict__ part, int nparts, i64 n, float out_scale, float dt,
                          float* __restrict__ scal) {
    const double ss = warp_fold(part, nparts, 1);
    if (threadIdx.x != 0) return;
    const float s = (float)sqrt(ss / (double)n);
    const float scale = __fmul_rn(s, out_scale);
    scal[0] = s;
    scal[1] = s > 0.f ? __fdiv_rn(1.f, s) : 0.f;
    scal[2] = scale;
    scal[3] = scale > 0.f ? __fdiv_rn(dt, scale) : 0.f;
}

__global__ void k_input(const float* __restrict__ b, const uint8_t* __restrict__ flags, const float* __restrict__ scal,
                        i64 n, bf16* __restrict__ X0) {
    const float inv_s = scal[1];
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (i64)gridDim.x * blockDim.x) {
        const float c0 = __fmul_rn(b[v], inv_s);
        const float c1 = __fmul_rn((float)__popc(flags[v] & 63u), 1.0f / 6.0f);
        // (channels 8 to 15 are zero from the start)
        *reinterpret_cast<uint4*>(X0 + v * 16) = make_uint4(pack_bf16(c0, c1), 0u, 0u, 0u);
    }
}

// ---------------------------------------------------------------------------
// Pooling and upsampling (fine level dims D, H, W; coarse = half).

// The kernels below move 8 channels (16 bytes) per thread: blockIdx.y walks over
// the z planes, a plane's index is split with multiplications.  One channel
// per thread and 64-bit divisions took 54, 47 and 107 us (pooling at 128^3,
// the two backward forms at 96^3).
struct Vec8 {
    float v[8];
};
__device__ __forceinline__ Vec8 load8(const bf16* p) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    Vec8 r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        __nv_bfloat162 h;
        memcpy(&h, &w[k], 4);
        r.v[2 * k] = __bfloat162float(h.x);
        r.v[2 * k + 1] = __bfloat162float(h.y);
    }
    return r;
}
__device__ __forceinline__ void store8(bf16* p, const Vec8& a) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(a.v[0], a.v[1]), pack_bf16(a.v[2], a.v[3]),
                                              pack_bf16(a.v[4], a.v[5]), pack_bf16(a.v[6], a.v[7]));
}
// The sum of the 8 children of coarse voxel (z, y, x), in (dz, dy, dx) order;
// voxels of ct channels, the first at c.
__device__ __forceinline__ Vec8 sum_children(const bf16* __restrict__ in, int ct, int c, int H, int W, int z, int y, int x) {
    Vec8 s = {};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int fz = 2 * z + (k >> 2), fy = 2 * y + ((k >> 1) & 1), fx = 2 * x + (k & 1);
        const Vec8 a = load8(in + (((size_t)fz * H + fy) * W + fx) * ct + c);
#pragma unroll
        for (int j = 0; j < 8; ++j) s.v[j] = __fadd_rn(s.v[j], a.v[j]);
    }
    return s;
}

// out[u][c] = bf16(0.125 * sum of the 8 children)
__global__ void k_pool(const bf16* __restrict__ in, int C, int D, int H, int W, FastDiv fv, FastDiv fw,
                       bf16* __restrict__ out) {
    const int ch = H / 2, cw = W / 2, nv = C / 8;
    for (int z = blockIdx.y; z < D / 2; z += gridDim.y)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ch * cw * nv; i += gridDim.x * blockDim.x) {
            int c, x;
            const int y = split(split(i, nv, fv, c), cw, fw, x);
            Vec8 s = sum_children(in, C, 8 * c, H, W, z, y, x);
#pragma unroll
            for (int j = 0; j < 8; ++j) s.v[j] = __fmul_rn(0.125f, s.v[j]);
            store8(out + (((size_t)z * ch + y) * cw + x) * C + 8 * c, s);
        }
}

// dz[u][c] = y[u][c] > 0 ? bf16(sum_children dcat[child][c]) : 0, c < ca
__global__ void k_upback_gate(const bf16* __restrict__ dcat, int ct, int ca, const bf16* __restrict__ y, int D, int H,
                              int W, FastDiv fv, FastDiv fw, bf16* __restrict__ dz) {
    const int ch = H / 2, cw = W / 2, nv = ca / 8;
    for (int z = blockIdx.y; z < D / 2; z += gridDim.y)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ch * cw * nv; i += gridDim.x * blockDim.x) {
            int c, x;
            const int yy = split(split(i, nv, fv, c), cw, fw, x);
            const size_t o = (((size_t)z * ch + yy) * cw + x) * ca + 8 * c;
            const Vec8 g = load8(y + o);
            Vec8 s = sum_children(dcat, ct, 8 * c, H, W, z, yy, x);
#pragma unroll
            for (int j = 0; j < 8; ++j) s.v[j] = g.v[j] > 0.f ? s.v[j] : 0.f;
            store8(dz + o, s);
        }
}

// dz[v][c] = y[v][c] > 0 ? bf16(dcat[v][off + c] + 0.125 * dp[parent(v)][c]) : 0
__global__ void k_poolback_gate(const bf16* __restrict__ dcat, int ct, int off, const bf16* __restrict__ dp, int C,
                                const bf16* __restrict__ y, int D, int H, int W, FastDiv fv, FastDiv fw,
                                bf16* __restrict__ dz) {
    const int nv = C / 8;
    for (int z = blockIdx.y; z < D; z += gridDim.y)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < H * W * nv; i += gridDim.x * blockDim.x) {
            int c, x;
            const int yy = split(split(i, nv, fv, c), W, fw, x);
            const size_t v = ((size_t)z * H + yy) * W + x, u = ((size_t)(z / 2) * (H / 2) + yy / 2) * (W / 2) + x / 2;
            const Vec8 a = load8(dcat + v * ct + off + 8 * c), b = load8(dp + u * C + 8 * c), g = load8(y + v * C + 8 * c);
            Vec8 s;
#pragma unroll
            for (int j = 0; j < 8; ++j) s.v[j] = g.v[j] > 0.f ? __fadd_rn(a.v[j], __fmul_rn(0.125f, b.v[j])) : 0.f;
            store8(dz + v * C + 8 * c, s);
        }
}

// out[v] = [coarse[parent(v)] (ca channels) | skip[v] (cb channels)], 8-channel vectors
__global__ void k_upcat(const bf16* __restrict__ coarse, int ca, const bf16* __restrict__ skip, int cb, int D, int H,
                        int W, bf16* __restrict__ out) {
    const int ct = ca + cb, nv = ct / 8;
    const i64 n = (i64)D * H * W * nv;
    const int ch = H / 2, cw = W / 2;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const int k = (int)(i % nv);
        const i64 v = i / nv;
        const int x = (int)(v % W), y = (int)((v / W) % H), z = (int)(v / ((i64)W * H));
        uint4 val;
        if (k * 8 < ca) {
            const i64 u = ((i64)(z / 2) * ch + y / 2) * cw + x / 2;
            val = *reinterpret_cast<const uint4*>(coarse + u * ca + k * 8);
        } else {
            val = *reinterpret_cast<const uint4*>(skip + v * cb + (k * 8 - ca));
        }
        *reinterpret_cast<uint4*>(out + v * ct + k * 8) = val;
    }
}

// ---------------------------------------------------------------------------
// Output layer, guess and loss.
//   q = sum_c y9[c] * wh[c] (0 on solid cells); p_out = q * scale / dt.
//   Training, e = q - p_true * dt / scale on open cells (0 elsewhere):
//     loss kind MSE:    L = sum e^2 / cells,        g = e
//     loss kind energy: L = sum e (A1 e) / cells,   g = A1 e  (ae input)
//   (A1 = the masked Laplacian at dt = 1: the error's energy norm, the
//   quantity CG reduces; blind to the null-space constant.)
//   dq = g * c2 (c2 = 2 / cells), dZ9[c] = y9[c] > 0 ? dq * wh[c] : 0,
//   part[block] = {dwh[16], loss}.  With e_out set, only e is written.
constexpr int kHeadThreads = 256;

__global__ void __launch_bounds__(kHeadThreads)
    k_head(const bf16* __restrict__ Y9, const uint8_t* __restrict__ flags, const float* __restrict__ wh,
           const float* __restrict__ scal, i64 n, float dt, float* __restrict__ p_out, const float* __restrict__ p_true,
           float* __restrict__ e_out, const float* __restrict__ ae, float c2, bf16* __restrict__ dZ9,
           double* __restrict__ part) {
    __shared__ double sm[kHeadThreads];
    float w[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) w[c] = wh[c];
    const float scale = scal[2], inv_ps = scal[3];
    const bool train = p_true && !e_out;
    double dw[16], loss = 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c) dw[c] = 0.0;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (i64)gridDim.x * blockDim.x) {
        float y[16];
        const uint4* yp = reinterpret_cast<const uint4*>(Y9 + v * 16);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 u = yp[h];
            const uint32_t wds[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                __nv_bfloat162 pr;
                memcpy(&pr, &wds[k], 4);
                y[h * 8 + 2 * k] = __bfloat162float(pr.x);
                y[h * 8 + 2 * k + 1] = __bfloat162float(pr.y);
            }
        }
        float q = 0.f;
#pragma unroll
        for (int c = 0; c < 16; ++c) q = __fadd_rn(q, __fmul_rn(y[c], w[c]));
        const bool m = (flags[v] & 63u) != 0;
        if (!m) q = 0.f;
        if (p_out) p_out[v] = __fdiv_rn(__fmul_rn(q, scale), dt);
        if (!p_true) continue;
        const float e = m ? __fsub_rn(q, __fmul_rn(p_true[v], inv_ps)) : 0.f;
        if (e_out) {
            e_out[v] = e;
            continue;
        }
        const float gv = ae ? ae[v] : e;
        const float dq = m ? __fmul_rn(gv, c2) : 0.f;
        if (m) loss += (double)e * (double)gv;
        uint32_t o[8];
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            dw[c] += (double)y[c] * (double)dq;
            dw[c + 1] += (double)y[c + 1] * (double)dq;
            o[c / 2] = pack_bf16(y[c] > 0.f ? __fmul_rn(dq, w[c]) : 0.f, y[c + 1] > 0.f ? __fmul_rn(dq, w[c + 1]) : 0.f);
        }
        uint4* dp = reinterpret_cast<uint4*>(dZ9 + v * 16);
        dp[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dp[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
    if (!train) return;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const double s = block_sum<kHeadThreads>(dw[c], sm);
        if (threadIdx.x == 0) part[blockIdx.x * 17 + c] = s;
    }
    const double s = block_sum<kHeadThreads>(loss, sm);
    if (threadIdx.x == 0) part[blockIdx.x * 17 + 16] = s;
}

// Line search of the learned guess along d for A x = b with residual r:
// part[block] = {d . r, d . Ad}; then alpha = (d.r) / (d.Ad) (0 if d.Ad <= 0),
// x += alpha d, r -= alpha Ad.
__global__ void __launch_bounds__(kRedThreads) k_dots(const float* __restrict__ d, const float* __restrict__ r,
                                                      const float* __restrict__ ad, i64 n, double* __restrict__ part) {
    __shared__ double sm[2 * kRedThreads];
    double a = 0.0, b = 0.0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const double di = d[i];
        a += di * (double)r[i];
        b += di * (double)ad[i];
    }
    block_sum2<kRedThreads>(a, b, sm);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

__global__ void k_alpha(const double* __restrict__ part, int nb, float* __restrict__ alpha) {
    const double a = warp_fold(part, nb, 2), b = warp_fold(part + 1, nb, 2);
    if (threadIdx.x != 0) return;
    *alpha = (b > 0.0 && isfinite(a / b)) ? (float)(a / b) : 0.f;
}

__global__ void k_step(float* __restrict__ x, float* __restrict__ r, const float* __restrict__ d,
                       const float* __restrict__ ad, const float* __restrict__ alpha, i64 n) {
    const float a = *alpha;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        x[i] = __fadd_rn(x[i], __fmul_rn(a, d[i]));
        r[i] = __fsub_rn(r[i], __fmul_rn(a, ad[i]));
    }
}

// grad_wh[c] += sum_blocks part[c]; loss_out = sum part[16] / n; a warp each
__global__ void k_head_sum(const double* __restrict__ part, int nb, i64 n, float* __restrict__ grad_wh,
                           double* __restrict__ loss_out) {
    const int c = threadIdx.x >> 5;
    const double s = warp_fold(part + c, nb, 17);
    if (threadIdx.x & 31) return;
    if (c < 16)
        grad_wh[c] += (float)s;
    else
        *loss_out = s / (double)n;
}

// ---------------------------------------------------------------------------
__global__ void k_adam(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       i64 n, float lr, float b1, float b2, float eps, float gscale, float c1, float c2) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const float gi = g[i] * gscale;
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
        g[i] = 0.f;
    }
}

}  // namespace unet
}  // namespace pg

// ---------------------------------------------------------------------------
// Host side.

using namespace pg;
using namespace pg::unet;

static uint64_t next_net_id() {
    static std::atomic<uint64_t> n{0};
    return ++n;
}

struct pg_unet {
    uint64_t id = next_net_id();  // never given out again
    int device = 0, num_sms = 0;
    int ld[3], lh[3], lw[3];
    i64 lv[3];
    cudaStream_t stream = nullptr;
    void* arena = nullptr;
    void* cat = nullptr;  // C0 and C1: the mma.sync path's
    float* params = nullptr;
    float* grads = nullptr;
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    uint2* wf[kL] = {};
    uint2* wt[kL] = {};
    bf16* tcf[kL] = {};  // tensor-core (tcgen05) weight layouts: forward
    bf16* tct[kL] = {};  // and backward-data
    int* err = nullptr;  // set by a kernel whose bounded wait gave up
    bool wdirty = true, wdirty_mma = true;  // the layouts' weights are older than the parameters
    bf16 *X0 = nullptr, *Y[kL] = {}, *P0 = nullptr, *P1 = nullptr, *C1 = nullptr, *C0 = nullptr;
    bf16 *G0a = nullptr, *G0b = nullptr, *dC0 = nullptr, *G1a = nullptr, *G1b = nullptr, *dC1 = nullptr,
         *dP0 = nullptr, *G2a = nullptr, *G2b = nullptr, *dP1 = nullptr;
    float* q = nullptr;    // guess scratch (V0)
    float* r = nullptr;    // residual scratch (V0)
    float* ad = nullptr;   // A d scratch (V0)
    int loss_kind = 1;     // 0 MSE, 1 energy norm
    float* scal = nullptr;  // 4 floats
    double* red = nullptr;  // reduction partials
    double* loss = nullptr;
    float* wpart[kL] = {};  // weight-gradient partials
    double out_scale = 1.0;
    i64 adam_t = 0;
};

namespace {

int ceil_div(i64 a, i64 b) { return (int)((a + b - 1) / b); }
int pow2_floor(int x) {
    int p = 1;
    while (p * 2 <= x) p *= 2;
    return p;
}

// Grid of the plane-walking kernels: d planes of n threads.
dim3 plane_grid(i64 n, int d) { return dim3((unsigned)((n + 255) / 256), (unsigned)std::min(d, 65535)); }

int blocks_for(const pg_unet* net, i64 n, int threads = 256) {
    i64 b = (n + threads - 1) / threads;
    return (int)std::max<i64>(1, std::min<i64>(b, (i64)net->num_sms * 16));
}

ConvGeom conv_geom(int D, int H, int W, int mt) {
    ConvGeom G;
    G.D = D;
    G.H = H;
    G.W = W;
    const int nv = 128 * mt;
    G.TX = std::min(32, pow2_floor(W));
    G.TY = std::min(4, pow2_floor(H));
    G.TZ = nv / (G.TX * G.TY);
    G.BX = G.TX + 2;
    G.BY = G.TY + 2;
    G.tiles_x = ceil_div(W, G.TX);
    G.tiles_y = ceil_div(H, G.TY);
    return G;
}

template <int CIN, int COUT>
int conv_t(const pg_unet* net, int lvl, const bf16* in, const uint2* w, bf16* out, const bf16* gate, int epi) {
    constexpr int MT = COUT <= 32 ? 4 : (COUT <= 64 ? 2 : 1);
    const ConvGeom G = conv_geom(net->ld[lvl], net->lh[lvl], net->lw[lvl], MT);
    const size_t smem = (size_t)G.BX * G.BY * (G.TZ + 2) * kRowBytes;
    if (const int rc = opt_in<k_conv<CIN, COUT, MT>>(96 * 1024)) return rc;
    if (smem > 96 * 1024) return bad_arg("pg_unet: conv tile does not fit in shared memory");
    const int nb = G.tiles_x * G.tiles_y * ceil_div(G.D, G.TZ);
    PG_LAUNCH(KK_UNET_CONV, net->stream, k_conv<CIN, COUT, MT><<<nb, kConvThreads, smem, net->stream>>>(in, w, out, gate, G, epi));
    PG_CHECK_LAUNCH();
    return PG_OK;
}

// The tensor-core convolution: CTAs that walk over the 8 x 16 x TZ output
// tiles; the launch's dynamic shared memory also caps the CTAs per SM so that
// their tensor-memory columns fit in the SM's 512.
template <int CIN, int COUT, int TZ, int CA>
int conv_tc_z(const pg_unet* net, int lvl, const bf16* in, const bf16* up, const bf16* wtc, bf16* out, const bf16* gate,
              int epi) {
    typedef tc::Cfg<CIN, COUT, TZ> Cf;
    const auto kernel = tc::k_conv_tc<CIN, COUT, TZ, CA>;
    struct Shape {
        size_t smem = Cf::kSmem + 256;
        int per_sm = 0;
    } shape;
    static PerDevice<Shape> known;
    PG_CUDA(known.get(
        [&](Shape* r) {
            const int maxb = 512 / Cf::kCols;
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r->per_sm, kernel, tc::kThreads, r->smem);
            if (!e && r->per_sm > maxb) {
                r->smem = std::max(r->smem, (size_t)(228 * 1024 / (maxb + 1) - 1024 + 128));
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r->per_sm, kernel, tc::kThreads, r->smem);
            }
            if (r->per_sm > maxb) r->per_sm = 0;
            return e;
        },
        &shape));
    if (shape.per_sm < 1) return bad_arg("pg_unet: tensor-core conv does not fit an SM");
    tc::Geom G;
    G.D = net->ld[lvl];
    G.H = net->lh[lvl];
    G.W = net->lw[lvl];
    G.tiles_x = ceil_div(G.W, tc::TX);
    G.tiles_y = ceil_div(G.H, tc::TY);
    G.tiles = G.tiles_x * G.tiles_y * ceil_div(G.D, TZ);
    CUtensorMap vox;
    if (!encode_map_voxels_bf16(&vox, in, CIN - CA, G.W, G.H, G.D, tc::BX, tc::BY, Cf::BZ)) {
        set_error("pg_unet: no tensor map for a layer's input");
        return PG_CUDA_ERROR;
    }
    const int nb = std::min(G.tiles, shape.per_sm * net->num_sms);
    PG_LAUNCH(KK_UNET_CONV, net->stream,
              kernel<<<nb, tc::kThreads, shape.smem, net->stream>>>(vox, up, wtc, out, gate, G, epi, net->err));
    PG_CHECK_LAUNCH();
    return PG_OK;
}

// Planes per tile: four (two for 96 channels, whose weights fill shared
// memory); two where tiles of four leave SMs without work.
template <int CIN, int COUT, int CA = 0>
int conv_tc_t(const pg_unet* net, int lvl, const bf16* in, const bf16* wtc, bf16* out, const bf16* gate, int epi,
              const bf16* up = nullptr) {
    constexpr int TZ = COUT >= 96 ? 2 : 4;
    const int tiles = ceil_div(net->lw[lvl], tc::TX) * ceil_div(net->lh[lvl], tc::TY) * ceil_div(net->ld[lvl], TZ);
    if (TZ == 4 && tiles < net->num_sms) return conv_tc_z<CIN, COUT, 2, CA>(net, lvl, in, up, wtc, out, gate, epi);
    return conv_tc_z<CIN, COUT, TZ, CA>(net, lvl, in, up, wtc, out, gate, epi);
}

// The tensor-core path unless PG_UNET_TC=0 (a diagnostic switch: the legacy
// warp-level mma.sync kernel, kept for comparison).
bool tc_enabled() {
    const char* env = getenv("PG_UNET_TC");
    return !(env && env[0] == '0');
}

int conv(const pg_unet* net, int lvl, int cin, int cout, const bf16* in, const uint2* w, const bf16* wtc, bf16* out,
         const bf16* gate, int epi) {
    if (tc_enabled()) {
#define PG_UNET_CONV_TC(A, B) \
    if (cin == A && cout == B) return conv_tc_t<A, B>(net, lvl, in, wtc, out, gate, epi);
        PG_UNET_CONV_TC(16, 16)
        PG_UNET_CONV_TC(16, 32)
        PG_UNET_CONV_TC(32, 32)
        PG_UNET_CONV_TC(32, 64)
        PG_UNET_CONV_TC(64, 64)
        PG_UNET_CONV_TC(96, 32)
        PG_UNET_CONV_TC(48, 16)
        PG_UNET_CONV_TC(16, 48)
        PG_UNET_CONV_TC(32, 96)
        PG_UNET_CONV_TC(64, 32)
        PG_UNET_CONV_TC(32, 16)
#undef PG_UNET_CONV_TC
        return bad_arg("pg_unet: no conv kernel for this channel pair");
    }
#define PG_UNET_CONV(A, B) \
    if (cin == A && cout == B) return conv_t<A, B>(net, lvl, in, w, out, gate, epi);
    PG_UNET_CONV(16, 16)
    PG_UNET_CONV(16, 32)
    PG_UNET_CONV(32, 32)
    PG_UNET_CONV(32, 64)
    PG_UNET_CONV(64, 64)
    PG_UNET_CONV(96, 32)
    PG_UNET_CONV(48, 16)
    PG_UNET_CONV(16, 48)
    PG_UNET_CONV(32, 96)
    PG_UNET_CONV(64, 32)
    PG_UNET_CONV(32, 16)
#undef PG_UNET_CONV
    return bad_arg("pg_unet: no conv kernel for this channel pair");
}

int wg_tiles(const pg_unet* net, int lvl) {
    return ceil_div(net->lw[lvl], kWgX) * ceil_div(net->lh[lvl], kWgY) * ceil_div(net->ld[lvl], kWgZ);
}
// CTAs (partial sums) per channel block of layer k's weight gradient.
int wg_ctas(const pg_unet* net, int k) {
    const int blocks = 3 * (kCin[k] / 16) * (kCout[k] / wg_co(kCout[k]));
    return std::max(1, std::min(wg_tiles(net, kLevel[k]), wg_ctas_per_sm(kCin[k]) * net->num_sms / blocks));
}

template <int CO> int wgrad_t(pg_unet* net, int k, const bf16* X, const bf16* up, const bf16* dZ) {
    if (const int rc = opt_in<k_wgrad<CO>>(2 * wg_stage(CO))) return rc;
    const int lvl = kLevel[k], S = wg_ctas(net, k);
    WgGeom G;
    G.D = net->ld[lvl];
    G.H = net->lh[lvl];
    G.W = net->lw[lvl];
    G.cin = kCin[k];
    G.cout = kCout[k];
    G.ca = up ? kCin[k] - kCout[kSkip[k]] : 0;
    G.tiles_x = ceil_div(G.W, kWgX);
    G.tiles_y = ceil_div(G.H, kWgY);
    G.tiles = wg_tiles(net, lvl);
    const dim3 grid(S, 3 * (kCin[k] / 16) * (kCout[k] / CO));
    PG_LAUNCH(KK_UNET_WGRAD, net->stream, k_wgrad<CO><<<grid, kWgThreads, 2 * wg_stage(CO), net->stream>>>(X, up, dZ, net->wpart[k], G));
    PG_CHECK_LAUNCH();
    return PG_OK;
}

// The partials of layer k's weight gradient; X, and up with a decoder's
// concatenation [up | X].
int wgrad(pg_unet* net, int k, const bf16* X, const bf16* dZ, const bf16* up = nullptr) {
    return wg_co(kCout[k]) == 16 ? wgrad_t<16>(net, k, X, up, dZ) : wgrad_t<32>(net, k, X, up, dZ);
}

// Every layer's partials folded into its gradient.
int wgrad_sums(pg_unet* net) {
    WgSumArgs A;
    int blocks = 0;
    for (int k = 0; k < kL; ++k) {
        A.part[k] = net->wpart[k];
        A.grad[k] = net->grads + param_offset(k);
        A.S[k] = wg_ctas(net, k);
        A.n[k] = 27 * kCin[k] * kCout[k];
        A.block0[k] = blocks;
        blocks += A.n[k] / 32;
    }
    PG_LAUNCH(KK_UNET_WGRAD, net->stream, k_wgrad_sum<<<blocks, 256, 0, net->stream>>>(A));
    PG_CHECK_LAUNCH();
    return PG_OK;
}

int prep_weights(pg_unet* net) {
    if (tc_enabled() ? !net->wdirty : !net->wdirty_mma) return PG_OK;
    if (tc_enabled()) {
        tc::PrepArgs A = {};
        int most = 0;
        for (int k = 0; k < kL; ++k) {
            A.cin[k] = kCin[k];
            A.cout[k] = kCout[k];
            A.W[2 * k] = A.W[2 * k + 1] = net->params + param_offset(k);
            A.wtc[2 * k] = net->tcf[k];
            A.wtc[2 * k + 1] = k ? net->tct[k] : nullptr;
            most = std::max(most, 27 * kCin[k] * kCout[k]);
        }
        PG_LAUNCH(KK_UNET_MISC, net->stream,
                  tc::k_wprep_tc<<<dim3(ceil_div(most, 1024), 2 * kL), 256, 0, net->stream>>>(A));
        PG_CHECK_LAUNCH();
        net->wdirty = false;
        return PG_OK;
    }
    for (int k = 0; k < kL; ++k) {
        const int n = 27 * kCin[k] * kCout[k] / 2;  // both layouts: 2 x (27 * cin/16 * cout/8 * 32)
        PG_LAUNCH(KK_UNET_MISC, net->stream,
                  k_wprep<<<ceil_div(n, 256), 256, 0, net->stream>>>(net->params + param_offset(k), kCin[k], kCout[k],
                                                                      net->wf[k], k ? net->wt[k] : nullptr));
    }
    PG_CHECK_LAUNCH();
    net->wdirty_mma = false;
    return PG_OK;
}

// PG_TIMEOUT (and the flag cleared) when a tensor-core wait gave up since
// the last check; synchronous.
int check_err(pg_unet* net) {
    int e = 0;
    PG_CUDA(cudaMemcpy(&e, net->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (!e) return PG_OK;
    PG_CUDA(cudaMemset(net->err, 0, sizeof(int)));
    set_error("pg_unet: a wait for the tensor cores gave up; the network's last results are not to be trusted");
    return PG_TIMEOUT;
}

int check_grid(const pg_unet* net, const pg_grid* g) {
    if (!g) return bad_arg("pg_unet: NULL grid");
    if (g->dims.nd != 3 || g->dims.d != net->ld[0] || g->dims.h != net->lh[0] || g->dims.w != net->lw[0])
        return bad_arg("pg_unet: grid shape differs from the network's");
    return PG_OK;
}

// Normalise b, run the encoder/decoder; Y[9] holds the last features.  The
// decoder's convolutions and weight gradients read their two inputs where
// they are; only the mma.sync convolutions need them written side by side
// (k_upcat: 99 us at 128^3).
int forward(pg_unet* net, const pg_grid* g, const float* b, double dt) {
    int rc;
    const bool cat = !tc_enabled();
    if ((rc = prep_weights(net))) return rc;
    if (cat && !net->cat) {
        const size_t n0 = 48 * (size_t)net->lv[0], n1 = 96 * (size_t)net->lv[1];
        PG_CUDA(cudaMalloc(&net->cat, sizeof(bf16) * (n0 + n1)));
        net->C0 = (bf16*)net->cat;
        net->C1 = net->C0 + n0;
    }
    const i64 V0 = net->lv[0];
    cudaStream_t s = net->stream;
    PG_LAUNCH(KK_UNET_MISC, s, k_sumsq<<<kRedBlocks, kRedThreads, 0, s>>>(b, V0, net->red));
    PG_LAUNCH(KK_UNET_MISC, s, k_scalars<<<1, 32, 0, s>>>(net->red, kRedBlocks, V0, (float)net->out_scale, (float)dt, net->scal));
    PG_LAUNCH(KK_UNET_MISC, s, k_input<<<blocks_for(net, V0), 256, 0, s>>>(b, g->flags, net->scal, V0, net->X0));
    PG_CHECK_LAUNCH();
    auto C = [&](int k, const bf16* in) {
        return conv(net, kLevel[k], kCin[k], kCout[k], in, net->wf[k], net->tcf[k], net->Y[k], nullptr, EPI_RELU);
    };
    if ((rc = C(0, net->X0)) || (rc = C(1, net->Y[0]))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_pool<<<plane_grid((i64)net->lh[1] * net->lw[1] * 2, net->ld[1]), 256, 0, s>>>(net->Y[1], 16, net->ld[0], net->lh[0], net->lw[0], fast_div(2), fast_div(net->lw[1]), net->P0));
    if ((rc = C(2, net->P0)) || (rc = C(3, net->Y[2]))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_pool<<<plane_grid((i64)net->lh[2] * net->lw[2] * 4, net->ld[2]), 256, 0, s>>>(net->Y[3], 32, net->ld[1], net->lh[1], net->lw[1], fast_div(4), fast_div(net->lw[2]), net->P1));
    if ((rc = C(4, net->P1)) || (rc = C(5, net->Y[4]))) return rc;
    if (cat) {
        PG_LAUNCH(KK_UNET_MISC, s, k_upcat<<<blocks_for(net, net->lv[1] * 12), 256, 0, s>>>(net->Y[5], 64, net->Y[3], 32, net->ld[1], net->lh[1], net->lw[1], net->C1));
        rc = C(6, net->C1);
    } else {
        rc = conv_tc_t<96, 32, 64>(net, 1, net->Y[3], net->tcf[6], net->Y[6], nullptr, EPI_RELU, net->Y[5]);
    }
    if (rc || (rc = C(7, net->Y[6]))) return rc;
    if (cat) {
        PG_LAUNCH(KK_UNET_MISC, s, k_upcat<<<blocks_for(net, net->lv[0] * 6), 256, 0, s>>>(net->Y[7], 32, net->Y[1], 16, net->ld[0], net->lh[0], net->lw[0], net->C0));
        rc = C(8, net->C0);
    } else {
        rc = conv_tc_t<48, 16, 32>(net, 0, net->Y[1], net->tcf[8], net->Y[8], nullptr, EPI_RELU, net->Y[7]);
    }
    if (rc || (rc = C(9, net->Y[8]))) return rc;
    PG_CHECK_LAUNCH();
    return PG_OK;
}

int backward(pg_unet* net) {
    int rc;
    cudaStream_t s = net->stream;
    const int d0 = net->ld[0], h0 = net->lh[0], w0 = net->lw[0];
    const int d1 = net->ld[1], h1 = net->lh[1], w1 = net->lw[1];
    auto BD = [&](int k, const bf16* dz, bf16* out, const bf16* gate, int epi) {
        return conv(net, kLevel[k], kCout[k], kCin[k], dz, net->wt[k], net->tct[k], out, gate, epi);
    };
    // level 0 decoder: dZ9 = G0a (from k_head)
    if ((rc = wgrad(net, 9, net->Y[8], net->G0a)) || (rc = BD(9, net->G0a, net->G0b, net->Y[8], EPI_GATE))) return rc;
    if ((rc = wgrad(net, 8, net->Y[1], net->G0b, net->Y[7])) || (rc = BD(8, net->G0b, net->dC0, nullptr, EPI_NONE))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_upback_gate<<<plane_grid((i64)h1 * w1 * 4, d1), 256, 0, s>>>(net->dC0, 48, 32, net->Y[7], d0, h0, w0, fast_div(4), fast_div(w1), net->G1a));
    // level 1 decoder
    if ((rc = wgrad(net, 7, net->Y[6], net->G1a)) || (rc = BD(7, net->G1a, net->G1b, net->Y[6], EPI_GATE))) return rc;
    if ((rc = wgrad(net, 6, net->Y[3], net->G1b, net->Y[5])) || (rc = BD(6, net->G1b, net->dC1, nullptr, EPI_NONE))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_upback_gate<<<plane_grid((i64)net->lh[2] * net->lw[2] * 8, net->ld[2]), 256, 0, s>>>(net->dC1, 96, 64, net->Y[5], d1, h1, w1, fast_div(8), fast_div(net->lw[2]), net->G2a));
    // level 2
    if ((rc = wgrad(net, 5, net->Y[4], net->G2a)) || (rc = BD(5, net->G2a, net->G2b, net->Y[4], EPI_GATE))) return rc;
    if ((rc = wgrad(net, 4, net->P1, net->G2b)) || (rc = BD(4, net->G2b, net->dP1, nullptr, EPI_NONE))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_poolback_gate<<<plane_grid((i64)h1 * w1 * 4, d1), 256, 0, s>>>(net->dC1, 96, 64, net->dP1, 32, net->Y[3], d1, h1, w1, fast_div(4), fast_div(w1), net->G1a));
    // level 1 encoder
    if ((rc = wgrad(net, 3, net->Y[2], net->G1a)) || (rc = BD(3, net->G1a, net->G1b, net->Y[2], EPI_GATE))) return rc;
    if ((rc = wgrad(net, 2, net->P0, net->G1b)) || (rc = BD(2, net->G1b, net->dP0, nullptr, EPI_NONE))) return rc;
    PG_LAUNCH(KK_UNET_MISC, s, k_poolback_gate<<<plane_grid((i64)h0 * w0 * 2, d0), 256, 0, s>>>(net->dC0, 48, 32, net->dP0, 16, net->Y[1], d0, h0, w0, fast_div(2), fast_div(w0), net->G0a));
    // level 0 encoder
    if ((rc = wgrad(net, 1, net->Y[0], net->G0a)) || (rc = BD(1, net->G0a, net->G0b, net->Y[0], EPI_GATE))) return rc;
    if ((rc = wgrad(net, 0, net->X0, net->G0b)) || (rc = wgrad_sums(net))) return rc;
    PG_CHECK_LAUNCH();
    return PG_OK;
}

// Blocks of the training form: its FP64 sums are the bound, so every SM gets as many.
int head_blocks(const pg_unet* net) { return 4 * net->num_sms; }

// out = A in on the network's stream (A = dt * the grid's masked Laplacian).
int apply_a(pg_unet* net, const pg_grid* g, float* out, const float* in, double dt) {
    pg_grid* gm = const_cast<pg_grid*>(g);
    cudaStream_t saved = gm->stream;
    gm->stream = net->stream;
    const int rc = launch_laplacian<float>(gm, out, in, dt);
    gm->stream = saved;
    return rc;
}

int head(pg_unet* net, const pg_grid* g, double dt, float* p_out, const float* p_true) {
    const i64 V0 = net->lv[0];
    const float c2 = 2.0f / (float)V0;
    cudaStream_t s = net->stream;
    const int nb = (int)std::min<i64>(head_blocks(net), std::max<i64>(1, (V0 + kHeadThreads - 1) / kHeadThreads));
    const int nw = blocks_for(net, V0, kHeadThreads);  // without sums
    const float* wh = net->params + param_offset(kL);
    const float* ae = nullptr;
    if (p_true && net->loss_kind == 1) {
        // e = q - t, then A1 e (dt = 1) into the scratch ad
        PG_LAUNCH(KK_UNET_MISC, s, k_head<<<nw, kHeadThreads, 0, s>>>(net->Y[9], g->flags, wh, net->scal, V0, (float)dt, nullptr, p_true, net->r, nullptr, c2, net->G0a, net->red));
        int rc;
        if ((rc = apply_a(net, g, net->ad, net->r, 1.0))) return rc;
        ae = net->ad;
    }
    PG_LAUNCH(KK_UNET_MISC, s, k_head<<<p_true ? nb : nw, kHeadThreads, 0, s>>>(net->Y[9], g->flags, wh, net->scal, V0, (float)dt, p_out, p_true, nullptr, ae, c2, net->G0a, net->red));
    if (p_true)
        PG_LAUNCH(KK_UNET_MISC, s, k_head_sum<<<1, 17 * 32, 0, s>>>(net->red, nb, V0, net->grads + param_offset(kL), net->loss));
    PG_CHECK_LAUNCH();
    return PG_OK;
}

// ---------------------------------------------------------------------------
// The network as a preconditioner correction inside the CG.  For a residual
// r: q = net(r), a = (q.r) / (q.Aq) (0 when q.Aq <= 0; the step along q that
// minimises the error's energy norm), then one Jacobi step on what that
// leaves:
//     z = M(r) = a q + D^-1 (r - a A q).
// M is not linear in r (a and the network depend on r), so the CG is the
// flexible one: beta is the Polak-Ribiere ratio z'.(r' - r) / (z.r), which
// with r' - r = -alpha A p is -alpha (z'.Ap) / (z.r) -- read from the A p
// vector the iteration just used, with no copy of the previous residual.

__global__ void k_lp_z(float* __restrict__ z, const float* __restrict__ r, const float* __restrict__ q,
                       const float* __restrict__ aq, const uint8_t* __restrict__ flags, const float* __restrict__ alpha,
                       i64 n, float dt, const CgState* st) {
    if (st->done) return;
    const float a = *alpha;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (i64)gridDim.x * blockDim.x) {
        const int open = __popc((unsigned)flags[v] & 63u);
        const float inv = open ? __frcp_rn((float)open * dt) : 0.f;
        z[v] = fmaf(a, q[v], (r[v] - a * aq[v]) * inv);
    }
}

// z.r and z.Ap (compensated FP32 per thread, FP64 across), then the last
// block folds them into the CG state: sigma = z.r; after the first
// iteration beta = -alpha (z.Ap) / sigma_old.
__global__ void __launch_bounds__(kRedThreads)
    k_lp_fold(const float* __restrict__ z, const float* __restrict__ r, const float* __restrict__ ap, i64 n,
              CgState* st, double* partials) {
    if (st->done) return;
    __shared__ double sm[2 * kRedThreads];
    Acc<float> zr, zap;
    const bool first = st->iter == 0;
    for (i64 v = (i64)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (i64)gridDim.x * blockDim.x) {
        const float zv = z[v];
        zr.add(zv * r[v]);
        if (!first) zap.add(zv * ap[v]);
    }
    double s1 = zr.value(), s2 = zap.value();
    block_sum2<kRedThreads>(s1, s2, sm);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s1;
        partials[kMaxBlocks + blockIdx.x] = s2;
    }
    if (!last_block(&st->counter[3])) return;
    double rz, za;
    reduce_partials2<kRedThreads>(partials, partials + kMaxBlocks, gridDim.x, sm, rz, za);
    if (threadIdx.x == 0) {
        st->counter[3] = 0;
        if (!isfinite(rz) || !isfinite(za)) {
            st->status = PG_NAN_DETECTED;
            st->done = 1;
        } else if (!(rz > 0.0)) {  // M(r) is not a descent direction for r
            st->status = PG_BREAKDOWN;
            st->done = 1;
        } else if (first) {
            st->sigma = rz;
        } else {
            st->beta = -st->alpha * za / st->sigma;
            st->sigma = rz;
            st->first = 0;
        }
    }
}

struct LearnedHook : ZHook {
    pg_unet* net = nullptr;
    double dt = 1.0;
    const float* ap = nullptr;
    void bind(const void* p) override { ap = (const float*)p; }
    // The network by a number of its own (another may come to lie at its
    // address), and the convolutions' path: each reads weights of its own layout.
    // (The top bit: a multigrid hierarchy's number never has it.)
    uintptr_t key() const override { return (uintptr_t)1 << 63 | (uintptr_t)net->id << 1 | (uintptr_t)tc_enabled(); }
    int apply(pg_grid* g, const void* rv, void* zv) override {
        const float* r = (const float*)rv;
        float* z = (float*)zv;
        const i64 V0 = net->lv[0];
        // the network's kernels run on the CG's stream (a graph capture's)
        cudaStream_t saved = net->stream;
        net->stream = g->stream;
        cudaStream_t s = g->stream;
        float* alpha = net->scal + 5;
        int rc = forward(net, g, r, dt);
        if (!rc) rc = head(net, g, dt, net->q, nullptr);
        if (!rc) rc = apply_a(net, g, net->ad, net->q, dt);
        if (!rc) {
            PG_LAUNCH(KK_UNET_MISC, s, k_dots<<<kRedBlocks, kRedThreads, 0, s>>>(net->q, r, net->ad, V0, net->red));
            PG_LAUNCH(KK_UNET_MISC, s, k_alpha<<<1, 32, 0, s>>>(net->red, kRedBlocks, alpha));
            PG_LAUNCH(KK_UNET_MISC, s,
                      k_lp_z<<<blocks_for(net, V0), 256, 0, s>>>(z, r, net->q, net->ad, g->flags, alpha, V0,
                                                                 (float)dt, g->ws.state));
            const int nb = (int)std::min<i64>(kRedBlocks, std::max<i64>(1, (V0 + kRedThreads - 1) / kRedThreads));
            PG_LAUNCH(KK_UNET_MISC, s,
                      k_lp_fold<<<nb, kRedThreads, 0, s>>>(z, r, ap, V0, g->ws.state, g->ws.partials));
            const cudaError_t e = cudaPeekAtLastError();
            if (e != cudaSuccess) rc = cuda_fail(e, "learned preconditioner launch");
        }
        net->stream = saved;
        return rc;
    }
};

}  // namespace

extern "C" {

int64_t pg_unet_num_params(void) { return num_params(); }

int pg_unet_create(int64_t d, int64_t h, int64_t w, pg_unet** out) {
    if (!out) return bad_arg("pg_unet_create: NULL out");
    *out = nullptr;
    if (d < 16 || h < 16 || w < 16 || d % 4 || h % 4 || w % 4)
        return bad_arg("pg_unet_create: every side must be a multiple of 4 and >= 16");
    if (d * h * w * 48 >= ((int64_t)1 << 31)) return bad_arg("pg_unet_create: grid too large");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        set_error("pg_unet_create: no CUDA device");
        return PG_NO_DEVICE;
    }
    pg_unet* net = new (std::nothrow) pg_unet();
    if (!net) return PG_OUT_OF_MEMORY;
    PG_CUDA(cudaGetDevice(&net->device));
    PG_CUDA(cudaDeviceGetAttribute(&net->num_sms, cudaDevAttrMultiProcessorCount, net->device));
    for (int l = 0; l < 3; ++l) {
        net->ld[l] = (int)(d >> l);
        net->lh[l] = (int)(h >> l);
        net->lw[l] = (int)(w >> l);
        net->lv[l] = (i64)net->ld[l] * net->lh[l] * net->lw[l];
    }
    const i64 P = num_params();
    // Arena layout (256-byte aligned pieces).
    std::vector<std::pair<void**, size_t>> parts;
    auto add = [&](void** p, size_t bytes) { parts.push_back({p, (bytes + 255) & ~(size_t)255}); };
    add((void**)&net->params, 4 * P);
    add((void**)&net->grads, 4 * P);
    add((void**)&net->adam_m, 4 * P);
    add((void**)&net->adam_v, 4 * P);
    for (int k = 0; k < kL; ++k) {
        add((void**)&net->wf[k], 8 * (size_t)27 * kCin[k] * kCout[k] / 4);
        if (k) add((void**)&net->wt[k], 8 * (size_t)27 * kCin[k] * kCout[k] / 4);
        add((void**)&net->tcf[k], 2 * (size_t)27 * kCin[k] * kCout[k]);
        if (k) add((void**)&net->tct[k], 2 * (size_t)27 * kCin[k] * kCout[k]);
    }
    add((void**)&net->err, sizeof(int));
    const i64 V0 = net->lv[0], V1 = net->lv[1], V2 = net->lv[2];
    add((void**)&net->X0, 2 * V0 * 16);
    for (int k = 0; k < kL; ++k) add((void**)&net->Y[k], 2 * (size_t)net->lv[kLevel[k]] * kCout[k]);
    add((void**)&net->P0, 2 * V1 * 16);
    add((void**)&net->P1, 2 * V2 * 32);
    add((void**)&net->G0a, 2 * V0 * 16);
    add((void**)&net->G0b, 2 * V0 * 16);
    add((void**)&net->dC0, 2 * V0 * 48);
    add((void**)&net->G1a, 2 * V1 * 32);
    add((void**)&net->G1b, 2 * V1 * 32);
    add((void**)&net->dC1, 2 * V1 * 96);
    add((void**)&net->dP0, 2 * V1 * 16);
    add((void**)&net->G2a, 2 * V2 * 64);
    add((void**)&net->G2b, 2 * V2 * 64);
    add((void**)&net->dP1, 2 * V2 * 32);
    add((void**)&net->q, 4 * V0);
    add((void**)&net->r, 4 * V0);
    add((void**)&net->ad, 4 * V0);
    add((void**)&net->scal, 32);
    add((void**)&net->red, 8 * std::max(2 * kRedBlocks, head_blocks(net) * 17));
    add((void**)&net->loss, 8);
    for (int k = 0; k < kL; ++k) add((void**)&net->wpart[k], 4 * (size_t)wg_ctas(net, k) * 27 * kCin[k] * kCout[k]);
    size_t total = 0;
    for (auto& p : parts) total += p.second;
    cudaError_t e = cudaMalloc(&net->arena, total);
    if (e != cudaSuccess) {
        delete net;
        return cuda_fail(e, "pg_unet_create: cudaMalloc");
    }
    char* base = (char*)net->arena;
    for (auto& p : parts) {
        *p.first = base;
        base += p.second;
    }
    PG_CUDA(cudaMemset(net->arena, 0, total));
    *out = net;
    return PG_OK;
}

int pg_unet_destroy(pg_unet* net) {
    if (!net) return PG_OK;
    cudaFree(net->cat);
    if (net->arena) cudaFree(net->arena);
    delete net;
    return PG_OK;
}

int pg_unet_set_stream(pg_unet* net, void* stream) {
    if (!net) return bad_arg("pg_unet_set_stream: NULL net");
    net->stream = (cudaStream_t)stream;
    return PG_OK;
}

int pg_unet_set_params(pg_unet* net, const float* host, double out_scale) {
    if (!net || !host) return bad_arg("pg_unet_set_params: NULL argument");
    if (!(out_scale > 0.0) || !std::isfinite(out_scale)) return bad_arg("pg_unet_set_params: out_scale must be > 0");
    const i64 P = num_params();
    PG_CUDA(cudaMemcpyAsync(net->params, host, 4 * P, cudaMemcpyHostToDevice, net->stream));
    PG_CUDA(cudaMemsetAsync(net->grads, 0, 4 * P, net->stream));
    PG_CUDA(cudaMemsetAsync(net->adam_m, 0, 4 * P, net->stream));
    PG_CUDA(cudaMemsetAsync(net->adam_v, 0, 4 * P, net->stream));
    PG_CUDA(cudaStreamSynchronize(net->stream));
    net->out_scale = out_scale;
    net->adam_t = 0;
    net->wdirty = net->wdirty_mma = true;
    return PG_OK;
}

int pg_unet_get_params(const pg_unet* net, float* host, double* out_scale) {
    if (!net) return bad_arg("pg_unet_get_params: NULL net");
    if (host) {
        PG_CUDA(cudaMemcpyAsync(host, net->params, 4 * num_params(), cudaMemcpyDeviceToHost, net->stream));
        PG_CUDA(cudaStreamSynchronize(net->stream));
    }
    if (out_scale) *out_scale = net->out_scale;
    return PG_OK;
}

int pg_unet_get_grads(const pg_unet* net, float* host) {
    if (!net || !host) return bad_arg("pg_unet_get_grads: NULL argument");
    PG_CUDA(cudaMemcpyAsync(host, net->grads, 4 * num_params(), cudaMemcpyDeviceToHost, net->stream));
    PG_CUDA(cudaStreamSynchronize(net->stream));
    return PG_OK;
}

int pg_unet_zero_grads(pg_unet* net) {
    if (!net) return bad_arg("pg_unet_zero_grads: NULL net");
    PG_CUDA(cudaMemsetAsync(net->grads, 0, 4 * num_params(), net->stream));
    return PG_OK;
}

int pg_unet_accumulate_f32(pg_unet* net, const pg_grid* g, const float* b, const float* p_true, double dt,
                           double* loss) {
    if (!net || !b || !p_true) return bad_arg("pg_unet_accumulate_f32: NULL argument");
    if (!(dt > 0.0)) return bad_arg("pg_unet_accumulate_f32: dt must be > 0");
    int rc;
    if ((rc = check_grid(net, g))) return rc;
    if ((rc = forward(net, g, b, dt)) || (rc = head(net, g, dt, nullptr, p_true)) || (rc = backward(net))) return rc;
    if (loss) {
        PG_CUDA(cudaMemcpyAsync(loss, net->loss, sizeof(double), cudaMemcpyDeviceToHost, net->stream));
        PG_CUDA(cudaStreamSynchronize(net->stream));
        return check_err(net);
    }
    return PG_OK;
}

int pg_unet_check(pg_unet* net) {
    if (!net) return bad_arg("pg_unet_check: NULL network");
    PG_CUDA(cudaStreamSynchronize(net->stream));
    return check_err(net);
}

int pg_unet_adam_step(pg_unet* net, const pg_adam_params* a) {
    if (!net || !a) return bad_arg("pg_unet_adam_step: NULL argument");
    net->adam_t += 1;
    const double c1 = 1.0 / (1.0 - std::pow(a->beta1, (double)net->adam_t));
    const double c2 = 1.0 / (1.0 - std::pow(a->beta2, (double)net->adam_t));
    const i64 P = num_params();
    PG_LAUNCH(KK_UNET_MISC, net->stream,
              k_adam<<<blocks_for(net, P), 256, 0, net->stream>>>(net->params, net->grads, net->adam_m, net->adam_v, P,
                                                                  (float)a->lr, (float)a->beta1, (float)a->beta2,
                                                                  (float)a->eps, (float)a->grad_scale, (float)c1,
                                                                  (float)c2));
    PG_CHECK_LAUNCH();
    net->wdirty = net->wdirty_mma = true;
    return PG_OK;
}

int pg_unet_set_loss(pg_unet* net, int kind) {
    if (!net) return bad_arg("pg_unet_set_loss: NULL net");
    if (kind != 0 && kind != 1) return bad_arg("pg_unet_set_loss: kind must be 0 (MSE) or 1 (energy norm)");
    net->loss_kind = kind;
    return PG_OK;
}

int pg_unet_forward_f32(pg_unet* net, const pg_grid* g, const float* b, double dt, float* p) {
    if (!net || !b || !p) return bad_arg("pg_unet_forward_f32: NULL argument");
    if (!(dt > 0.0)) return bad_arg("pg_unet_forward_f32: dt must be > 0");
    int rc;
    if ((rc = check_grid(net, g))) return rc;
    if ((rc = forward(net, g, b, dt)) || (rc = head(net, g, dt, p, nullptr))) return rc;
    return PG_OK;
}

int pg_unet_guess_f32(pg_unet* net, const pg_grid* g, const float* b, double dt, int corrections, float* x) {
    if (!net || !b || !x) return bad_arg("pg_unet_guess_f32: NULL argument");
    if (!(dt > 0.0)) return bad_arg("pg_unet_guess_f32: dt must be > 0");
    if (corrections < 0 || corrections > 16) return bad_arg("pg_unet_guess_f32: corrections must be in 0..16");
    if (x == b) return bad_arg("pg_unet_guess_f32: x must not alias b");
    int rc;
    if ((rc = check_grid(net, g))) return rc;
    const i64 V0 = net->lv[0];
    cudaStream_t s = net->stream;
    PG_CUDA(cudaMemsetAsync(x, 0, 4 * V0, s));
    PG_CUDA(cudaMemcpyAsync(net->r, b, 4 * V0, cudaMemcpyDeviceToDevice, s));
    float* alpha = net->scal + 4;
    for (int c = 0; c <= corrections; ++c) {
        // d = net(r); x += alpha d, r -= alpha A d with the A-optimal alpha.
        if ((rc = forward(net, g, net->r, dt)) || (rc = head(net, g, dt, net->q, nullptr))) return rc;
        if ((rc = apply_a(net, g, net->ad, net->q, dt))) return rc;
        PG_LAUNCH(KK_UNET_MISC, s, k_dots<<<kRedBlocks, kRedThreads, 0, s>>>(net->q, net->r, net->ad, V0, net->red));
        PG_LAUNCH(KK_UNET_MISC, s, k_alpha<<<1, 32, 0, s>>>(net->red, kRedBlocks, alpha));
        PG_LAUNCH(KK_UNET_MISC, s, k_step<<<blocks_for(net, V0), 256, 0, s>>>(x, net->r, net->q, net->ad, alpha, V0));
    }
    PG_CHECK_LAUNCH();
    return PG_OK;
}


// z = the learned correction (see LearnedHook) inside a flexible CG, with or
// without FP64-class refinement as params say.
int pg_solve_pressure_learned_f32(const pg_grid* g, const pg_solver_params* prm, pg_unet* net, float* x,
                                  const float* b, double dt, pg_pcg_stats* stats) {
    if (!g || !prm || !net || !x || !b) return bad_arg("pg_solve_pressure_learned_f32: NULL argument");
    if (!(dt > 0.0)) return bad_arg("pg_solve_pressure_learned_f32: dt must be > 0");
    int rc;
    if ((rc = check_grid(net, g))) return rc;
    if ((rc = prep_weights(net))) return rc;  // outside any capture of the CG loop
    LearnedHook hook;
    hook.net = net;
    hook.dt = dt;
    pg_pcg_stats s{};
    if ((rc = solve_pressure_hooked(const_cast<pg_grid*>(g), prm, x, b, dt, &hook, &s))) return rc;
    if ((rc = check_err(net))) return rc;
    if (stats) *stats = s;
    return s.status;
}

}  // extern "C"
