// pg_batch_mg.cu -- geometric multigrid V-cycle for batches of 2D grids
// (PG_PRECOND_MG in pg_batch_step_f32; an extension behind the reference's
// `Preconditioner` trait, pcg.rs:4-6).
//
// Every grid gets the hierarchy of the single-grid preconditioner
// (pg_mg.cu): cell-centred levels halving each side (rounded up) until the
// shorter side is <= 2 or the level has <= 64 cells; coarse face weights are
// half the sum of the fine weights crossing the coarse face; restriction sums
// the children's residuals, prolongation adds the parent's correction;
// red-black Gauss-Seidel, `nsmooth` sweeps (red, black) before and (black,
// red) after, so the V-cycle is symmetric; the coarsest level is solved in
// shared memory by symmetric sweeps.  Grids have different depths: level l
// of the batch packs level l of every grid that has it.
//
// The large levels are smoothed by warps that march down strips of 64
// columns (k_bmg_pair: both half-sweeps of a pair from one read of the
// level, restriction and z.r on the way), one launch for all grids; the
// rest of a grid's hierarchy, from its first level of kBmgTailCells cells or
// fewer in all, is one block's work in shared memory (k_bmg_tail), one
// launch as well.  The CG kernels around the V-cycle march likewise.  Grids
// whose CG has converged return at once.  Every warp writes one partial
// sum; a per-grid block folds them in a fixed order.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "pg_batch.cuh"

namespace pg {

constexpr int kBmgMaxLevels = 16;
constexpr int kBmgCoarseMax = 2048;
constexpr int kRtX = 32, kRtY = 8;  // setup tile: 32 x 8 coarse cells
// Cells (of all its levels together, 20 bytes each) that a block keeps in
// shared memory, two blocks per SM: 64 x 64 and the levels below it are 5440.
constexpr int kBmgTailCells = 5600;
constexpr int kBmgTailThreads = 512;
constexpr int kUpdateCells = 2048;  // cells per warp of the CG update

// A grid at a level (off: in the level's packed arrays; level 0: the batch's).
struct BLevel : MarchLevel {
    int coarse;   // the grid's coarsest level
    int tail;     // its first level of k_bmg_tail
    int t0, t1;   // its smoothing strips (level 0)
};

// Cells [c0, c1) of a grid in the packed fields.
struct Chunk {
    int grid, pad;
    i64 c0, c1;
};

struct BatchMg {
    int nlev = 0;  // levels of the deepest grid
    float dt = 0.f;
    unsigned long long mask_version = 0;
    uint64_t id = 0;
    std::vector<void*> allocs;
    BLevel* info[kBmgMaxLevels] = {};
    Strip* strips[kBmgMaxLevels] = {};
    int nst[kBmgMaxLevels] = {};
    int nsmoothing[kBmgMaxLevels] = {};  // grids smoothing at this level by k_bmg_pair
    Tile* rtiles[kBmgMaxLevels] = {};
    int nrt[kBmgMaxLevels] = {};
    float* wx[kBmgMaxLevels] = {};
    float* wy[kBmgMaxLevels] = {};
    float* invd[kBmgMaxLevels] = {};
    float* e[kBmgMaxLevels] = {};
    float* e2[kBmgMaxLevels] = {};  // k_bmg_pair writes e and e2 in turn (level 0: z and ap)
    float* f[kBmgMaxLevels] = {};
    int tail_cells = 0;             // of the grid with the largest tail
    Strip* cg_strips = nullptr;     // the SpMV's: 64 columns each, no overlap
    int ncg = 0;
    int2* cg_range = nullptr;
    Chunk* chunks = nullptr;        // the CG update's
    int nchunk = 0;
    int2* chunk_range = nullptr;
    double* partials = nullptr;     // 2 per strip or chunk
    Pockets pockets;  // fluid components of the grids with more than one
};

// Device view of one level of the batch.
struct BLv : MarchView {
    const BLevel* info;
    int level;
};

template <bool L0> struct BCell {
    float wxl, wxh, wyl, wyh, inv;
    __device__ __forceinline__ BCell(const BLv& v, i64 c, int y, int x, int h, int w) {
        if (L0) {
            const uint8_t f = v.flags[c];
            wxl = (f & XLO) ? v.dt : 0.f;
            wxh = (f & XHI) ? v.dt : 0.f;
            wyl = (f & YLO) ? v.dt : 0.f;
            wyh = (f & YHI) ? v.dt : 0.f;
            const int n = __popc((unsigned)f);
            inv = n ? __frcp_rn((float)n * v.dt) : 0.f;
        } else {
            wxl = v.wx[c];
            wxh = x + 1 < w ? v.wx[c + 1] : 0.f;
            wyl = v.wy[c];
            wyh = y + 1 < h ? v.wy[c + w] : 0.f;
            inv = v.invd[c];
        }
    }
};

// A smoothing pair at one level of every grid that smooths there, from ein
// to eout.  RZ (level 0, last): also z.r and sum(z) per strip, for grids
// that don't smooth on level 0 as well (z, left by k_bmg_tail, is in eout).
//
// Bound by memory: a pair reads f, flags and e and writes e, 13 bytes per
// cell on level 0, where two half-sweeps of a launch each read all of it and
// wrote half, 8 launches and a restriction per V-cycle.  In a strip the rows
// are read once (registers hold them while they are neighbours), x neighbours
// come by shuffle; two lanes at an inner edge of a strip and two or three
// rows at its ends are recomputed: the pair needs two cells beyond its own,
// the residual three.  256 grids of 21 M cells, all running: 47 us the first
// pair, 80 with the restriction (issue bound at 0.74 per cycle), 62 with the
// prolongation, 67 with z.r (loads in flight: 28 warps of 70 registers), where
// the eight half-sweeps took 75 to 141 each and the restriction 98.
template <bool L0, int MODE, int C1, bool RZ, bool REST>
__global__ void __launch_bounds__(kMarchThreads, L0 ? (RZ || REST ? 7 : 8) : 5)
    k_bmg_pair(BLv v, const float* __restrict__ ein, float* __restrict__ eout, const Strip* __restrict__ strips, int n,
               const BState* __restrict__ st, double* __restrict__ partials) {
    const int i = blockIdx.x * (kMarchThreads / 32) + (threadIdx.x >> 5);
    if (i >= n) return;
    const Strip S = strips[i];
    if (st[S.grid].done) return;
    const BLevel L = v.info[S.grid];
    F2 a{0.f, 0.f}, b{0.f, 0.f};
    if (L.tail > v.level) {
        if (((L.off | (i64)L.w) & 1) == 0) {
            March<L0, MODE, C1, RZ, REST, true> m(v, L, S, ein, eout);
            m.run();
            a = f2_of(m.acc);
            b = f2_of(m.zs);
        } else {
            March<L0, MODE, C1, RZ, REST, false> m(v, L, S, ein, eout);
            m.run();
            a = f2_of(m.acc);
            b = f2_of(m.zs);
        }
    } else if (RZ) {
        const int lo = S.x0 ? S.x0 + 4 : 0, hi = S.x0 + 64 >= L.w ? L.w : S.x0 + 60;
        Acc<float> acc, zs;
        for (int y = S.y0; y < S.y1; ++y)
            for (int x = lo + (threadIdx.x & 31); x < hi; x += 32) {
                const i64 c = L.off + (i64)y * L.w + x;
                acc.add(eout[c] * v.f[c]);
                zs.add(eout[c]);
            }
        a = f2_of(acc);
        b = f2_of(zs);
    }
    if (RZ) {
        a = f2_warp(a);
        b = f2_warp(b);
        if ((threadIdx.x & 31) == 0) {
            partials[2 * (i64)i] = (double)a.hi + (double)a.lo;
            partials[2 * (i64)i + 1] = (double)b.hi + (double)b.lo;
        }
    }
}

// Device view of the levels of k_bmg_tail.
struct BTail {
    const BLevel* info[kBmgMaxLevels];
    const float* wx[kBmgMaxLevels];
    const float* wy[kBmgMaxLevels];
    const float* invd[kBmgMaxLevels];
    const float* f[kBmgMaxLevels];
    float* e[kBmgMaxLevels];
    const uint8_t* flags;
    float dt;
    int nsmooth;
};

// One level in shared memory: n cells each of e, f, wx, wy, 1 / diagonal.
struct TailLevel {
    float* e;
    int h, w, n;
    unsigned magic;  // i / w = umulhi(i, magic) (w >= 2)
    __device__ __forceinline__ TailLevel(float* at, int h_, int w_) : e(at), h(h_), w(w_), n(h_ * w_) {
        magic = 0xffffffffu / (unsigned)w + 1u;
    }
    __device__ __forceinline__ float* f() const { return e + n; }
    __device__ __forceinline__ float* wx() const { return e + 2 * n; }
    __device__ __forceinline__ float* wy() const { return e + 3 * n; }
    __device__ __forceinline__ float* inv() const { return e + 4 * n; }
    // Cell i of a colour, in row-major order: of the pair 2i, 2i + 1 one cell
    // has the colour (rows of odd length: always the same one).  It may be n.
    __device__ __forceinline__ int cell(int i, int color) const {
        return 2 * i + ((w & 1) ? color : (((int)__umulhi(2u * (unsigned)i, magic) + color) & 1));
    }
};

// One half-sweep; C: the next level, whose correction the neighbours get
// (PROLONG).  A neighbour behind a closed face is not added, outside the grid
// the cell itself is read.
template <bool PROLONG>
__device__ __forceinline__ void tail_sweep(const TailLevel& T, const TailLevel& C, int color, int t, int nt) {
    const int items = (T.n + 1) >> 1;
#pragma unroll 2
    for (int i = t; i < items; i += nt) {
        const int c = T.cell(i, color);
        if (c >= T.n) continue;
        const int y = (int)__umulhi((unsigned)c, T.magic), x = c - y * T.w;
        const bool xl = x > 0, xh = x + 1 < T.w, yl = y > 0, yh = y + 1 < T.h;
        const int l = xl ? c - 1 : c, r = xh ? c + 1 : c, u = yl ? c - T.w : c, d = yh ? c + T.w : c;
        const float wl = T.wx()[c], wr = xh ? T.wx()[r] : 0.f, wu = T.wy()[c], wd = yh ? T.wy()[d] : 0.f;
        float nl = T.e[l], nr = T.e[r], nu = T.e[u], nd = T.e[d];
        if (PROLONG) {
            const float* row = C.e + (y >> 1) * C.w;
            nl += row[(xl ? x - 1 : x) >> 1];
            nr += row[(xh ? x + 1 : x) >> 1];
            nu += C.e[((yl ? y - 1 : y) >> 1) * C.w + (x >> 1)];
            nd += C.e[((yh ? y + 1 : y) >> 1) * C.w + (x >> 1)];
        }
        T.e[c] = nb_sum(T.f()[c], wl, wr, wu, wd, nl, nr, nu, nd) * T.inv()[c];
    }
}

// The rest of a grid's V-cycle, one block per grid: from level L.tail (its
// right-hand side restricted there by k_bmg_pair, or r itself) down to the
// coarsest level, solved by symmetric sweeps from e = 0, and up again; the
// correction of level L.tail (or z) is written out.
//
// Bound by latency: a half-sweep of 64 x 64 cells is four cells per thread,
// and each launch that it was cost 6 to 8 us.  A coarsest level of up to 64
// cells is one warp's work, a cell of each colour per lane, neighbours by
// shuffle (512 threads took 38 us for the 128 half-sweeps, nearly all of it
// at barriers).  37 us for 256 grids at once, 15 for a few, where the launches
// of these levels took 250.
__global__ void __launch_bounds__(kBmgTailThreads, 2) k_bmg_tail(BTail v, const BState* __restrict__ st) {
    extern __shared__ float smem[];
    const int g = blockIdx.x, tid = threadIdx.x, nt = kBmgTailThreads;
    if (st[g].done) return;
    const int lt = v.info[0][g].tail, lc = v.info[0][g].coarse;
    {
        float* at = smem;
        for (int l = lt; l <= lc; ++l) {
            const BLevel L = v.info[l][g];
            const TailLevel T(at, L.h, L.w);
#pragma unroll 4
            for (int c = tid; c < T.n; c += nt) {
                float inv, wx, wy;
                if (l == 0) {
                    const unsigned fl = v.flags[L.off + c];
                    wx = (fl & XLO) ? v.dt : 0.f;
                    wy = (fl & YLO) ? v.dt : 0.f;
                    const int k = __popc(fl);
                    inv = k ? __frcp_rn((float)k * v.dt) : 0.f;
                } else {
                    wx = v.wx[l][L.off + c];
                    wy = v.wy[l][L.off + c];
                    inv = v.invd[l][L.off + c];
                }
                const float f = l == lt ? v.f[l][L.off + c] : 0.f;
                T.wx()[c] = wx;
                T.wy()[c] = wy;
                T.inv()[c] = inv;
                if (l == lt) {
                    T.f()[c] = f;
                    T.e[c] = inv != 0.f ? f * inv : 0.f;  // the first half-sweep (the other colour is not read)
                }
            }
            at += 5 * T.n;
        }
    }
    __syncthreads();
    float* at = smem;
    for (int l = lt; l < lc; ++l) {
        const BLevel L = v.info[l][g];
        const TailLevel T(at, L.h, L.w), C(at + 5 * T.n, L.ch, L.cw);
        tail_sweep<false>(T, T, 1, tid, nt);
        __syncthreads();
        for (int k = 1; k < v.nsmooth; ++k) {
            tail_sweep<false>(T, T, 0, tid, nt);
            __syncthreads();
            tail_sweep<false>(T, T, 1, tid, nt);
            __syncthreads();
        }
        for (int c = tid; c < C.n; c += nt) {
            const int Y = (int)__umulhi((unsigned)c, C.magic), X = c - Y * C.w;
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int y = 2 * Y + (k >> 1), x = 2 * X + (k & 1);
                if (y >= T.h || x >= T.w) continue;
                const int i = y * T.w + x;
                const bool xh = x + 1 < T.w, yh = y + 1 < T.h;
                const float wl = T.wx()[i], wr = xh ? T.wx()[i + 1] : 0.f, wu = T.wy()[i],
                            wd = yh ? T.wy()[i + T.w] : 0.f;
                const float e = T.e[i];
                sum += T.f()[i] - nb_sum(0.f, wl, wr, wu, wd, e - T.e[x > 0 ? i - 1 : i], e - T.e[xh ? i + 1 : i],
                                         e - T.e[y > 0 ? i - T.w : i], e - T.e[yh ? i + T.w : i]);
            }
            C.f()[c] = sum;
            const float inv = C.inv()[c];
            C.e[c] = l + 1 < lc && inv != 0.f ? sum * inv : 0.f;
        }
        at += 5 * T.n;
        __syncthreads();
    }
    {
        const BLevel L = v.info[lc][g];
        const TailLevel T(at, L.h, L.w);
        if (lt == lc) {
            for (int c = tid; c < T.n; c += nt) T.e[c] = 0.f;
            __syncthreads();
        }
        const int pairs = coarse_pairs(1, L.h, L.w);
        if (T.n <= 64) {
            if (tid < 32) {
                // per colour: the lane's cell, its weights (0 at closed faces and
                // past the grid) and the lanes that hold its neighbours
                float f[2], inv[2], w[2][4], e[2] = {0.f, 0.f};
                int nb[2][4];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int c = T.cell(tid, q);
                    const bool in = c < T.n;
                    const int y = (int)__umulhi((unsigned)c, T.magic), x = c - y * T.w;
                    f[q] = in ? T.f()[c] : 0.f;
                    inv[q] = in ? T.inv()[c] : 0.f;
                    const bool face[4] = {in && x > 0, in && x + 1 < T.w, in && y > 0, in && y + 1 < T.h};
                    const int to[4] = {c - 1, c + 1, c - T.w, c + T.w};
                    const float* from[4] = {T.wx() + c, T.wx() + to[1], T.wy() + c, T.wy() + to[3]};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        nb[q][j] = face[j] ? to[j] >> 1 : tid;
                        w[q][j] = face[j] ? *from[j] : 0.f;
                    }
                }
                auto sweep = [&](auto colour) {
                    constexpr int q = decltype(colour)::value;
                    float n[4], s = f[q];
#pragma unroll
                    for (int j = 0; j < 4; ++j) n[j] = __shfl_sync(0xffffffffu, e[1 - q], nb[q][j]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) s = fmaf(w[q][j], n[j], s);
                    e[q] = s * inv[q];
                };
                using Zero = std::integral_constant<int, 0>;
                using One = std::integral_constant<int, 1>;
                for (int p = 0; p < pairs; ++p) {
                    sweep(Zero{});
                    sweep(One{});
                }
                for (int p = 0; p < pairs; ++p) {
                    sweep(One{});
                    sweep(Zero{});
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int c = T.cell(tid, q);
                    if (c < T.n) T.e[c] = e[q];
                }
            }
            __syncthreads();
        } else {
            for (int it = 0; it < 4 * pairs; ++it) {
                tail_sweep<false>(T, T, it < 2 * pairs ? (it & 1) : ((it & 1) ^ 1), tid, nt);
                __syncthreads();
            }
        }
    }
    for (int l = lc - 1; l >= lt; --l) {
        const BLevel L = v.info[l][g];
        const TailLevel C(at, L.ch, L.cw);
        at -= 5 * L.h * L.w;
        const TailLevel T(at, L.h, L.w);
        tail_sweep<true>(T, C, 1, tid, nt);
        __syncthreads();
        for (int k = 0; k < v.nsmooth; ++k) {
            if (k > 0) {
                tail_sweep<false>(T, T, 1, tid, nt);
                __syncthreads();
            }
            tail_sweep<false>(T, T, 0, tid, nt);
            __syncthreads();
        }
    }
    const BLevel L = v.info[lt][g];
    for (int c = tid; c < L.h * L.w; c += nt) v.e[lt][L.off + c] = smem[c];
}

// p = z + beta p (z - zmean on fluid cells; ping-pong by the grid's iteration
// count), A p and p.Ap over strips of 64 columns, 17 bytes per cell.  The
// cells beside a strip are read by its edge lanes, the rows above and below
// once more by the strips there.  72 us for 21 M cells (54 at the copy rate)
// where a block per tile of 256 cells, its state and tile loaded and its sum
// folded for each, took 211.
template <bool VEC>
__device__ __forceinline__ F2 bmg_spmv_strip(const BLevel& L, const Strip& S, const BState& st, const float* z, float* p0,
                                             float* p1, float* ap, const uint8_t* flags, float dt) {
    const int lane = threadIdx.x & 31, x = S.x0 + 2 * lane;
    const bool va = x < L.w, vb = x + 1 < L.w;
    const bool first = st.first != 0;
    const float beta = st.fbeta, zm = st.fzm;
    const float* __restrict__ p_old = (st.iter & 1) ? p1 : p0;
    float* __restrict__ p_new = (st.iter & 1) ? p0 : p1;
    // the cell beside the strip: left of lane 0, right of lane 31
    const int dx = lane == 0 ? -1 : 2;
    const bool edge = (lane == 0 && S.x0 > 0) || (lane == 31 && S.x0 + 64 < L.w);
    struct Row {
        float2 z, p;
        Flag2 fl;
        float ez, ep;
    };
    i64 at = L.off + (i64)(S.y0 - 1) * L.w + x;
    int next = S.y0 - 1;
    auto fetch = [&]() {
        Row q;
        q.z = q.p = make_float2(0.f, 0.f);
        q.fl.a = q.fl.b = 0;
        q.ez = q.ep = 0.f;
        if (next >= 0 && next < L.h && next <= S.y1) {
            q.z = ld2<VEC>(z + at, va, vb);
            q.fl.template load<VEC>(flags + at, va, vb);
            if (edge) q.ez = z[at + dx];
            if (!first) {
                q.p = ld2<VEC>(p_old + at, va, vb);
                if (edge) q.ep = p_old[at + dx];
            }
        }
        ++next;
        at += L.w;
        return q;
    };
    // p_new; the projected z applies to cells with an open face (a neighbour
    // behind an open face always has one)
    auto pn = [&](float zv, float pv, bool fluid) {
        const float zz = fluid ? zv - zm : zv;
        return first ? zz : fmaf(beta, pv, zz);
    };
    auto of = [&](const Row& q) {
        const unsigned f = q.fl.template both<VEC>();
        return make_float2(pn(q.z.x, q.p.x, (f & 0xffu) != 0), pn(q.z.y, q.p.y, (f >> 8) != 0));
    };
    Row q0 = fetch(), q1 = fetch(), q2 = fetch();
    float2 up = of(q0), cur = of(q1);
    unsigned fl = q1.fl.template both<VEC>();
    float ext = pn(q1.ez, q1.ep, true);
    q0 = q2;
    q1 = fetch();
    Acc<float> acc;
    i64 out = L.off + (i64)S.y0 * L.w + x;
#pragma unroll 2
    for (int y = S.y0; y < S.y1; ++y, out += L.w) {
        const Row q = q0;  // row y + 1
        q0 = q1;
        q1 = fetch();
        const float2 dn = of(q);
        float l = __shfl_up_sync(0xffffffffu, cur.y, 1), r = __shfl_down_sync(0xffffffffu, cur.x, 1);
        l = lane == 0 ? ext : l;
        r = lane == 31 ? ext : r;
        auto apply = [&](unsigned f, float pc, float pl, float pr, float pu, float pd) {
            const float gy_lo = (f & YLO) ? -sub_rn(pc, pu) : 0.f;
            const float gy_hi = (f & YHI) ? -sub_rn(pd, pc) : 0.f;
            const float gx_lo = (f & XLO) ? sub_rn(pl, pc) : 0.f;
            const float gx_hi = (f & XHI) ? sub_rn(pc, pr) : 0.f;
            return mul_rn(add_rn(sub_rn(sub_rn(gy_hi, gy_lo), gx_lo), gx_hi), dt);
        };
        const float2 a = make_float2(apply(fl, cur.x, l, cur.y, up.x, dn.x), apply(fl >> 8, cur.y, cur.x, r, up.y, dn.y));
        st2<VEC>(p_new + out, cur, va, vb);
        st2<VEC>(ap + out, a, va, vb);
        if (va) acc.add(cur.x * a.x);
        if (vb) acc.add(cur.y * a.y);
        up = cur;
        cur = dn;
        fl = q.fl.template both<VEC>();
        ext = pn(q.ez, q.ep, true);
    }
    return f2_of(acc);
}

__global__ void __launch_bounds__(kMarchThreads, 7)
    k_bmg_spmv(const BLevel* __restrict__ info, const Strip* __restrict__ strips, int n, const BState* __restrict__ st,
               const float* __restrict__ z, float* p0, float* p1, float* __restrict__ ap,
               const uint8_t* __restrict__ flags, float dt, double* __restrict__ partials) {
    const int i = blockIdx.x * (kMarchThreads / 32) + (threadIdx.x >> 5);
    if (i >= n) return;
    const Strip S = strips[i];
    const BState& B = st[S.grid];
    if (B.done) return;
    const BLevel L = info[S.grid];
    F2 a = ((L.off | (i64)L.w) & 1) == 0 ? bmg_spmv_strip<true>(L, S, B, z, p0, p1, ap, flags, dt)
                                         : bmg_spmv_strip<false>(L, S, B, z, p0, p1, ap, flags, dt);
    a = f2_warp(a);
    if ((threadIdx.x & 31) == 0) {
        partials[2 * (i64)i] = (double)a.hi + (double)a.lo;
        partials[2 * (i64)i + 1] = 0.0;
    }
}

// A warp's walk over its chunk of a grid's cells, four at a time where the
// fields' 16-byte groups allow it (vec), the cells around them one by one:
// four(c) and single(c).
template <class F4, class F1>
__device__ __forceinline__ void walk_chunk(const Chunk& C, int vec, F4&& four, F1&& single) {
    const int lane = threadIdx.x & 31;
    const i64 g0 = vec ? (C.c0 + 3) / 4 * 4 : C.c1, g1 = vec ? C.c1 / 4 * 4 : C.c1;
    if (g0 < g1) {
        for (i64 c = g0 + 4 * lane; c < g1; c += 128) four(c);
        if (C.c0 + lane < g0) single(C.c0 + lane);
        if (g1 + lane < C.c1) single(g1 + lane);
    } else {
        for (i64 c = C.c0 + lane; c < C.c1; c += 32) single(c);
    }
}
__device__ __forceinline__ float abs_or_inf(float v) { return isfinite(v) ? fabsf(v) : __int_as_float(0x7f800000); }
__device__ __forceinline__ void chunk_partials(float rm, const Acc<float>& sum, double* __restrict__ out) {
    for (int o = 16; o > 0; o >>= 1) rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, o));
    const F2 t = f2_warp(f2_of(sum));
    if ((threadIdx.x & 31) == 0) {
        out[0] = (double)rm;
        out[1] = (double)t.hi + (double)t.lo;
    }
}

// x += alpha p, r -= alpha Ap, max|r| and sum(r) (for the lazy projection);
// 24 bytes per cell.  71 us for 21 M cells (76 at the copy rate, part of it in
// L2), 181 with a block per tile.
__global__ void __launch_bounds__(256)
    k_bmg_update(const Chunk* __restrict__ chunks, int n, const BState* __restrict__ st, float* __restrict__ x,
                 float* __restrict__ r, const float* p0, const float* p1, const float* __restrict__ ap, int vec,
                 double* __restrict__ partials) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const Chunk C = chunks[i];
    const BState& S = st[C.grid];
    if (S.done) return;
    const float* __restrict__ p = ((S.iter + 1) & 1) ? p1 : p0;
    const float al = S.falpha, nal = -al;
    float rm = 0.f;
    Acc<float> sum;
    auto one = [&](float& xv, float& rv, float pv, float av) {
        xv = fmaf(al, pv, xv);
        rv = fmaf(nal, av, rv);
        rm = fmaxf(rm, abs_or_inf(rv));
        sum.add(rv);
    };
    walk_chunk(
        C, vec,
        [&](i64 c) {
            float4 xv = *reinterpret_cast<const float4*>(x + c), rv = *reinterpret_cast<const float4*>(r + c);
            const float4 pv = *reinterpret_cast<const float4*>(p + c), av = *reinterpret_cast<const float4*>(ap + c);
            one(xv.x, rv.x, pv.x, av.x);
            one(xv.y, rv.y, pv.y, av.y);
            one(xv.z, rv.z, pv.z, av.z);
            one(xv.w, rv.w, pv.w, av.w);
            *reinterpret_cast<float4*>(x + c) = xv;
            *reinterpret_cast<float4*>(r + c) = rv;
        },
        [&](i64 c) {
            float xv = x[c], rv = r[c];
            one(xv, rv, p[c], ap[c]);
            x[c] = xv;
            r[c] = rv;
        });
    chunk_partials(rm, sum, partials + 2 * (i64)i);
}

// x = 0, r = b, max|b| and sum(b).
__global__ void __launch_bounds__(256)
    k_bmg_init(const Chunk* __restrict__ chunks, int n, float* __restrict__ x, float* __restrict__ r,
               const float* __restrict__ b, int vec, double* __restrict__ partials) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const Chunk C = chunks[i];
    float bm = 0.f;
    Acc<float> sum;
    auto one = [&](float bv) {
        bm = fmaxf(bm, abs_or_inf(bv));
        sum.add(bv);
    };
    walk_chunk(
        C, vec,
        [&](i64 c) {
            const float4 bv = *reinterpret_cast<const float4*>(b + c);
            one(bv.x);
            one(bv.y);
            one(bv.z);
            one(bv.w);
            *reinterpret_cast<float4*>(x + c) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4*>(r + c) = bv;
        },
        [&](i64 c) {
            const float bv = b[c];
            one(bv);
            x[c] = 0.f;
            r[c] = bv;
        });
    chunk_partials(bm, sum, partials + 2 * (i64)i);
}

// Coarse face weights of level l+1 from level l (tiles over level l+1).
template <bool L0>
__global__ void k_bmg_coarsen(BLv v, float* __restrict__ wxc, float* __restrict__ wyc, const Tile* __restrict__ tiles,
                              int ntiles) {
    FOR_TILES(tiles, ntiles) {
        const Tile t = tiles[ti];
        const BLevel L = v.info[t.grid];
        const int Y = t.y0 + (int)threadIdx.x / kRtX, X = t.x0 + (int)threadIdx.x % kRtX;
        if (Y >= L.ch || X >= L.cw) continue;
        const int y0 = 2 * Y, y1 = min(2 * Y + 2, L.h), x0 = 2 * X, x1 = min(2 * X + 2, L.w);
        float sx = 0.f, sy = 0.f;
        for (int y = y0; y < y1; ++y)
            for (int x = x0; x < x1; ++x) {
                const i64 c = L.off + (i64)y * L.w + x;
                const BCell<L0> cl(v, c, y, x, L.h, L.w);
                if (x == x0) sx += cl.wxl;
                if (y == y0) sy += cl.wyl;
            }
        const i64 C = L.coff + (i64)Y * L.cw + X;
        wxc[C] = 0.5f * sx;
        wyc[C] = 0.5f * sy;
    }
}

// 1 / diagonal of level l+1 (v = level l+1's view; tiles over its cells).
__global__ void k_bmg_invd(BLv v, float* __restrict__ invd, const Tile* __restrict__ tiles, int ntiles) {
    FOR_TILES(tiles, ntiles) {
        const Tile t = tiles[ti];
        const BLevel L = v.info[t.grid];
        const int y = t.y0 + (int)threadIdx.x / kRtX, x = t.x0 + (int)threadIdx.x % kRtX;
        if (y >= L.h || x >= L.w) continue;
        const i64 c = L.off + (i64)y * L.w + x;
        float s = v.wx[c] + v.wy[c];
        if (x + 1 < L.w) s += v.wx[c + 1];
        if (y + 1 < L.h) s += v.wy[c + L.w];
        invd[c] = s > 0.f ? 1.f / s : 0.f;
    }
}

// Per grid: z.r = sum of its level-0 strips' partials (fixed order).
// first: sigma = z.r; else beta = z.r / sigma, sigma = z.r.
__global__ void k_bmg_rz_finalize(const BLevel* __restrict__ info0, BState* __restrict__ st,
                                  const double* __restrict__ partials, int n, int first) {
    __shared__ double sm[32];
    const int g = blockIdx.x;
    if (g >= n) return;
    BState& S = st[g];
    if (S.done) return;
    const BLevel L = info0[g];
    double a = 0.0, zsum = 0.0;
    for (int t = L.t0 + threadIdx.x; t < L.t1; t += blockDim.x) {
        a += partials[2 * (i64)t];
        zsum += partials[2 * (i64)t + 1];
    }
    a = bsum(a, sm);
    zsum = bsum(zsum, sm);
    if (threadIdx.x != 0) return;
    if (S.nfluid > 0.0) {  // z stands for z - m on the fluid cells: (z - m).r = z.r - m sum(r)
        const double m = zsum / S.nfluid;
        S.zmean = m;
        S.fzm = (float)m;
        a -= m * S.rsum;
    }
    if (!isfinite(a)) {
        S.status = PG_NAN_DETECTED;
        S.done = 1;
        return;
    }
    if (first) {
        S.sigma = a;
    } else {
        S.beta = a / S.sigma;
        S.fbeta = (float)S.beta;
        S.sigma = a;
    }
}

// ---------------------------------------------------------------------------
// host side

static uint64_t next_bmg_id() {
    static std::atomic<uint64_t> n{0};
    return ++n;
}

void bmg_release(pg_batch* B) {
    if (!B->mg) return;
    release_pockets(&B->mg->pockets);
    for (void* p : B->mg->allocs) cudaFree(p);
    delete B->mg;
    B->mg = nullptr;
}

uint64_t bmg_id(const pg_batch* B) { return B->mg ? B->mg->id : 0; }

static BLv view(const pg_batch* B, int l) {
    const BatchMg& M = *B->mg;
    BLv v;
    v.info = M.info[l];
    v.wx = M.wx[l];
    v.wy = M.wy[l];
    v.invd = M.invd[l];
    v.f = l == 0 ? B->r : M.f[l];
    v.flags = B->flags;
    v.ec = l + 1 < M.nlev ? M.e[l + 1] : nullptr;
    v.fc = l + 1 < M.nlev ? M.f[l + 1] : nullptr;
    v.dt = M.dt;
    v.level = l;
    return v;
}

static int bmg_blocks(const pg_batch* B, int ntiles) { return std::max(1, std::min(ntiles, B->num_sms * 8)); }

static int bmg_build(pg_batch* B, float dt);

int bmg_ensure(pg_batch* B, float dt) {
    if (B->mg && B->mg->dt == dt && B->mg->mask_version == B->mask_version) return PG_OK;
    bmg_release(B);
    if (!B->z) PG_CUDA(cudaMalloc(&B->z, sizeof(float) * (size_t)B->ncells));
    const int rc = bmg_build(B, dt);
    if (rc) bmg_release(B);
    return rc;
}

static int bmg_build(pg_batch* B, float dt) {
    BatchMg* M = new BatchMg();
    M->dt = dt;
    M->mask_version = B->mask_version;
    M->id = next_bmg_id();
    const int n = B->n;
    // level shapes per grid (the single-grid rule)
    std::vector<std::vector<int>> hs(n), wsz(n);
    std::vector<int> coarse(n);
    int nlev = 1;
    for (int g = 0; g < n; ++g) {
        int h = B->h[g], w = B->w[g];
        hs[g].push_back(h);
        wsz[g].push_back(w);
        while ((int)hs[g].size() < kBmgMaxLevels) {
            if (std::min(h, w) <= 2 || (i64)h * w <= 64) break;
            h = (h + 1) / 2;
            w = (w + 1) / 2;
            hs[g].push_back(h);
            wsz[g].push_back(w);
        }
        coarse[g] = (int)hs[g].size() - 1;
        if ((i64)hs[g].back() * wsz[g].back() > kBmgCoarseMax) {
            delete M;
            return bad_arg("PG_PRECOND_MG: a grid of the batch does not coarsen to a small enough level");
        }
        nlev = std::max(nlev, coarse[g] + 1);
    }
    M->nlev = nlev;
    B->mg = M;
    // packed offsets per level, tiles
    std::vector<std::vector<BLevel>> info(nlev, std::vector<BLevel>(n));
    std::vector<i64> lvcells(nlev, 0);
    for (int l = 0; l < nlev; ++l)
        for (int g = 0; g < n; ++g) {
            BLevel& L = info[l][g];
            L = BLevel{};
            L.coarse = coarse[g];
            if (l > coarse[g]) continue;
            L.h = hs[g][l];
            L.w = wsz[g][l];
            L.off = l == 0 ? B->coff[g] : lvcells[l];
            if (l > 0) lvcells[l] += ((i64)L.h * L.w + 1) & ~(i64)1;  // (even: rows of pairs stay aligned)
        }
    lvcells[0] = B->ncells;
    for (int l = 0; l < nlev; ++l)
        for (int g = 0; g < n; ++g)
            if (l < coarse[g]) {
                info[l][g].ch = hs[g][l + 1];
                info[l][g].cw = wsz[g][l + 1];
                info[l][g].coff = info[l + 1][g].off;
            }
    for (int g = 0; g < n; ++g) {
        int t = coarse[g];
        i64 cells = (i64)hs[g][t] * wsz[g][t];
        while (t > 0 && cells + (i64)hs[g][t - 1] * wsz[g][t - 1] <= kBmgTailCells) {
            --t;
            cells += (i64)hs[g][t] * wsz[g][t];
        }
        M->tail_cells = std::max(M->tail_cells, (int)cells);
        for (int l = 0; l < nlev; ++l) info[l][g].tail = t;
    }
    // strips of a level: `step` columns apart, chunks of up to `rows` rows (an
    // even number; fewer where the strips would not fill the chip)
    auto make_strips = [&](int l, bool all, int step, std::vector<Strip>& st) {
        for (int rows = 32; rows >= 8; rows /= 2) {
            st.clear();
            for (int g = 0; g < n; ++g) {
                BLevel& L = info[l][g];
                const int t0 = (int)st.size();
                if (all || l < L.tail) march_strips(g, L.h, L.w, step, rows, st);
                L.t0 = t0;
                L.t1 = (int)st.size();
            }
            if ((i64)st.size() >= (i64)B->num_sms * 24) break;
        }
    };
    auto dalloc = [&](void** p, size_t bytes) -> int {
        cudaError_t e = cudaMalloc(p, std::max<size_t>(bytes, 16));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(batch mg)");
        M->allocs.push_back(*p);
        return PG_OK;
    };
    int rc;
    auto upload = [&](void** p, const void* src, size_t bytes) -> int {
        const int e = dalloc(p, bytes);
        if (e) return e;
        if (bytes) PG_CUDA(cudaMemcpy(*p, src, bytes, cudaMemcpyHostToDevice));
        return PG_OK;
    };
    {  // the CG kernels' work lists
        std::vector<Strip> st;
        std::vector<Chunk> ch;
        std::vector<int2> sr(n), cr(n);
        make_strips(0, true, 64, st);
        for (int g = 0; g < n; ++g) {
            sr[g] = make_int2(info[0][g].t0, info[0][g].t1);
            cr[g].x = (int)ch.size();
            for (i64 c = B->coff[g]; c < B->coff[g + 1]; c += kUpdateCells)
                ch.push_back(Chunk{g, 0, c, std::min(c + kUpdateCells, B->coff[g + 1])});
            cr[g].y = (int)ch.size();
        }
        M->ncg = (int)st.size();
        M->nchunk = (int)ch.size();
        if ((rc = upload((void**)&M->cg_strips, st.data(), sizeof(Strip) * st.size())) ||
            (rc = upload((void**)&M->cg_range, sr.data(), sizeof(int2) * n)) ||
            (rc = upload((void**)&M->chunks, ch.data(), sizeof(Chunk) * ch.size())) ||
            (rc = upload((void**)&M->chunk_range, cr.data(), sizeof(int2) * n)))
            return rc;
    }
    for (int l = 0; l < nlev; ++l) {
        std::vector<Strip> st;
        std::vector<Tile> rt;
        make_strips(l, l == 0, 56, st);  // (every grid on level 0: z.r)
        for (int g = 0; g < n; ++g) {
            const BLevel& L = info[l][g];
            M->nsmoothing[l] += l < L.tail;
            if (l < coarse[g])
                for (int y0 = 0; y0 < L.ch; y0 += kRtY)
                    for (int x0 = 0; x0 < L.cw; x0 += kRtX) rt.push_back(Tile{g, y0, x0});
        }
        M->nst[l] = (int)st.size();
        M->nrt[l] = (int)rt.size();
        if ((rc = upload((void**)&M->info[l], info[l].data(), sizeof(BLevel) * n)) ||
            (rc = upload((void**)&M->strips[l], st.data(), sizeof(Strip) * st.size())) ||
            (rc = upload((void**)&M->rtiles[l], rt.data(), sizeof(Tile) * rt.size())))
            return rc;
        if (l >= 1) {
            const size_t b = sizeof(float) * (size_t)lvcells[l];
            if ((rc = dalloc((void**)&M->wx[l], b)) || (rc = dalloc((void**)&M->wy[l], b)) ||
                (rc = dalloc((void**)&M->invd[l], b)) || (rc = dalloc((void**)&M->e[l], b)) ||
                (rc = dalloc((void**)&M->f[l], b)))
                return rc;
            if (M->nsmoothing[l] && (rc = dalloc((void**)&M->e2[l], b))) return rc;
        }
    }
    if ((rc = dalloc((void**)&M->partials, 2 * sizeof(double) * std::max({M->nst[0], M->ncg, M->nchunk})))) return rc;
    PG_CUDA(cudaFuncSetAttribute(k_bmg_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(5 * sizeof(float)) * kBmgTailCells));
    // fluid components of every grid with more than one (host labelling, once per mask)
    {
        std::vector<uint8_t> hf((size_t)B->ncells);
        PG_CUDA(cudaMemcpy(hf.data(), B->flags, hf.size(), cudaMemcpyDeviceToHost));
        std::vector<i64> cells;
        std::vector<int> start, owner;
        for (int g = 0; g < n; ++g) {
            find_pockets(hf.data() + B->coff[g], 2, 1, B->h[g], B->w[g], B->coff[g], cells, start);
            owner.resize(start.empty() ? 0 : start.size() - 1, g);
        }
        if ((rc = upload_pockets(cells, start, &M->pockets, owner))) return rc;
    }
    // coarse operators
    cudaStream_t s = B->stream;
    for (int l = 0; l + 1 < nlev; ++l) {
        if (!M->nrt[l]) continue;
        const BLv v = view(B, l);
        const int nb = bmg_blocks(B, M->nrt[l]);
        if (l == 0)
            PG_LAUNCH(KK_MG_SETUP, s, k_bmg_coarsen<true><<<nb, kRtX * kRtY, 0, s>>>(v, M->wx[1], M->wy[1], M->rtiles[0], M->nrt[0]));
        else
            PG_LAUNCH(KK_MG_SETUP, s, k_bmg_coarsen<false><<<nb, kRtX * kRtY, 0, s>>>(v, M->wx[l + 1], M->wy[l + 1], M->rtiles[l], M->nrt[l]));
        const BLv cv = view(B, l + 1);
        PG_LAUNCH(KK_MG_SETUP, s, k_bmg_invd<<<nb, kRtX * kRtY, 0, s>>>(cv, M->invd[l + 1], M->rtiles[l], M->nrt[l]));
    }
    PG_CHECK_LAUNCH();
    return PG_OK;
}

template <bool L0, int MODE, int C1, bool RZ, bool REST>
static void bpair(pg_batch* B, cudaStream_t s, int l, const float* ein, float* eout) {
    BatchMg& M = *B->mg;
    const BLv v = view(B, l);
    PG_LAUNCH(l == 0 ? KK_MG_SMOOTH : KK_MG_SMOOTH_C, s,
              k_bmg_pair<L0, MODE, C1, RZ, REST><<<march_blocks(M.nst[l]), kMarchThreads, 0, s>>>(
                  v, ein, eout, M.strips[l], M.nst[l], B->state, M.partials));
}

// The pairs before (and the restriction) or after the coarser levels; they
// write e and its twin in turn, so that the last one leaves it in e.
template <bool L0> static void bmg_down(pg_batch* B, cudaStream_t s, int l, int nsmooth) {
    float *to = L0 ? B->ap : B->mg->e2[l], *other = L0 ? B->z : B->mg->e[l];  // (A p is dead here)
    if (nsmooth == 1) {
        bpair<L0, BP_SELF, 0, false, true>(B, s, l, nullptr, to);
        return;
    }
    bpair<L0, BP_SELF, 0, false, false>(B, s, l, nullptr, to);
    for (int k = 1; k < nsmooth; ++k, std::swap(to, other)) {
        if (k == nsmooth - 1) bpair<L0, BP_PLAIN, 0, false, true>(B, s, l, to, other);
        else bpair<L0, BP_PLAIN, 0, false, false>(B, s, l, to, other);
    }
}

template <bool L0> static void bmg_up(pg_batch* B, cudaStream_t s, int l, int nsmooth) {
    float *to = L0 ? B->ap : B->mg->e2[l], *other = L0 ? B->z : B->mg->e[l];
    if (nsmooth & 1) std::swap(to, other);  // (where bmg_down ended: `other`)
    if (nsmooth == 1) {
        bpair<L0, BP_PROLONG, 1, L0, false>(B, s, l, other, to);
        return;
    }
    bpair<L0, BP_PROLONG, 1, false, false>(B, s, l, other, to);
    for (int k = 1; k < nsmooth; ++k, std::swap(to, other)) {
        if (k == nsmooth - 1) bpair<L0, BP_PLAIN, 1, L0, false>(B, s, l, to, other);
        else bpair<L0, BP_PLAIN, 1, false, false>(B, s, l, to, other);
    }
}

// z = P V(P r), P removing the mean of every fluid component of the grids
// with more than one (r in place).
void bmg_vcycle(pg_batch* B, cudaStream_t s, int nsmooth) {
    BatchMg& M = *B->mg;
    pocket_project(s, B->r, M.pockets, &B->state[0].done, sizeof(BState));
    int deepest = 0;  // levels [0, deepest) have grids that smooth there
    while (deepest < M.nlev && M.nsmoothing[deepest]) ++deepest;
    for (int l = 0; l < deepest; ++l) {
        if (l == 0) bmg_down<true>(B, s, l, nsmooth);
        else bmg_down<false>(B, s, l, nsmooth);
    }
    BTail v;
    for (int l = 0; l < kBmgMaxLevels; ++l) {
        v.info[l] = M.info[l];
        v.wx[l] = M.wx[l];
        v.wy[l] = M.wy[l];
        v.invd[l] = M.invd[l];
        v.f[l] = l == 0 ? B->r : M.f[l];
        v.e[l] = l == 0 ? B->z : M.e[l];
    }
    v.flags = B->flags;
    v.dt = M.dt;
    v.nsmooth = nsmooth;
    PG_LAUNCH(KK_MG_COARSE, s,
              k_bmg_tail<<<B->n, kBmgTailThreads, 5 * sizeof(float) * M.tail_cells, s>>>(v, B->state));
    for (int l = deepest - 1; l >= 0; --l) {
        if (l == 0) bmg_up<true>(B, s, l, nsmooth);
        else bmg_up<false>(B, s, l, nsmooth);
    }
    // No grid smooths on level 0 (all are small): the z.r partials alone.
    if (deepest == 0) bpair<true, BP_PLAIN, 1, true, false>(B, s, 0, B->ap, B->z);
    pocket_project(s, B->z, M.pockets, &B->state[0].done, sizeof(BState));
}

void bmg_spmv(pg_batch* B, cudaStream_t s, float dt) {
    BatchMg& M = *B->mg;
    PG_LAUNCH(KK_CG_SPMV, s,
              k_bmg_spmv<<<march_blocks(M.ncg), kMarchThreads, 0, s>>>(M.info[0], M.cg_strips, M.ncg, B->state, B->z, B->p0,
                                                                       B->p1, B->ap, B->flags, dt, M.partials));
}

void bmg_update(pg_batch* B, cudaStream_t s, float* x) {
    BatchMg& M = *B->mg;
    const int vec = ((uintptr_t)x & 15) == 0;  // (the batch's own fields are)
    PG_LAUNCH(KK_CG_UPDATE, s,
              k_bmg_update<<<(M.nchunk + 7) / 8, 256, 0, s>>>(M.chunks, M.nchunk, B->state, x, B->r, B->p0, B->p1, B->ap,
                                                              vec, M.partials));
}

void bmg_init(pg_batch* B, cudaStream_t s, float* x) {
    BatchMg& M = *B->mg;
    const int vec = ((uintptr_t)x & 15) == 0;
    PG_LAUNCH(KK_CG_INIT, s,
              k_bmg_init<<<(M.nchunk + 7) / 8, 256, 0, s>>>(M.chunks, M.nchunk, x, B->r, B->b, vec, M.partials));
}

const double* bmg_partials(const pg_batch* B) { return B->mg->partials; }
const int2* bmg_spmv_range(const pg_batch* B) { return B->mg->cg_range; }
const int2* bmg_update_range(const pg_batch* B) { return B->mg->chunk_range; }

void bmg_rz_finalize(pg_batch* B, cudaStream_t s, int first) {
    BatchMg& M = *B->mg;
    PG_LAUNCH(KK_STEP_MISC, s, k_bmg_rz_finalize<<<B->n, 128, 0, s>>>(M.info[0], B->state, M.partials, B->n, first));
}

}  // namespace pg
