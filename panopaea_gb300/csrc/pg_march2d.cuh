// pg_march2d.cuh -- red-black smoothing of 2D multigrid levels by warps that
// march down strips of 64 columns, for batches of grids (pg_batch_mg.cu) and
// single ones (pg_mg.cu).
#pragma once
#include <algorithm>
#include <vector>

#include "pg_internal.cuh"

namespace pg {

// A strip: up to 64 columns of one grid from the even column x0 on, marched
// down rows [y0, y1) by one warp that holds two neighbouring columns per lane.
struct Strip {
    int grid, y0, y1, x0;
};

// Two neighbouring values of a row; VEC: the pair is 8-byte aligned and whole.
template <bool VEC> __device__ __forceinline__ float2 ld2(const float* p, bool a, bool b) {
    float2 v = make_float2(0.f, 0.f);
    if (VEC) {
        if (a) v = *reinterpret_cast<const float2*>(p);
    } else {
        if (a) v.x = p[0];
        if (b) v.y = p[1];
    }
    return v;
}

template <bool VEC> __device__ __forceinline__ void st2(float* p, float2 v, bool a, bool b) {
    if (VEC) {
        if (a) *reinterpret_cast<float2*>(p) = v;
    } else {
        if (a) p[0] = v.x;
        if (b) p[1] = v.y;
    }
}

// Two flag bytes, kept apart until they are used (a load must not be waited
// for where it is issued).
struct Flag2 {
    unsigned a, b;
    template <bool VEC> __device__ __forceinline__ void load(const uint8_t* p, bool va, bool vb) {
        a = b = 0;
        if (VEC) {
            if (va) a = *reinterpret_cast<const unsigned short*>(p);
        } else {
            if (va) a = p[0];
            if (vb) b = p[1];
        }
    }
    // the second cell's in bits 8 and up
    template <bool VEC> __device__ __forceinline__ unsigned both() const { return VEC ? a : a | b << 8; }
};

// A grid's level: its dims, its first cell in the level's arrays, and the same
// of the next level (0 if none).
struct MarchLevel {
    int h, w;
    i64 off;
    int ch, cw;
    i64 coff;
};

// A level's arrays.
struct MarchView {
    const float* wx;
    const float* wy;
    const float* invd;
    const float* f;
    const uint8_t* flags;  // level 0
    const float* ec;       // next level's correction (prolongation)
    float* fc;             // next level's right-hand side (restriction)
    float dt;
};

constexpr int kMarchThreads = 128;  // four strips per block
inline int march_blocks(int n) { return (n + kMarchThreads / 32 - 1) / (kMarchThreads / 32); }

// Strips of a level: `step` columns apart, chunks of up to `rows` rows (an even
// number).
inline void march_strips(int grid, int h, int w, int step, int rows, std::vector<Strip>& st) {
    const int per = (h + rows - 1) / rows, rc = ((h + per - 1) / per + 1) & ~1;
    for (int y0 = 0; y0 < h; y0 += rc)
        for (int x0 = 0;; x0 += step) {
            st.push_back(Strip{grid, y0, std::min(y0 + rc, h), x0});
            if (x0 + 64 >= w) break;
        }
}

enum { BP_PLAIN = 0, BP_SELF = 1, BP_PROLONG = 2 };

// s + weight * neighbour over a cell's open faces (x-, x+, y-, y+).
__device__ __forceinline__ float nb_sum(float s, float wl, float wr, float wu, float wd, float nl, float nr, float nu,
                                        float nd) {
    if (wl != 0.f) s = fmaf(wl, nl, s);
    if (wr != 0.f) s = fmaf(wr, nr, s);
    if (wu != 0.f) s = fmaf(wu, nu, s);
    if (wd != 0.f) s = fmaf(wd, nd, s);
    return s;
}

// What a lane holds of a row: e and f of its two cells, and their flags
// (level 0) or weights and 1 / diagonal (coarser levels).
template <bool L0> struct BRow {
    float2 e, f;
    Flag2 raw;  // as loaded; fl: both
    unsigned fl;
    float2 wx, wy, inv;
    float wr;   // the second cell's x+ weight, from the next lane
    float ec;   // as loaded: the correction to prolong
};

// One red-black pair over a strip: the first colour of row y (from the old
// values of the rows around it), then the second colour of row y - 1 (from
// the new ones), which finishes that row; with REST the residual of row y - 2
// follows and is summed to the next level, with RZ the finished row's z.r and
// sum(z).  C1: the parity of x + y of the first colour.  FA: the first
// colour in this row is the lane's first cell.
template <bool L0, int MODE, int C1, bool RZ, bool REST, bool VEC> struct March {
    const MarchView& v;
    const MarchLevel& L;
    const float* __restrict__ ein;
    float* __restrict__ eout;
    int lane, x, y0, y1;
    bool va, vb, own, ownb;
    float tab;  // lane f: 1 / diagonal of a cell with face-open bits f (level 0)
    i64 at;     // index of the lane's first cell in the next row to fetch
    int next;   // that row
    int stop;   // the last row needed
    BRow<L0> r[5];  // rows y - 3 .. y + 1
    float rsum = 0.f;
    Acc<float> acc, zs;

    __device__ __forceinline__ March(const MarchView& v_, const MarchLevel& L_, const Strip& S, const float* ein_, float* eout_)
        : v(v_), L(L_), ein(ein_), eout(eout_) {
        lane = threadIdx.x & 31;
        x = S.x0 + 2 * lane;
        y0 = S.y0;
        y1 = S.y1;
        va = x < L.w;
        vb = x + 1 < L.w;
        const int lo = S.x0 ? S.x0 + 4 : 0, hi = S.x0 + 64 >= L.w ? L.w : S.x0 + 60;
        own = x >= lo && x < hi;
        ownb = own && vb;
        const int n = __popc(lane & 15);
        tab = L0 && n ? __frcp_rn((float)n * v.dt) : 0.f;
    }

    // Row `next` (zeros outside the grid, so that no weight points there).
    __device__ __forceinline__ BRow<L0> fetch() {
        BRow<L0> q;
        q.e = q.f = q.wx = q.wy = q.inv = make_float2(0.f, 0.f);
        q.fl = q.raw.a = q.raw.b = 0;
        q.wr = q.ec = 0.f;
        if (next >= 0 && next <= stop) {  // uniform per warp
            q.f = ld2<VEC>(v.f + at, va, vb);
            if (L0) {
                q.raw.template load<VEC>(v.flags + at, va, vb);
            } else {
                q.wx = ld2<VEC>(v.wx + at, va, vb);
                q.wy = ld2<VEC>(v.wy + at, va, vb);
                q.inv = ld2<VEC>(v.invd + at, va, vb);
            }
            if (MODE != BP_SELF) q.e = ld2<VEC>(ein + at, va, vb);
            if (MODE == BP_PROLONG && va) q.ec = v.ec[L.coff + (i64)(next >> 1) * L.cw + (x >> 1)];
        }
        ++next;
        at += L.w;
        return q;
    }

    __device__ __forceinline__ void push(const BRow<L0>& q) {
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = r[k + 1];
        r[4] = q;
        if (MODE == BP_PROLONG) {
            r[4].e.x += q.ec;
            r[4].e.y += q.ec;
        }
        if (L0) {
            r[4].fl = q.raw.template both<VEC>();
        } else {
            const float n = __shfl_down_sync(0xffffffffu, q.wx.x, 1);
            r[4].wr = lane < 31 ? n : 0.f;
        }
    }

    // Weights of the first (A) or second cell of row k.
    template <bool A> __device__ __forceinline__ void weights(int k, float& wl, float& wr, float& wu, float& wd) const {
        if (L0) {
            const unsigned f = A ? r[k].fl : r[k].fl >> 8;
            wl = (f & XLO) ? v.dt : 0.f;
            wr = (f & XHI) ? v.dt : 0.f;
            wu = (f & YLO) ? v.dt : 0.f;
            wd = (f & YHI) ? v.dt : 0.f;
        } else {
            wl = A ? r[k].wx.x : r[k].wx.y;
            wr = A ? r[k].wx.y : r[k].wr;
            wu = A ? r[k].wy.x : r[k].wy.y;
            wd = A ? r[k + 1].wy.x : r[k + 1].wy.y;
        }
    }
    template <bool A> __device__ __forceinline__ float inv(int k) const {
        if (L0) return __shfl_sync(0xffffffffu, tab, A ? r[k].fl : r[k].fl >> 8);
        return A ? r[k].inv.x : r[k].inv.y;
    }
    // The four neighbours' values.
    template <bool A> __device__ __forceinline__ void around(int k, float& nl, float& nr, float& nu, float& nd) const {
        if (A) {
            nl = __shfl_up_sync(0xffffffffu, r[k].e.y, 1);
            nr = r[k].e.y;
        } else {
            nl = r[k].e.x;
            nr = __shfl_down_sync(0xffffffffu, r[k].e.x, 1);
        }
        nu = A ? r[k - 1].e.x : r[k - 1].e.y;
        nd = A ? r[k + 1].e.x : r[k + 1].e.y;
    }
    template <bool A> __device__ __forceinline__ float updated(int k) const {
        float wl, wr, wu, wd, nl, nr, nu, nd;
        weights<A>(k, wl, wr, wu, wd);
        around<A>(k, nl, nr, nu, nd);
        return nb_sum(A ? r[k].f.x : r[k].f.y, wl, wr, wu, wd, nl, nr, nu, nd) * inv<A>(k);
    }
    template <bool A> __device__ __forceinline__ float residual(int k) const {
        float wl, wr, wu, wd, nl, nr, nu, nd;
        weights<A>(k, wl, wr, wu, wd);
        around<A>(k, nl, nr, nu, nd);
        const float c = A ? r[k].e.x : r[k].e.y;
        return (A ? r[k].f.x : r[k].f.y) - nb_sum(0.f, wl, wr, wu, wd, c - nl, c - nr, c - nu, c - nd);
    }

    template <bool FA> __device__ __forceinline__ void step(int y) {
        float n;
        if (MODE == BP_SELF) {
            const float i = inv<FA>(3), f = FA ? r[3].f.x : r[3].f.y;
            n = i != 0.f ? f * i : 0.f;
        } else {
            n = updated<FA>(3);
        }
        (FA ? r[3].e.x : r[3].e.y) = n;
        const float m = updated<FA>(2);  // (the colours swap cells from row to row)
        (FA ? r[2].e.x : r[2].e.y) = m;
        if (y - 1 >= y0 && y - 1 < y1) {  // uniform per warp
            st2<VEC>(eout + (at - 5 * (i64)L.w), r[2].e, own, ownb);  // (fetched: rows up to y + 3)
            if (RZ) {
                if (own) {
                    acc.add(r[2].e.x * r[2].f.x);
                    zs.add(r[2].e.x);
                }
                if (ownb) {
                    acc.add(r[2].e.y * r[2].f.y);
                    zs.add(r[2].e.y);
                }
            }
        }
        if (REST && y - 2 >= y0) {
            const float a = residual<true>(1), b = residual<false>(1);
            if ((y & 1) == 0) rsum = a + b;
            else {
                rsum += a;
                rsum += b;
                const int Y = (y - 2) >> 1;
                if (Y < L.ch && 2 * Y < y1 && own) v.fc[L.coff + (i64)Y * L.cw + (x >> 1)] = rsum;
            }
        }
    }

    __device__ __forceinline__ void run() {
        int y = y0 - (REST ? 2 : 1);
        const int last = y0 + ((y1 - y0 + 1) & ~1) + (REST ? 1 : 0);
        constexpr bool FA = REST ? C1 == 0 : C1 == 1;
        next = y - 1;
        stop = min(L.h - 1, last + 1);
        at = L.off + (i64)next * L.w + x;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            r[k].e = r[k].f = r[k].wx = r[k].wy = r[k].inv = make_float2(0.f, 0.f);
            r[k].fl = r[k].raw.a = r[k].raw.b = 0;
            r[k].wr = r[k].ec = 0.f;
        }
        push(fetch());
        push(fetch());
        BRow<L0> q0 = fetch(), q1 = fetch();  // two rows ahead
        for (; y < last; y += 2) {
            push(q0);
            q0 = fetch();
            step<FA>(y);
            push(q1);
            q1 = fetch();
            step<!FA>(y + 1);
        }
    }
};

}  // namespace pg
