// pg_wavelet_pass.cuh -- the mirror-sampled 1D wavelet passes
// (panopaea/src/math/wavelet/mod.rs:52-112) over every line of a 2D block,
// out of place, for lines of at least twice the filter length.
//
// GB300 runs FP64 at 1/64 of its FP32 rate (two operations per clock and
// SM), so a pass is bound by its FP64 operations long before HBM: a thread
// owns P neighbouring output pairs, the taps are compile-time constants, and
// everything the sums do not need is left out without changing a bit --
//   - zero taps (a product x * 0 adds +-0 to a sum that is never -0) as long
//     as the samples are finite: a window with an infinity or a NaN takes
//     the loop over all taps;
//   - a product is formed once per (sample, |tap|) and used for every output
//     that has it (the sign goes into an addition or a subtraction);
//   - the addition to the initial 0 (only the sign of a zero is set).
// A bior 2.2 output pair then takes 11 operations instead of 24, analysis
// and synthesis alike.  Measured at 1024^2 (ncu): an analysis pass 19-20 us
// (a thread per sample over all taps: 32), a synthesis pass 18-20 us (a
// thread per sample gathering and sorting its contributions: 40); with the
// copies to the scratch array gone, fwt_2d + ifwt_2d of 5 levels 378 -> 166
// us per pair of transforms.
#pragma once

#include "pg_internal.cuh"
#include "pg_wavelet_border.cuh"

namespace pg {
namespace wv {

template <int W> struct Bank {
    static constexpr WFilter F = kFilters[W];
    static constexpr int n = F.n, fh = n / 2, q = fh - 1;
    static constexpr int TM = fh / 2;      // synthesis: samples m - TM .. m + TM feed outputs 2m, 2m + 1
    static constexpr int XW = n - 2;       // analysis: window of P pairs = 2 P + XW samples from 2 i0 - q
};

__device__ __forceinline__ bool nonfinite(double v) {
    return (unsigned)(__double2hiint(v) & 0x7ff00000) == 0x7ff00000u;
}
// 0.0 + p without an FP64 operation: only a negative zero changes.
__device__ __forceinline__ double from_zero(double p) {
    return __double_as_longlong(p) == (long long)0x8000000000000000ull ? 0.0 : p;
}

// acc = x * c + acc (fold of mod.rs:60-77); `begun` is a compile-time fact
// once the tap loop is unrolled.
template <bool ALL> __device__ __forceinline__ void tap(double x, double c, double& acc, bool& begun) {
    if (ALL) {
        acc = __dadd_rn(__dmul_rn(x, c), acc);
        return;
    }
    if (c == 0.0) return;
    const double p = __dmul_rn(x, c < 0.0 ? -c : c);
    if (!begun)
        acc = from_zero(c < 0.0 ? -p : p);
    else
        acc = c < 0.0 ? __dsub_rn(acc, p) : __dadd_rn(acc, p);
    begun = true;
}

// x[k]: sample 2 i0 - q + k of the mirrored line.
template <int W, int P, bool ALL>
__device__ __forceinline__ void down_eval(const double (&x)[2 * P + Bank<W>::XW], double (&lo)[P], double (&hi)[P]) {
    constexpr WFilter F = Bank<W>::F;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        double a = 0.0, b = 0.0;
        bool sa = false, sb = false;
#pragma unroll
        for (int f = 0; f < F.n; ++f) {
            tap<ALL>(x[2 * i + f], F.down_low[F.n - 1 - f], a, sa);
            tap<ALL>(x[2 * i + f], F.down_high[F.n - 1 - f], b, sb);
        }
        lo[i] = a;
        hi[i] = b;
    }
}
template <int W, int P>
__device__ __forceinline__ void down_pairs(const double (&x)[2 * P + Bank<W>::XW], double (&lo)[P], double (&hi)[P]) {
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 2 * P + Bank<W>::XW; ++k) bad |= nonfinite(x[k]);
    if (bad)
        down_eval<W, P, true>(x, lo, hi);
    else
        down_eval<W, P, false>(x, lo, hi);
}

// The contribution a * low[f] + b * high[f] (mod.rs:104-109).
template <bool ALL> __device__ __forceinline__ double both(double a, double b, double cl, double ch) {
    if (ALL) return __dadd_rn(__dmul_rn(a, cl), __dmul_rn(b, ch));
    if (ch == 0.0) {
        const double p = __dmul_rn(a, cl < 0.0 ? -cl : cl);
        return cl < 0.0 ? -p : p;
    }
    const double h = __dmul_rn(b, ch < 0.0 ? -ch : ch);
    if (cl == 0.0) return ch < 0.0 ? -h : h;
    const double l = __dmul_rn(a, cl < 0.0 ? -cl : cl);
    if (cl < 0.0 && ch < 0.0) return -__dadd_rn(l, h);
    if (cl < 0.0) return __dsub_rn(h, l);
    return ch < 0.0 ? __dsub_rn(l, h) : __dadd_rn(l, h);
}

// a[k], b[k]: samples m0 - TM + k of the two halves, wrapped over the half
// length.  The reference scatters in increasing sample order, so a sample
// that wrapped down to the line's start is added first and one that wrapped
// up to its end last: a rotation of the window order, which is that order
// everywhere else.  EDGE: some thread of the warp has a wrapped sample; the
// same products and sums, the addends picked by the rotation.
template <int W, int P, bool ALL, bool EDGE>
__device__ __forceinline__ void up_eval(const double (&a)[P + 2 * Bank<W>::TM], const double (&b)[P + 2 * Bank<W>::TM],
                                        double (&out)[2 * P], int m0, int half) {
    constexpr WFilter F = Bank<W>::F;
    constexpr int TM = Bank<W>::TM, q = Bank<W>::q, T = 2 * TM + 1;
#pragma unroll
    for (int j = 0; j < 2 * P; ++j) {
        const int p = j / 2, odd = j & 1;
        double v[T];
        int K = 0, below = 0, above = 0;  // addends (a compile-time count); those wrapped up / down
#pragma unroll
        for (int t = -TM; t <= TM; ++t) {
            const int f = q + odd - 2 * t;
            if (f < 0 || f >= F.n) continue;
            if (!ALL && F.up_low[f] == 0.0 && F.up_high[f] == 0.0) continue;
            v[K++] = both<ALL>(a[p + t + TM], b[p + t + TM], F.up_low[f], F.up_high[f]);
            if (EDGE) {
                below += m0 + p + t < 0;
                above += m0 + p + t >= half;
            }
        }
        const int first = EDGE ? (above ? K - above : below) : 0;
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < T; ++k) {
            if (k >= K) continue;
            double w = v[k];
            if (EDGE) {
                const int at = first + k >= K ? first + k - K : first + k;
#pragma unroll
                for (int c = 0; c < T; ++c)
                    if (c < K && at == c) w = v[c];
            }
            s = ALL || k ? __dadd_rn(s, w) : from_zero(w);
        }
        out[j] = s;
    }
}
// Called by whole warps.
template <int W, int P>
__device__ __forceinline__ void up_pairs(const double (&a)[P + 2 * Bank<W>::TM], const double (&b)[P + 2 * Bank<W>::TM],
                                         double (&out)[2 * P], int m0, int half) {
    constexpr int TM = Bank<W>::TM;
    const bool edge = TM > 0 && (m0 < TM || m0 + P + TM > half);
    bool bad = false;
#pragma unroll
    for (int k = 0; k < P + 2 * TM; ++k) bad |= nonfinite(a[k]) | nonfinite(b[k]);
    if (__any_sync(0xffffffffu, bad))
        up_eval<W, P, true, true>(a, b, out, m0, half);
    else if (__any_sync(0xffffffffu, edge))
        up_eval<W, P, false, true>(a, b, out, m0, half);
    else
        up_eval<W, P, false, false>(a, b, out, m0, half);
}

// mod.rs:38-48 for lines of at least the window's length on either side
__device__ __forceinline__ int mirror_index(int k, int len) { return k < 0 ? -k : (k >= len ? 2 * len - 1 - k : k); }

// ---------------------------------------------------------------------------
// Passes along y: lanes across x (coalesced rows), a thread per column and P
// pairs of rows, the window straight from global memory.
template <int W, int P>
__global__ void __launch_bounds__(256) k_wdown_y(const double* __restrict__ src, double* __restrict__ dst, int len,
                                                 int cols, i64 stride) {
    constexpr int XN = 2 * P + Bank<W>::XW, q = Bank<W>::q;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int half = len / 2, i0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * P;
    if (x >= cols || i0 >= half) return;
    double v[XN], lo[P], hi[P];
#pragma unroll
    for (int k = 0; k < XN; ++k) v[k] = src[mirror_index(min(2 * i0 - q + k, len + q), len) * stride + x];
    down_pairs<W, P>(v, lo, hi);
#pragma unroll
    for (int i = 0; i < P; ++i)
        if (i0 + i < half) {
            dst[(i0 + i) * stride + x] = lo[i];
            dst[(half + i0 + i) * stride + x] = hi[i];
        }
}

template <int W, int P>
__global__ void __launch_bounds__(256) k_wup_y(const double* __restrict__ src, double* __restrict__ dst, int len,
                                               int cols, i64 stride) {
    constexpr int TM = Bank<W>::TM, N = P + 2 * TM;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int half = len / 2, m0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * P;
    if (m0 >= half) return;  // the whole warp
    double a[N], b[N], out[2 * P];
    const int xc = min(x, cols - 1);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        int i = min(m0 - TM + k, half + TM - 1);  // past that only outputs that are not stored
        i = i < 0 ? i + half : (i >= half ? i - half : i);
        a[k] = src[i * stride + xc];
        b[k] = src[(i + half) * stride + xc];
    }
    up_pairs<W, P>(a, b, out, m0, half);
    if (x >= cols) return;
#pragma unroll
    for (int j = 0; j < 2 * P; ++j)
        if (2 * m0 + j < len) dst[(2 * m0 + j) * stride + x] = out[j];
}

// ---------------------------------------------------------------------------
// Passes along x: a warp covers 32 P output pairs of a row, or of several
// short rows (G lanes, a power of two >= 4, per row); the window goes through
// shared memory so that loads and stores are whole lines, at indices padded
// by one per thread's share (odd strides: no bank conflicts).
template <int S> __device__ __forceinline__ int padded(int k) { return S > 2 ? k + k / S : k; }
constexpr int kPassSm = 416;  // doubles per warp (the largest: synthesis, G = 4, P = 4, 10 taps: 16 x 26)

template <int W, int P>
__global__ void __launch_bounds__(256) k_wdown_x(const double* __restrict__ src, double* __restrict__ dst, int rows,
                                                 int len, i64 stride, int glog, int segs) {
    constexpr int XN = 2 * P + Bank<W>::XW, q = Bank<W>::q;
    __shared__ double sm_all[8][kPassSm];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* sm = sm_all[warp];
    const int G = 1 << glog, per = 32 >> glog;  // rows per warp
    const int item = blockIdx.x * 8 + warp, seg = item % segs, row0 = item / segs * per;
    if (row0 >= rows) return;
    const int half = len / 2, s0 = seg * G * P;  // first pair of the segment
    const int in_n = 2 * G * P + Bank<W>::XW;    // samples of a row's window
    const int cells = padded<2 * P>(in_n) + 1;   // its place in shared memory
    for (int r = 0; r < per && row0 + r < rows; ++r)
        for (int k = lane; k < in_n; k += 32)
            sm[r * cells + padded<2 * P>(k)] =
                src[(row0 + r) * stride + mirror_index(min(2 * s0 - q + k, len + q), len)];
    __syncwarp();
    const int slot = lane >> glog, g = lane & (G - 1);
    double v[XN], lo[P], hi[P];
#pragma unroll
    for (int k = 0; k < XN; ++k) v[k] = sm[slot * cells + padded<2 * P>(2 * P * g + k)];
    down_pairs<W, P>(v, lo, hi);
    __syncwarp();
    const int oc = padded<P>(G * P) + 1;  // one band's place
#pragma unroll
    for (int i = 0; i < P; ++i) {
        sm[(2 * slot) * oc + padded<P>(P * g + i)] = lo[i];
        sm[(2 * slot + 1) * oc + padded<P>(P * g + i)] = hi[i];
    }
    __syncwarp();
    const int nout = min(G * P, half - s0);
    for (int r = 0; r < per && row0 + r < rows; ++r)
        for (int k = lane; k < nout; k += 32) {
            dst[(row0 + r) * stride + s0 + k] = sm[(2 * r) * oc + padded<P>(k)];
            dst[(row0 + r) * stride + half + s0 + k] = sm[(2 * r + 1) * oc + padded<P>(k)];
        }
}

template <int W, int P>
__global__ void __launch_bounds__(256) k_wup_x(const double* __restrict__ src, double* __restrict__ dst, int rows,
                                               int len, i64 stride, int glog, int segs) {
    constexpr int TM = Bank<W>::TM, N = P + 2 * TM;
    __shared__ double sm_all[8][kPassSm];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* sm = sm_all[warp];
    const int G = 1 << glog, per = 32 >> glog;
    const int item = blockIdx.x * 8 + warp, seg = item % segs, row0 = item / segs * per;
    if (row0 >= rows) return;
    const int half = len / 2, s0 = seg * G * P;
    const int in_n = G * P + 2 * TM;
    const int cells = padded<P>(in_n) + 1;
    for (int r = 0; r < per && row0 + r < rows; ++r)
        for (int k = lane; k < in_n; k += 32) {
            int i = min(s0 - TM + k, half + TM - 1);
            i = i < 0 ? i + half : (i >= half ? i - half : i);
            sm[(2 * r) * cells + padded<P>(k)] = src[(row0 + r) * stride + i];
            sm[(2 * r + 1) * cells + padded<P>(k)] = src[(row0 + r) * stride + half + i];
        }
    __syncwarp();
    const int slot = lane >> glog, g = lane & (G - 1), m0 = s0 + P * g;
    double a[N], b[N], out[2 * P];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const bool own = m0 < half && row0 + slot < rows;
        a[k] = own ? sm[(2 * slot) * cells + padded<P>(P * g + k)] : 0.0;
        b[k] = own ? sm[(2 * slot + 1) * cells + padded<P>(P * g + k)] : 0.0;
    }
    up_pairs<W, P>(a, b, out, m0, half);
    __syncwarp();
    const int oc = padded<2 * P>(2 * G * P) + 1;
    if (m0 < half && row0 + slot < rows) {
#pragma unroll
        for (int j = 0; j < 2 * P; ++j) sm[slot * oc + padded<2 * P>(2 * P * g + j)] = out[j];
    }
    __syncwarp();
    const int nout = min(2 * G * P, len - 2 * s0);
    for (int r = 0; r < per && row0 + r < rows; ++r)
        for (int k = lane; k < nout; k += 32)
            dst[(row0 + r) * stride + 2 * s0 + k] = sm[r * oc + padded<2 * P>(k)];
}

// ---------------------------------------------------------------------------
// Launches.  False where the pass does not apply (lines shorter than twice
// the filter, where a window could wrap onto itself; sizes beyond 31 bits).
struct PassShape {
    i64 lines, len, stride;  // `len` samples of each of `lines` lines; the block's row stride
    bool along_x;
};

// The blocks (256 threads) of a pass with P pairs per thread.
struct PassGrid {
    int glog = 2, segs = 0;  // along x: log2 of the lanes per row, segments per row
    i64 x, y = 1;
    PassGrid(const PassShape& s, int P) {
        const i64 groups = (s.len / 2 + P - 1) / P;
        if (s.along_x) {
            while (glog < 5 && (1 << glog) < groups) ++glog;
            segs = (int)((groups + (1 << glog) - 1) >> glog);
            const int per = 32 >> glog;
            x = ((s.lines + per - 1) / per * segs + 7) / 8;
        } else {
            x = (s.lines + 31) / 32;
            y = (groups + 7) / 8;
        }
    }
};

// Pairs per thread, four or one.  Four share products (bior 2.2: 11 FP64
// operations a pair, 14 alone): kFourGain, in percent, is what that gives with
// every SM busy (4096^2).  Against it stands that blocks of four times the work
// fill the SMs less evenly -- a pass takes as long as the SM with the most
// blocks, FP64 units being its bound -- and that a thread's FP64 chain is
// longer, which shows while an SM has few blocks.  Measured, one / four pairs,
// two analysis and two synthesis passes, us: 384^2 bior 2.2 15.6 / 23.2; 512^2
// (one block per SM) haar 11.5 / 13.1, bior 2.2 24.5 / 23.6; 640^2 (two, on a
// third of the SMs) haar 14.2 / 17.7, bior 2.2 33.2 / 38.5; 1024^2 haar 24.0 /
// 28.1, bior 2.2 67.6 / 69.1, bior 2.4 104 / 110; 2048^2 haar 73 / 76, bior 2.2
// 241 / 218, bior 2.4 377 / 357; 4096^2 haar 278 / 273, bior 2.2 938 / 816.
constexpr int kFourGain[5] = {102, 106, 115, 110, 103};  // by PG_WAVELET_*
inline int pass_pairs(int wavelet, const PassShape& s, int num_sms) {
    auto blocks = [&](int pairs) {  // on the SM that gets most
        const PassGrid g(s, pairs);
        return (g.x * g.y + num_sms - 1) / num_sms;
    };
    const i64 four = blocks(4);
    return 4 * four * 102 <= blocks(1) * kFourGain[wavelet] && (four >= 4 || kFourGain[wavelet] >= 110) ? 4 : 1;
}

template <int W, int P> inline void pass_launch(cudaStream_t st, bool down, const double* src, double* dst, const PassShape& s) {
    const PassGrid g(s, P);
    const dim3 nb((unsigned)g.x, (unsigned)g.y);
    if (s.along_x) {
        if (down)
            k_wdown_x<W, P><<<nb, 256, 0, st>>>(src, dst, (int)s.lines, (int)s.len, s.stride, g.glog, g.segs);
        else
            k_wup_x<W, P><<<nb, 256, 0, st>>>(src, dst, (int)s.lines, (int)s.len, s.stride, g.glog, g.segs);
    } else {
        if (down)
            k_wdown_y<W, P><<<nb, 256, 0, st>>>(src, dst, (int)s.len, (int)s.lines, s.stride);
        else
            k_wup_y<W, P><<<nb, 256, 0, st>>>(src, dst, (int)s.len, (int)s.lines, s.stride);
    }
}

inline bool pass_run(cudaStream_t st, int num_sms, int wavelet, bool down, const double* src, double* dst,
                     const PassShape& s) {
    const i64 most = (i64)1 << 30;
    if (wavelet < 0 || wavelet > 4 || s.len < 2 * kFilters[wavelet].n || s.len > most || s.lines > most) return false;
    if (!s.along_x && (s.len / 2 + 7) / 8 > 65535) return false;  // grid.y
    if (s.along_x && s.lines * ((s.len + 7) / 8) > most) return false;
    const bool four = pass_pairs(wavelet, s, num_sms) == 4;
#define PG_WPASS(W)                                              \
    case W:                                                      \
        if (four)                                                \
            pass_launch<W, 4>(st, down, src, dst, s);            \
        else                                                     \
            pass_launch<W, 1>(st, down, src, dst, s);            \
        break;
    switch (wavelet) {
        PG_WPASS(0)
        PG_WPASS(1)
        PG_WPASS(2)
        PG_WPASS(3)
        PG_WPASS(4)
    }
#undef PG_WPASS
    return true;
}

}  // namespace wv
}  // namespace pg
