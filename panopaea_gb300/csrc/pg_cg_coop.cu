// pg_cg_coop.cu -- conjugate gradient (pcg.rs:14-82) on small double grids as
// ONE cooperative kernel: every block keeps its cells' x, r, p and A p in
// registers over all iterations, and the two dot products of an iteration
// are the only points where blocks wait for one another.
//
// What bounds a small solve is latency: the two kernels of an iteration took
// 16 us on a 128^2 grid whose arithmetic is 1 us -- launch, state load,
// reduction tree, ticket, fold by the last block, twice.  Here an iteration is
//   p = z + beta p on the block's cells and on one row (plane) of neighbours
//   on either side, whose r and old p are read from global memory; A p and p.Ap;
//   exchange; x += alpha p, r -= alpha Ap, ||r||inf and z.r; exchange.
// The exchange is an all-gather: a block writes its partial sums as 64-bit
// words that each carry the exchange's number, every block polls every
// block's words and folds them in the same order -- one trip through L2, no
// atomics, no second broadcast.  The words follow a fence, so the r and p
// rows that the neighbours read next are visible behind them.  Every poll is
// bounded; a block that gives up sets PG_TIMEOUT and leaves, and the others
// give up in turn.
//
// Per-cell arithmetic is that of k_cg_spmv and k_cg_update; the FP64 sums run
// in another order.  (Float grids keep the loop: sums taken in another order
// there move alpha by an FP32 ulp now and then, and 100 iterations on the
// residual by 5e-6 of its norm, no closer to the exact one.)
//
// Measured, plain CG (Jacobi) per iteration, the loop of two kernels against
// this: 128^2 13.9 / 8.0 us (17.2 / 8.2), 384^2 21.4 / 13.3 (37.0 / 14.1), 550 x
// 560 32.2 / 18.3 (56.3 / 19.8), 64^3 39.9 / 23.6 (65.7 / 25.7).  Of the 8.0 us
// each exchange is about 3 (FP64 folds and a division at 60 to 100 cycles per
// dependent operation, the trip through L2, fences).  Above kCoopMaxCells
// cells per thread the loop is at its memory traffic and stays, and so it does
// where rows or planes are large beside a block's cells (coop_pays).
#include <algorithm>
#include <cstdlib>

#include "pg_cg.cuh"
#include "pg_tma.cuh"

namespace pg {

namespace {

constexpr int kCoopMaxThreads = 512;
constexpr int kCoopMaxCells = 8;          // cells per thread, in registers
constexpr int kCoopMaxBlocks = 256;
constexpr int kCoopSmemMax = 200 * 1024;  // p of the block's cells and of the rows around them

// One block's words of an exchange: {number, half of a double} each; the
// first number's top bit flags a non-finite value.  256 bytes apart, so that
// the blocks' polls spread over the L2's slices (packed, their polling held up
// the very words and fences they waited for: 12.5 us per iteration at 128^2
// instead of 8.2).
struct alignas(256) CoopSlot {
    unsigned long long w[4];
    unsigned long long pad[28];
};

struct CoopArgs {
    double *x, *r, *p0, *p1, *ap;
    const double* b;
    const uint8_t* flags;
    int n, w, H, C;  // cells; row length; cells of a row (2D) or plane (3D); cells per block
    double dt, thr, rel_tol;
    i64 max_iter;
    CgState* st;
    CoopSlot* slots;  // 2 x gridDim.x, used in turn
};

// (Each word carries its tag, so a pair need not arrive as one.)
__device__ __forceinline__ void coop_ld2(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void coop_st2(unsigned long long* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}

// z = M^-1 r at a cell with face-open bits f (as zof).  inv_diag[k]: 1 / (k dt),
// formed once per block: an FP64 reciprocal for every cell and halo cell took
// half of a Jacobi iteration (64^3 41.5 us, 26.0 with the table).
template <int PM> __device__ __forceinline__ double coop_z(double rv, unsigned f, const double* inv_diag) {
    if (PM == PM_JACOBI) return f ? rv * inv_diag[__popc(f)] : 0.0;
    return rv;
}

struct CoopShared {
    double fold[kCoopMaxThreads + 32];
    double v[kCoopMaxBlocks], m[kCoopMaxBlocks];
    double sum, max;
    double scale;  // alpha or beta for the block
    int stop, bad;
    double inv_diag[8];  // Jacobi
};

// Sum and, with MAX, maximum (>= 0) of every thread of the grid, the number of
// the exchange (1, 2, ...) given; in sh.sum, sh.max and sh.bad, for thread 0 of
// every block.  DATA: global memory written before the exchange is read by
// other blocks after it (two fences: 1000 to 5000 cycles each, so only the
// second exchange of an iteration, which covers p and r, has them; the first
// orders only this: a block overwrites r with values computed from every
// block's word, and those were computed from the rows of r read before).  between()
// runs while the words are under way.  False: a poll gave up.
template <bool MAX, bool DATA, class F>
__device__ __forceinline__ bool coop_exchange(CoopShared& sh, CoopSlot* slots, unsigned number, double s, double m,
                                              bool bad, F between) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const int nw = nt >> 5, nb = gridDim.x;
    double* const wm = sh.fold + kCoopMaxThreads;
    sh.fold[tid] = s;
    if (tid == 0) sh.bad = 0;
    int anybad = 0;
    if (MAX) {
        m = warp_max0(m);
        if (lane == 0) wm[tid >> 5] = m;
        anybad = __syncthreads_or(bad);
    } else {
        __syncthreads();
    }
    slots += (number & 1) * nb;
    if (tid < 32) {
        double a = 0.0;
        for (int k = lane; k < nt; k += 32) a += sh.fold[k];
        a = warp_sum(a);
        const double mm = MAX ? warp_max0(lane < nw ? wm[lane] : 0.0) : 0.0;
        if (lane == 0) {
            const unsigned long long va = (unsigned long long)__double_as_longlong(a);
            const unsigned long long tag = (unsigned long long)number << 32;
            CoopSlot* mine = slots + blockIdx.x;
            if (DATA) __threadfence();  // the block's r and p before its words
            coop_st2(&mine->w[0], tag | (anybad ? 1ull << 63 : 0ull) | (va >> 32), tag | (va & 0xffffffffull));
            if (MAX) {
                const unsigned long long vm = (unsigned long long)__double_as_longlong(mm);
                coop_st2(&mine->w[2], tag | (vm >> 32), tag | (vm & 0xffffffffull));
            }
        }
    }
    between();
    const unsigned limit = c_stage_wait_polls;
    bool ok = limit != 0, seen_bad = false;
    for (int k = tid; k < nb && ok; k += nt) {
        const CoopSlot* s4 = slots + k;
        unsigned long long w[4];
        uint64_t t0 = 0;
        auto is = [&](unsigned long long v) { return ((unsigned)(v >> 32) & 0x7fffffffu) == number; };
        for (unsigned poll = 0;; ++poll) {
            coop_ld2(&s4->w[0], w[0], w[1]);
            if (MAX) coop_ld2(&s4->w[2], w[2], w[3]);
            if (is(w[0]) && is(w[1]) && (!MAX || (is(w[2]) && is(w[3])))) break;
            if (poll == 0) t0 = global_ns();
            if (poll >= limit || ((poll & 255) == 255 && global_ns() - t0 > kMbarWaitNs)) {
                ok = false;
                break;
            }
        }
        seen_bad |= (w[0] >> 63) != 0;
        sh.v[k] = __longlong_as_double((long long)((w[0] << 32) | (w[1] & 0xffffffffull)));
        if (MAX) sh.m[k] = __longlong_as_double((long long)((w[2] << 32) | (w[3] & 0xffffffffull)));
    }
    if (DATA) __threadfence();  // and the others' r and p behind their words
    if (MAX && ok && seen_bad) sh.bad = 1;
    const int failed = __syncthreads_or(!ok);
    if (tid < 32) {
        double a = 0.0, mm = 0.0;
        for (int k = lane; k < nb; k += 32) {
            a += sh.v[k];
            if (MAX) mm = max0(mm, sh.m[k]);
        }
        a = warp_sum(a);
        if (MAX) mm = warp_max0(mm);
        if (lane == 0) {
            sh.sum = a;
            sh.max = mm;
        }
    }
    return !failed;
}

template <int ND, int PM, int K>
__global__ void __launch_bounds__(kCoopMaxThreads) k_cg_coop(CoopArgs a) {
    extern __shared__ double S[];  // p of cells base - H .. base + C + H
    __shared__ CoopShared sh;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int base = blockIdx.x * a.C, cnt = min(a.C, a.n - base);
    CgState* const st = a.st;
    double x[K], r[K], p[K], ap[K];  // of cells base + j nt + tid
    unsigned f[K];
    unsigned number = 0;
    double sig = 0.0, bm = 0.0;
    bool bad = false;
    if (PM == PM_JACOBI) {
        if (tid < 8) sh.inv_diag[tid] = tid ? __drcp_rn((double)tid * a.dt) : 0.0;
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        x[j] = p[j] = ap[j] = r[j] = 0.0;
        f[j] = 0;
        const int l = j * nt + tid;
        if (l >= cnt) continue;
        const double bv = a.b[base + l];
        f[j] = a.flags[base + l];
        r[j] = bv;
        a.r[base + l] = bv;
        bm = fmax(bm, fabs(bv));
        bad |= !isfinite(bv);
        sig += coop_z<PM>(bv, f[j], sh.inv_diag) * bv;
    }
    double sigma = 0.0, thr = 0.0, bmax = 0.0, rmax = 0.0, pap = 0.0, alpha = 0.0, beta = 0.0;  // thread 0
    int status = PG_NOT_CONVERGED;
    bool live = coop_exchange<true, true>(sh, a.slots, ++number, sig, bm, bad, [] {});
    if (tid == 0) {  // as cg_init_finish
        sigma = sh.sum;
        bmax = rmax = sh.max;
        thr = a.rel_tol > 0.0 ? a.rel_tol * bmax : a.thr;
        sh.stop = 1;
        if (sh.bad || !isfinite(sigma))
            status = PG_NAN_DETECTED;
        else if (bmax < thr || bmax == 0.0)
            status = PG_OK;
        else if (a.max_iter > 0)
            sh.stop = 0;
        sh.scale = 0.0;
    }
    __syncthreads();
    i64 it = 0;
    while (live && !sh.stop) {
        const bool first = it == 0;
        const double bt = sh.scale;  // beta
        const double* __restrict__ p_old = (it & 1) ? a.p1 : a.p0;
        double* __restrict__ p_new = (it & 1) ? a.p0 : a.p1;
        // the rows around the block's cells, recomputed from the neighbours'
        // r and p; then the cells
        for (int k = tid; k < 2 * a.H; k += nt) {
            const int c = k < a.H ? base - a.H + k : base + cnt + (k - a.H);
            if (c < 0 || c >= a.n) continue;
            const double z = coop_z<PM>(__ldcg(a.r + c), PM == PM_JACOBI ? a.flags[c] : 0u, sh.inv_diag);
            S[c - base + a.H] = first ? z : z + bt * __ldcg(p_old + c);
        }
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int l = j * nt + tid;
            if (l >= cnt) continue;
            const double z = coop_z<PM>(r[j], f[j], sh.inv_diag);
            p[j] = first ? z : z + bt * p[j];
            S[l + a.H] = p[j];
            p_new[base + l] = p[j];
        }
        __syncthreads();
        double dot = 0.0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int l = j * nt + tid;
            if (l >= cnt) continue;
            const double* q = S + l + a.H;
            const double pc = p[j];
            const double gy_lo = (f[j] & YLO) ? -sub_rn(pc, q[-a.w]) : 0.0;
            const double gy_hi = (f[j] & YHI) ? -sub_rn(q[a.w], pc) : 0.0;
            const double gx_lo = (f[j] & XLO) ? sub_rn(q[-1], pc) : 0.0;
            const double gx_hi = (f[j] & XHI) ? sub_rn(pc, q[1]) : 0.0;
            double v = add_rn(sub_rn(sub_rn(gy_hi, gy_lo), gx_lo), gx_hi);
            if (ND == 3) {
                const double gz_lo = (f[j] & ZLO) ? -sub_rn(pc, q[-a.H]) : 0.0;
                const double gz_hi = (f[j] & ZHI) ? -sub_rn(q[a.H], pc) : 0.0;
                v = add_rn(sub_rn(v, gz_lo), gz_hi);
            }
            ap[j] = mul_rn(v, a.dt);
            dot += pc * ap[j];
        }
        live = coop_exchange<false, false>(sh, a.slots, ++number, dot, 0.0, false, [] {});
        if (tid == 0) {
            pap = sh.sum;
            if (!isfinite(pap)) {
                status = PG_NAN_DETECTED;
                sh.stop = 1;
            } else if (!(pap > 0.0)) {
                status = sigma == 0.0 ? PG_NOT_CONVERGED : PG_BREAKDOWN;
                sh.stop = 1;
            } else {
                alpha = sigma / pap;  // pcg.rs:53
                sh.scale = alpha;
            }
        }
        __syncthreads();
        if (!live || sh.stop) break;
        const double al = sh.scale, nal = -al;
        double rz = 0.0, rm = 0.0;
        bad = false;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int l = j * nt + tid;
            if (l >= cnt) continue;
            const double rv = r[j] + nal * ap[j];  // pcg.rs:56
            r[j] = rv;
            a.r[base + l] = rv;
            rm = fmax(rm, fabs(rv));
            bad |= !isfinite(rv);
            rz += coop_z<PM>(rv, f[j], sh.inv_diag) * rv;
        }
        live = coop_exchange<true, true>(sh, a.slots, ++number, rz, rm, bad, [&] {
#pragma unroll
            for (int j = 0; j < K; ++j) x[j] = x[j] + al * p[j];  // pcg.rs:55
        });
        ++it;
        if (tid == 0) {
            rmax = sh.max;
            if (sh.bad || !isfinite(rmax)) {
                status = PG_NAN_DETECTED;
                sh.stop = 1;
            } else if (rmax < thr) {  // pcg.rs:58-63
                status = PG_OK;
                sh.stop = 1;
            } else if (!isfinite(sh.sum)) {
                status = PG_NAN_DETECTED;
                sh.stop = 1;
            } else {
                beta = sh.sum / sigma;  // pcg.rs:65-68
                sigma = sh.sum;
                sh.scale = beta;
                if (it >= a.max_iter) sh.stop = 1;  // loop bound, pcg.rs:48
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int l = j * nt + tid;
        if (l >= cnt) continue;
        a.x[base + l] = x[j];
        if (number > 1) a.ap[base + l] = ap[j];
    }
    if (tid != 0) return;
    if (!live) {
        st->status = PG_TIMEOUT;
        st->done = 1;
        return;
    }
    if (blockIdx.x != 0) return;
    st->sigma = sigma;
    st->pap = pap;
    st->alpha = alpha;
    st->beta = beta;
    st->rmax = rmax;
    st->bmax = bmax;
    st->threshold = thr;
    st->iter = it;
    st->max_iter = a.max_iter;
    st->first = it <= 1 ? 1 : 0;
    if (st->status != PG_TIMEOUT) st->status = status;
    st->done = 1;
}

template <int ND, int PM, int K>
int coop_launch(cudaStream_t s, int blocks, int threads, size_t smem, CoopArgs& args, bool* fits) {
    int n = 0;
    if (cudaFuncSetAttribute(k_cg_coop<ND, PM, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoopSmemMax) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_cg_coop<ND, PM, K>, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    *fits = n >= 1;
    if (!*fits) return PG_OK;
    void* params[] = {&args};
    cudaError_t e = cudaSuccess;
    PG_LAUNCH(KK_CG_UPDATE, s,
              e = cudaLaunchCooperativeKernel((const void*)k_cg_coop<ND, PM, K>, dim3(blocks), dim3(threads), params,
                                              smem, s));
    return e == cudaSuccess ? PG_OK : cuda_fail(e, "cooperative CG launch");
}

// Whether an iteration with C cells per block and rows (planes) of H cells is
// faster here than in the loop.  A block computes p of its 2 H halo cells from
// global memory, 0.27 us per 512 of them, which the loop does not.  An
// iteration of the loop is at its launch latency on small grids, 14 us in 2D
// (and from 30 K cells on grows, 1 us per 15 K), 20 in 3D up to about 120 K
// cells (C of 800) and 33 beyond, so the halo may be as large as what that
// leaves.  Measured, plain CG per iteration, the loop / this: 10 x 3000 14.3 /
// 13.3, 5 x 5000 14.5 / 15.5, 20 x 6000 20.1 / 19.0, 18 x 9000 23.3 / 24.1, 25 x
// 10000 29.9 / 27.8; 16 x 80 x 80 20.5 / 19.7, 8 x 100 x 100 20.3 / 23.6, 12 x 90
// x 90 20.2 / 21.5, 12 x 100 x 100 33.4 / 24.9.  (Jacobi gains more everywhere.)
bool coop_pays(int nd, i64 C, i64 H) {
    if (nd == 2) return 2 * H <= 6000 + 9 * C;
    return C >= 800 || H <= 6400;
}

bool coop_enabled() {
    const char* env = getenv("PG_CG_COOP");
    return !(env && env[0] == '0');
}

}  // namespace

int set_stage_wait_polls_coop(unsigned polls) {
    PG_CUDA(cudaMemcpyToSymbol(c_stage_wait_polls, &polls, sizeof(polls)));
    return PG_OK;
}

size_t cg_coop_bytes() { return 2 * kCoopMaxBlocks * sizeof(CoopSlot); }

// The whole solve in one cooperative launch where it applies (*done): grids
// whose cells fit the registers of one block per SM, whose rows (planes) around
// a block's cells fit its shared memory and cost less than the loop's launches.  PG_CG_COOP=0 keeps the
// two-kernel loop (a diagnostic switch); so does profiling, which times those
// kernels one by one.
int cg_coop_run(pg_grid* g, const CgConfig& cfg, const CgBuffers<double>& buf, int pm, bool* done) {
    *done = false;
    const Dims& D = g->dims;
    const i64 n = D.nc();
    if (!coop_enabled() || !graphs_enabled() || (pm != PM_NONE && pm != PM_JACOBI) || !cfg.zero_x) return PG_OK;
    const int sms = std::min(g->num_sms, kCoopMaxBlocks);
    // cells per block: a share of the grid, in whole warps; cells per thread:
    // the fewest that kCoopMaxThreads threads can hold
    const i64 C = ((n + sms - 1) / sms + 31) / 32 * 32;
    int K = 1;
    while (K < kCoopMaxCells && C > (i64)K * kCoopMaxThreads) K *= 2;
    if (C > (i64)K * kCoopMaxThreads) return PG_OK;
    const i64 H = D.nd == 3 ? D.h * D.w : D.w;
    if (H > (i64)1 << 24 || (size_t)(C + 2 * H) * sizeof(double) > (size_t)kCoopSmemMax) return PG_OK;
    if (!coop_pays(D.nd, C, H)) return PG_OK;
    // threads: one per polled block, all of the block's cells, an eighth of its
    // halo (4 x 64 x 64, 8192 halo cells: 160 threads 21.5 us, 512 13.1)
    auto warps = [](i64 v) { return (v + 31) / 32 * 32; };
    const int threads =
        (int)std::min<i64>(kCoopMaxThreads, std::max({(i64)160, warps((C + K - 1) / K), warps((2 * H + 7) / 8)}));
    const size_t smem = (size_t)(C + 2 * H) * sizeof(double);
    CoopArgs a;
    a.x = buf.x;
    a.r = buf.r;
    a.p0 = buf.p[0];
    a.p1 = buf.p[1];
    a.ap = buf.ap;
    a.b = buf.b;
    a.flags = g->flags;
    a.n = (int)n;
    a.w = (int)D.w;
    a.H = (int)H;
    a.C = (int)C;
    a.dt = cfg.dt;
    a.thr = cfg.threshold;
    a.rel_tol = cfg.rel_tol;
    a.max_iter = cfg.max_iter;
    a.st = g->ws.state;
    a.slots = (CoopSlot*)g->ws.coop;
    cudaStream_t s = g->stream;
    const int blocks = (int)((n + C - 1) / C);
    PG_CUDA(cudaMemsetAsync(g->ws.coop, 0, 2 * (size_t)blocks * sizeof(CoopSlot), s));  // no exchange has happened
    bool fits = false;
    int rc = PG_OK;
#define PG_COOP(ND, PM)                                                                  \
    rc = K == 1   ? coop_launch<ND, PM, 1>(s, blocks, threads, smem, a, &fits)           \
         : K == 2 ? coop_launch<ND, PM, 2>(s, blocks, threads, smem, a, &fits)           \
         : K == 4 ? coop_launch<ND, PM, 4>(s, blocks, threads, smem, a, &fits)           \
                  : coop_launch<ND, PM, 8>(s, blocks, threads, smem, a, &fits)
    if (D.nd == 2) {
        if (pm == PM_JACOBI)
            PG_COOP(2, PM_JACOBI);
        else
            PG_COOP(2, PM_NONE);
    } else {
        if (pm == PM_JACOBI)
            PG_COOP(3, PM_JACOBI);
        else
            PG_COOP(3, PM_NONE);
    }
#undef PG_COOP
    *done = fits && rc == PG_OK;
    return rc;
}

}  // namespace pg
