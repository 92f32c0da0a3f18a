// lsdev.cu -- the line search of maxdLqdt on the device: the controller and
// the bookkeeping kernels of the conditional graph that runs mnbrak and Brent
// (optimization.f90:613-951) without a host round trip per trial.
//
// Compiled without multiply-add contraction (-fmad=false) so that every
// trial value and every step of the search rounds as on the host.
#include "linesearch.cuh"

namespace mlq {

namespace {

__device__ bool ls_memo_add(LsDevState* s, double tau, const double R[3], double lqq, int fft) {
    const int k = s->ntr;
    if (k >= LS_MEMO) return false;
    s->mtau[k] = tau;
    for (int i = 0; i < 3; ++i) s->mR[k][i] = R[i];
    s->mlqq[k] = lqq;
    s->mJ[k] = ls_J(R[1], R[2], lqq, s->par.q, s->par.B);
    s->mfft[k] = fft;
    s->ntr = k + 1;
    return true;
}

// What the controller reads, in shared memory: it is one thread, and a trial
// is a chain of dependent reads of these.
struct LsShared {
    LsPoly poly;
    LsParams par;
    double tau[LS_MEMO], J[LS_MEMO];
};

// J(tau) from the table, or from the polynomials inside [tlo, thi];
// anything else suspends the search at tau.
struct DevEval {
    LsDevState* s;
    LsShared* sh;
    int n;  // entries of the table
    int count = 0;
    int err = 0;
    double ptau = 0.0;
    __device__ bool operator()(double tau, double* J) {
        ++count;
        const LsParams& p = sh->par;
        int k = -1;
        for (int i = 0; i < n; ++i)
            if (sh->tau[i] == tau) {
                k = i;
                break;
            }
        if (k < 0) {
            if (p.transform_trials || !ls_free(sh->poly, tau)) {
                ptau = tau;
                return false;
            }
            double R[3], lqq;
            ls_poly_R(sh->poly, p.q, p.cv, p.cp, tau, R, &lqq);
            if (!ls_memo_add(s, tau, R, lqq, 0)) {
                err = LS_ERR_CAP;
                return false;
            }
            k = n++;
            sh->tau[k] = tau;
            sh->J[k] = s->mJ[k];
        }
        *J = sh->J[k];
        if (isnan(*J)) {
            err = MLQ_ERR_NAN;
            return false;
        }
        return true;
    }
};

__device__ void ls_stop(LsDevState* s, int status, cudaGraphConditionalHandle h_loop,
                        cudaGraphConditionalHandle h_chk) {
    s->out.status = status;
    cudaGraphSetConditional(h_loop, 0);
    cudaGraphSetConditional(h_chk, 0);
}

}  // namespace

constexpr int LS_COEF_THREADS = 512;

// The coefficients of this line search from the setup's sums (results[100..],
// [140..], [149..]) and the per-block interval ends (partials, 2 per block);
// clears the table for a new search.
__global__ void __launch_bounds__(LS_COEF_THREADS)
    ls_coef_kernel(LsDevState* s, const double* __restrict__ results, const double* __restrict__ partials, int nblocks,
                   LsAnchorSet an) {
    pdl_begin();
    // max and min are exact, so any order gives the same ends; one warp alone
    // took 20 us over the 592 blocks of 64^3
    constexpr int K = LS_ANCHORS + 1, W = 2 * K, NW = LS_COEF_THREADS / 32;
    __shared__ double slo[NW][K], shi[NW][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double lo[K], hi[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        lo[k] = -1e300;
        hi[k] = 1e300;
    }
    for (int g = threadIdx.x; g < nblocks; g += LS_COEF_THREADS)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            lo[k] = fmax(lo[k], partials[W * g + 2 * k]);
            hi[k] = fmin(hi[k], partials[W * g + 2 * k + 1]);
        }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fmax(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmin(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        if (lane == 0) {
            slo[warp][k] = lo[k];
            shi[warp][k] = hi[k];
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int k = 0; k < K; ++k)
        for (int w = 1; w < NW; ++w) {
            lo[k] = fmax(lo[k], slo[w][k]);
            hi[k] = fmin(hi[k], shi[w][k]);
        }
    ls_assemble(results + 100, results + 140, results + 149, lo[0], hi[0], lo + 1, hi + 1, an.a, s->poly);
    s->ntr = 0;
    s->need = 0;
    s->checked = 0;
    s->ptau = 0.0;
    s->out = LsOut{};
    s->out.status = LS_RUNNING;
}

// One pass of the controller: the value of the last tau, then mnbrak and Brent
// from the start over the table; ends the loop when the search completes (or
// fails), else leaves the first tau without a value in ptau and opens the
// branch h_next (the check, or with `direct` the transform).  sums: those of a
// transform trial.
__global__ void ls_ctrl_kernel(LsDevState* s, const double* __restrict__ sums, int direct,
                               cudaGraphConditionalHandle h_loop, cudaGraphConditionalHandle h_next) {
    __shared__ LsShared sh;
    for (int i = threadIdx.x; i < (int)(sizeof(LsPoly) / sizeof(double)); i += blockDim.x)
        reinterpret_cast<double*>(&sh.poly)[i] = reinterpret_cast<const double*>(&s->poly)[i];
    if (threadIdx.x == 0) {
        sh.par = s->par;
        if (s->need >= 2) {
            const LsParams& p = s->par;
            double R[3], lqq;
            if (s->need == 2)
                ls_fft_R(s->poly, p.q, p.cv, p.cp, sums, s->ptau, R, &lqq);
            else
                ls_poly_R(s->poly, p.q, p.cv, p.cp, s->ptau, R, &lqq);
            if (!ls_memo_add(s, s->ptau, R, lqq, s->need == 2)) s->out.status = LS_ERR_CAP;
            s->need = 0;
        }
    }
    __syncwarp();
    const int n = s->ntr;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        sh.tau[i] = s->mtau[i];
        sh.J[i] = s->mJ[i];
    }
    __syncwarp();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    LsOut& o = s->out;
    if (o.status != LS_RUNNING) {
        ls_stop(s, o.status, h_loop, h_next);
        return;
    }
    if (o.loops >= LS_MAX_LOOPS) {
        ls_stop(s, LS_ERR_CAP, h_loop, h_next);
        return;
    }
    ++o.loops;
    DevEval ev{s, &sh, n};
    double tb[2] = {0.0, 0.0}, x = 0.0, fx = 0.0;
    int mflag = 0;
    int r = ls_mnbrak(ev, s->par.tA0, s->par.tB0, tb, &mflag);
    if (r == 0) r = ls_brent(ev, tb, &x, &fx);
    if (ev.err) {
        ls_stop(s, ev.err, h_loop, h_next);
        return;
    }
    if (r == LS_SUSPEND) {
        s->need = direct ? 2 : 1;
        s->ptau = ev.ptau;
        if (!direct) ++o.checks;
        cudaGraphSetConditional(h_loop, 1);
        cudaGraphSetConditional(h_next, 1);
        return;
    }
    o.mflag = mflag;
    o.tb[0] = tb[0];
    o.tb[1] = tb[1];
    o.evals = ev.count;
    for (int i = 0; i < s->ntr; ++i) {
        if (s->mfft[i])
            ++o.nfft;
        else
            ++o.npoly;
    }
    if (mflag == 0) {
        o.tau1 = x;
        o.fx = fx;
        for (int i = 0; i < s->ntr; ++i)
            if (s->mtau[i] == x) {
                for (int c = 0; c < 3; ++c) o.R1[c] = s->mR[i][c];
                o.lqq1 = s->mlqq[i];
                o.fft1 = s->mfft[i];
                break;
            }
    }
    ls_stop(s, 0, h_loop, h_next);
}

void ls_launch_coef(LsDevState* s, const double* results, const double* partials, int nblocks, const LsAnchorSet& an,
                    bool pdl, cudaStream_t st) {
    MLQ_CUDA(launch_pdl(pdl, ls_coef_kernel, 1, LS_COEF_THREADS, 0, st, s, results, partials, nblocks, an));
}
void ls_launch_ctrl(LsDevState* s, const double* r, int direct, cudaGraphConditionalHandle h_loop,
                    cudaGraphConditionalHandle h_next, cudaStream_t st) {
    ls_ctrl_kernel<<<1, 32, 0, st>>>(s, r, direct, h_loop, h_next);
}

}  // namespace mlq
