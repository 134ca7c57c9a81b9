// mcmc_kernels.cu -- Metropolis-Hastings and Goodman-Weare ensemble MCMC.
//
// Goodman-Weare: a block holds VPB voxels; each voxel's ensemble lives in
// shared memory and one thread advances one walker (simultaneous update) or
// one walker of each half (red-black).  Proposals use counter-based Philox
// keyed by (voxel, walker, step, repetition), the partner draws are shared by
// all voxels as in the reference, the likelihood is accumulated in FP64 and
// kept samples are folded into FP64 running sums on the fly (optionally
// written out as the full posterior).  Reference: utils/mcmc.m
// (metropolis_hastings :82-190, goodman_weare :192-383, find_partner
// :797-803, res2out :806-862), utils/logP_Gaussian.m.
#include <algorithm>

#include "gx_internal.h"

namespace gx {

constexpr int kMaxWalker = 256;

// find_partner (mcmc.m:797-803): a uniform random derangement of the W
// walkers (Fisher-Yates, fixed points rejected), from the Philox stream
// (step, attempt, draw/4, tag).
__device__ void derangement_dev(uint64_t seed, int k, uint32_t tag, int W, int* out) {
    int perm[kMaxWalker];
    bool ok = false;
    for (uint32_t attempt = 0; attempt < 4096 && !ok; ++attempt) {
        for (int i = 0; i < W; ++i) perm[i] = i;
        U4 u{0, 0, 0, 0};
        for (int i = W - 1, d = 0; i >= 1; --i, ++d) {
            if ((d & 3) == 0) u = philox((uint32_t)k, attempt, (uint32_t)(d >> 2), tag, seed);
            uint32_t r = (d & 3) == 0 ? u.x : (d & 3) == 1 ? u.y : (d & 3) == 2 ? u.z : u.w;
            int j = (int)rand_below(r, (uint32_t)(i + 1));
            int t = perm[i]; perm[i] = perm[j]; perm[j] = t;
        }
        ok = true;
        for (int i = 0; i < W; ++i) ok = ok && perm[i] != i;
    }
    for (int i = 0; i < W; ++i) out[i] = ok ? perm[i] : (i + 1) % W;
}

// Red-black anchors (mcmc.m:328-329): the a-th active walker of half `half`
// anchors on frozen(randi(numel(frozen))); written as absolute walker indices.
__device__ void rb_anchors_dev(uint64_t seed, int k, uint32_t tag, int W, int* out) {
    int h = W / 2;
    for (int half = 0; half < 2; ++half) {
        int na = half == 0 ? h : W - h, nf = half == 0 ? W - h : h, f0 = half == 0 ? h : 0;
        int a0 = half == 0 ? 0 : h;
        U4 u{0, 0, 0, 0};
        for (int a = 0; a < na; ++a) {
            if ((a & 3) == 0) u = philox((uint32_t)k, (uint32_t)half, (uint32_t)(a >> 2), tag, seed);
            uint32_t r = (a & 3) == 0 ? u.x : (a & 3) == 1 ? u.y : (a & 3) == 2 ? u.z : u.w;
            out[a0 + a] = f0 + (int)rand_below(r, (uint32_t)nf);
        }
    }
}

// Partner tables [rep][nsteps][W]: simultaneous -> one derangement per step,
// red-black -> the anchors of both halves.  Rows past `iteration` are the
// global warm-up steps 1..(nsteps - iteration).  global_block selects the
// global block's streams (goodman_weare_wglobal_constant).
__global__ void gw_partner_kernel(McmcParams p, int* partner, int nsteps, int global_block) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= p.repetition * nsteps) return;
    int rr = idx / nsteps, kk = idx % nsteps + 1;
    int k = kk <= p.iteration ? kk : kk - p.iteration;
    uint32_t bits = ((uint32_t)rr << 16) | (kk > p.iteration ? kTagWarmup : 0u);
    int* out = partner + (size_t)idx * p.nwalker;
    if (p.update == 0) derangement_dev(p.seed, k, (global_block ? kTagGwGPerm : kTagGwPerm) | bits, p.nwalker, out);
    else rb_anchors_dev(p.seed, k, (global_block ? kTagGwGRbPart : kTagGwRbPart) | bits, p.nwalker, out);
}

// Residual of one R2* echo, M0 exp(-te R2*) - y, with its roundings stated: the
// log-likelihood and the screen below form it alike, whatever the compiler fuses.
__device__ __forceinline__ float r2s_residual(float te_l2e, float M0, float R2, float y) {
    return fma1(M0, ex2_ftz(mul1(-te_l2e, R2)), -y);
}

// logP_Gaussian (utils/logP_Gaussian.m:18-20) of the model's parameters and
// the noise sigma (the last of the NV variables, a compile-time index so that
// the caller's parameter vector stays in registers); y / w with strides.
template <int MODEL, int NV>
__device__ __forceinline__ double log_prob_t(int nm, const DevProtocol& P, const float (&x)[NV], const float* y,
                                             int ys, const float* w, int ws, const VoxAux& va) {
    constexpr int NP = ModelNP<MODEL>::value;
    static_assert(NV == NP + 1, "the variables are the model's parameters and the noise sigma");
    double sos = 0.0;
    if constexpr (MODEL == kR2S) {
        for (int m = 0; m < P.nm; ++m) {
            const float r = r2s_residual(P.te_l2e[m], x[0], x[1], y[m * ys]);
            const float ww = w ? w[m * ws] : 1.0f;
            sos += (double)(ww * r * r);
        }
    } else {
        SosSink<NP> sink{y, ys, w, ws, 0.0};
        model_eval<MODEL>(P, x, va, sink);
        sos = sink.sos;
    }
    const double noise = (double)x[NV - 1];
    const double n2 = noise * noise;
    return -sos / (2.0 * n2) - 0.5 * nm * log(6.283185307179586 * n2);
}

// Screened acceptance (R2*, unit weights, up to kScreenM measurements).
//
// The decision lr > log u needs the FP64 log-likelihoods (division, logarithm
// and an FP64 sum: a third of a step's instructions, and its longest
// dependent chain) only when the two sides are close.  The screen evaluates
// both in FP32 with a bound on its error, and the FP64 form (log_prob_t, the
// same values whenever it is evaluated) decides inside the bound, about one
// proposal in 10^4; so every decision is the FP64 one.  With n the noise,
// a = sos / (2 n^2) and the constant nm log(2 pi) / 2 cancelling,
//   log p' - log p = (a - a') + nm (log n - log n').
// Error, with e = 2^-24: the residuals are the FP64 form's (r2s_residual);
// the FP32 sum of their nm squares and the FP64 sum of the rounded squares
// differ by at most (nm + 1) e relative, a by at most another 6 e (n^2,
// reciprocal of 1 ulp, two products): (nm + 20) e.  __logf is within
// 2^-21.4 absolute or 3 ulp relative of the logarithm, and the roundings of
// the sums are below 2^-21 of their terms: 2^-20 of every term's magnitude
// plus 2^-20 for every logarithm.  NaN and infinities fail both tests and go
// to the FP64 form.  The noise's bounds have to keep 2 n^2 and its reciprocal
// in FP32's normal range (kScreenMaxNoise), and n large enough that the squares
// below 2^-126, which FP32 flushes, do not count: nm 2^-126 / (2 n^2) is at most
// nm 2^-20 from 1e-16 on (kScreenMinNoise).
// Measurements in registers, echo constants in the constant bank; kernels for
// up to 8, 12 and 16 echoes, since a test per echo and one chain of sums cost a
// tenth of the kernel.  12,013 voxels x 50 walkers x 500
// steps, 12 echoes: 6.93 (all FP64) -> 3.65 ms; red-black, 12,000 x 50 x 300,
// whole call: 6.50 -> 3.72 ms (124-152 bytes spilled); Metropolis-Hastings, 4096
// voxels x 10,000 steps: 15.4 -> 6.1 ms (one dependent chain a voxel, 1.4-2.1
// -> 0.6 us a step).
constexpr int kScreenM = 16;
constexpr float kScreenMinNoise = 1e-16f, kScreenMaxNoise = 1e18f;

struct Screen {
    float a, ln;  // sos / (2 n^2), log n
};

// P: the protocol in the constant bank (compile-time indices); up to MAXM
// echoes, without a test when the protocol fills the bound.
template <int MAXM>
__device__ __forceinline__ Screen screen_eval(const DevProtocol& P, int nm, const float (&x)[3],
                                              const float (&y)[MAXM]) {
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // short chains
    auto echo = [&](int m) {
        const float r = r2s_residual(P.te_l2e[m], x[0], x[1], y[m]);
        s[m & 3] = fma1(r, r, s[m & 3]);
    };
    if (nm == MAXM) {
#pragma unroll
        for (int m = 0; m < MAXM; ++m) echo(m);
    } else {
#pragma unroll
        for (int m = 0; m < MAXM; ++m)
            if (m < nm) echo(m);
    }
    return Screen{((s[0] + s[1]) + (s[2] + s[3])) * rcp_ftz(2.0f * x[2] * x[2]), __logf(x[2])};
}

// 1 accept, 0 reject, -1 undecided: cz log(zz) + (log p(n) - log p(c)) > log(u)
__device__ __forceinline__ int screen_decide(int nm, const Screen& c, const Screen& n, float cz, float zz, float u) {
    const float fm = (float)nm;
    const float lz = cz * __logf(zz), lu = __logf(u);
    const float d = ((c.a - n.a) + fm * (c.ln - n.ln)) + (lz - lu);
    const float tol = (fm + 20.0f) * 5.9604645e-8f * (c.a + n.a) +
                      9.536743e-7f * (fm * (2.0f + fabsf(c.ln) + fabsf(n.ln)) + fabsf(lz) + fabsf(lu) + cz + 2.0f);
    return d > tol ? 1 : (d < -tol ? 0 : -1);
}

// The FP64 decision, kept out of line: cz log(zz) + (log p(n) - log p(c)) > log(u).
__device__ __noinline__ bool exact_accept(const DevProtocol& P, int nm, float c0, float c1, float c2, float n0, float n1,
                                          float n2, const float* y, int ys, float cz, float zz, float u) {
    const float xc[3] = {c0, c1, c2}, xn[3] = {n0, n1, n2};
    VoxAux va{1.0f, nullptr, nullptr, 1};
    const double lr = (double)cz * (double)logf(zz) +
                      (log_prob_t<kR2S, 3>(nm, P, xn, y, ys, nullptr, 1, va) - log_prob_t<kR2S, 3>(nm, P, xc, y, ys, nullptr, 1, va));
    return lr > (double)logf(u);
}

// Steps k with a kept sample, k > nburnin and (k - nburnin + 1) % thinning
// == 0: the first one at or after k0 (a launch steps from it by thinning).
__device__ __forceinline__ int first_kept(const McmcParams& p, int k0) {
    const int k = max(k0, p.nburnin + 1);
    const int r = (k - p.nburnin + 1) % p.thinning;
    return r ? k + p.thinning - r : k;
}

__device__ __forceinline__ int kept_index(const McmcParams& p, int k) {
    if (k <= p.nburnin) return -1;
    int j = k - p.nburnin + 1;
    if (j % p.thinning) return -1;
    int c = j / p.thinning - (p.thinning == 1 ? 1 : 0) - 1;
    return c < p.ns ? c : -1;
}

// Walker start (mcmc.m:267-275): x0 + (ub-lb)*startRange*randn, clamped; the
// normal draws of walker w of voxel v come four at a time from the Philox
// stream (v, w, j, kTagGwInit).
template <int NV>
__device__ __forceinline__ void gw_walker_start(const McmcParams& p, int v, int w, float (&x)[NV]) {
    float nrm[(NV + 3) / 4 * 4];
#pragma unroll
    for (int j = 0; j * 4 < NV; ++j) {
        U4 u = philox((uint32_t)v, (uint32_t)w, (uint32_t)j, kTagGwInit, p.seed);
        box_muller(u.x, u.y, nrm[4 * j], nrm[4 * j + 1]);
        box_muller(u.z, u.w, nrm[4 * j + 2], nrm[4 * j + 3]);
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        float val = p.x0[(size_t)q * p.nvox + v] + (p.ub[q] - p.lb[q]) * p.start_range * nrm[q];
        x[q] = fminf(fmaxf(val, p.lb[q]), p.ub[q]);
    }
}

// Goodman-Weare, steps [k0, k1] of repetition rr.  State between launches:
// xstate [nvar][nvox][W], lpstate [nvox][W].  NV = parameters + noise, fixed
// at compile time, and RB (red-black: a thread owns a walker of each half)
// keep every per-walker vector in registers; the running sums of the kept
// samples live in shared memory (each thread its own walkers' slots) and are
// folded into the per-voxel sums at the end of the launch.
// SCREEN > 0: acceptance decided by the FP32 screen where it can (up to SCREEN
// measurements); the walkers' log-likelihoods are then not kept (xstate
// determines them).
template <int MODEL, int NV, bool RB, int SCREEN>
__global__ void __launch_bounds__(1024, 1)
gw_kernel(McmcParams p, int rr, int k0, int k1, int init, float* xstate, double* lpstate, double* sum,
          double* sumsq) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ DevProtocol s_P;
    stage_protocol(p.P, &s_P);
    const int W = p.nwalker, nm = p.nm;
    const int h = W / 2;
    const int tpv = RB ? (W - h) : W;
    const int vpb = blockDim.x / tpv;
    const int vl = threadIdx.x / tpv, a = threadIdx.x % tpv;
    const int v = blockIdx.x * vpb + vl;
    const bool in_block = vl < vpb;
    const bool live = in_block && v < p.nvox;
    double* ssum = reinterpret_cast<double*>(smem_raw);           // [2][vpb][W][NV] kept-sample sums
    float* xs = reinterpret_cast<float*>(ssum + 2 * vpb * W * NV); // [vpb][W][NV]
    float* ys = xs + vpb * W * NV;                                // [vpb][nm]
    float* ws = ys + vpb * nm;                                    // [vpb][nm]
    float* xv = xs + (in_block ? vl : 0) * W * NV;
    double* sv1 = ssum + (in_block ? vl : 0) * W * NV;
    double* sv2 = sv1 + vpb * W * NV;
    const float* yv = ys + (in_block ? vl : 0) * nm;
    const float* wv = p.weights ? ws + (in_block ? vl : 0) * nm : nullptr;
    if (live)
        for (int m = a; m < nm; m += tpv) {
            ys[vl * nm + m] = p.data[(size_t)m * p.nvox + v];
            if (p.weights) ws[vl * nm + m] = p.weights[(size_t)m * p.nvox + v];
        }
    float b1 = (live && p.b1) ? p.b1[v] : 1.0f;
    float sa[MODEL == kR1R2S ? kMaxFA : 1], ca[MODEL == kR1R2S ? kMaxFA : 1];
    if (MODEL == kR1R2S)
        for (int f = 0; f < p.P.n_fa; ++f) sincosf(b1 * p.P.fa_rad[f], &sa[f], &ca[f]);
    VoxAux va{b1, sa, ca, 1};
    if constexpr (kIsNexi<MODEL>)
        if (p.node_smem) {  // behind the rest, at a 16-byte boundary
            NexiNodes* s_nodes = reinterpret_cast<NexiNodes*>(
                smem_raw + ((sizeof(double) * 2 * vpb * W * NV + sizeof(float) * (vpb * W * NV + 2 * vpb * nm) + 15) & ~(size_t)15));
            stage_nodes(p.nodes, s_nodes);
            va.nodes = s_nodes;
        }

    // walkers owned by this thread: slot 0 (simultaneous: walker a; red-black:
    // walker a of the first half, if any) and, red-black, slot 1 (walker h + a)
    const int wown0 = RB ? (a < h ? a : -1) : a, wown1 = RB ? h + a : -1;
    const bool own0 = live && wown0 >= 0 && wown0 < W, own1 = RB && live && wown1 >= 0 && wown1 < W;
    float x0s[NV], x1s[RB ? NV : 1];
    double lp0 = 0.0, lp1 = 0.0;
    Screen c0{0.0f, 0.0f}, c1{0.0f, 0.0f};
    float yr[SCREEN > 0 ? SCREEN : 1];
#pragma unroll
    for (int q = 0; q < NV; ++q) x0s[q] = 0.0f;
#pragma unroll
    for (int q = 0; q < (RB ? NV : 1); ++q) x1s[q] = 0.0f;
    if (own0)
#pragma unroll
        for (int q = 0; q < NV; ++q) { sv1[wown0 * NV + q] = 0.0; sv2[wown0 * NV + q] = 0.0; }
    if (own1)
#pragma unroll
        for (int q = 0; q < NV; ++q) { sv1[wown1 * NV + q] = 0.0; sv2[wown1 * NV + q] = 0.0; }
    __syncthreads();
    if (own0) {
        if (init) gw_walker_start<NV>(p, v, wown0, x0s);
        else
#pragma unroll
            for (int q = 0; q < NV; ++q) x0s[q] = xstate[((size_t)q * p.nvox + v) * W + wown0];
#pragma unroll
        for (int q = 0; q < NV; ++q) xv[wown0 * NV + q] = x0s[q];
    }
    if constexpr (RB) {
        if (own1) {
            if (init) gw_walker_start<NV>(p, v, wown1, x1s);
            else
#pragma unroll
                for (int q = 0; q < NV; ++q) x1s[q] = xstate[((size_t)q * p.nvox + v) * W + wown1];
#pragma unroll
            for (int q = 0; q < NV; ++q) xv[wown1 * NV + q] = x1s[q];
        }
    }
    __syncthreads();
    if constexpr (SCREEN > 0) {
#pragma unroll
        for (int m = 0; m < SCREEN; ++m) yr[m] = live && m < nm ? yv[m] : 0.0f;
        if (own0) c0 = screen_eval(p.P, nm, x0s, yr);
        if constexpr (RB)
            if (own1) c1 = screen_eval(p.P, nm, x1s, yr);
    } else {
        if (own0) lp0 = init ? log_prob_t<MODEL, NV>(nm, s_P, x0s, yv, 1, wv, 1, va) : lpstate[(size_t)v * W + wown0];
        if constexpr (RB)
            if (own1) lp1 = init ? log_prob_t<MODEL, NV>(nm, s_P, x1s, yv, 1, wv, 1, va) : lpstate[(size_t)v * W + wown1];
    }
    unsigned int nacc = 0;
    const float amin1 = p.a - 1.0f;
    int kept_k = first_kept(p, k0);

    // stretch proposal of walker w (state xw, log-likelihood lpw) about its
    // partner: xn and its log-likelihood lpp, and whether it is accepted
    auto propose = [&](int w, int k, uint32_t flags, const float (&xw)[NV], double lpw, const Screen& cw,
                       float (&xn)[NV], double& lpp, Screen& cn) -> bool {
        const int* pt = p.partner + ((size_t)rr * p.iteration + (k - 1)) * W;
        const int q = pt[w];
        U4 u = philox((uint32_t)v, (uint32_t)w, (uint32_t)k, kTagGwMove | ((uint32_t)rr << 16) | flags, p.seed);
        float t = amin1 * u01(u.x) + 1.0f;
        float zz = t * t / p.a;
        bool oob = false;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            float xq = xv[q * NV + j];
            float xp = xq + (xw[j] - xq) * zz;
            oob |= (xp < p.lb[j]) || (xp > p.ub[j]);
            xn[j] = fminf(fmaxf(xp, p.lb[j]), p.ub[j]);
        }
        if constexpr (SCREEN > 0) {
            cn = screen_eval(p.P, nm, xn, yr);
            int d = screen_decide(nm, cw, cn, (float)(NV - 1), zz, u01(u.y));
            if (d < 0 && !oob)
                d = exact_accept(s_P, nm, xw[0], xw[1], xw[2], xn[0], xn[1], xn[2], yv, 1, (float)(NV - 1), zz, u01(u.y));
            return !oob && d > 0;
        }
        lpp = log_prob_t<MODEL, NV>(nm, s_P, xn, yv, 1, wv, 1, va);
        double lr = (double)(NV - 1) * (double)logf(zz) + (lpp - lpw);
        return !oob && lr > (double)logf(u01(u.y));
    };
    auto commit = [&](int w, const float (&xn)[NV], double lpp, const Screen& cn, float (&xw)[NV], double& lpw,
                      Screen& cw) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            xw[j] = xn[j];
            xv[w * NV + j] = xn[j];
        }
        if constexpr (SCREEN > 0) cw = cn;
        else lpw = lpp;
        ++nacc;
    };
    auto keep = [&](int w, int c, const float (&xw)[NV]) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double d = (double)xw[j] - (double)p.shift[(size_t)j * p.nvox + v];
            sv1[w * NV + j] += d;
            sv2[w * NV + j] += d * d;
            if (p.posterior)
                p.posterior[((((size_t)j * p.repetition + rr) * p.ns + c) * W + w) * p.nvox + v] = xw[j];
        }
    };

    for (int k = k0; k <= k1; ++k) {
        if constexpr (!RB) {
            float xn[NV];
            double lpp = 0.0;
            Screen cn{0.0f, 0.0f};
            const bool acc = own0 && propose(wown0, k, 0u, x0s, lp0, c0, xn, lpp, cn);
            __syncthreads();  // every walker has read the old ensemble
            if (acc) commit(wown0, xn, lpp, cn, x0s, lp0, c0);
            __syncthreads();
        } else {
            // the active half moves about anchors in the frozen half
            if (own0) {
                float xn[NV];
                double lpp = 0.0;
                Screen cn{0.0f, 0.0f};
                if (propose(wown0, k, 1u << 8, x0s, lp0, c0, xn, lpp, cn)) commit(wown0, xn, lpp, cn, x0s, lp0, c0);
            }
            __syncthreads();  // the moved half is visible before the other half anchors on it
            if (own1) {
                float xn[NV];
                double lpp = 0.0;
                Screen cn{0.0f, 0.0f};
                if (propose(wown1, k, 1u << 8, x1s, lp1, c1, xn, lpp, cn)) commit(wown1, xn, lpp, cn, x1s, lp1, c1);
            }
            __syncthreads();
        }
        if (k == kept_k) {
            kept_k += p.thinning;
            const int c = kept_index(p, k);
            if (c >= 0) {
                if (own0) keep(wown0, c, x0s);
                if constexpr (RB)
                    if (own1) keep(wown1, c, x1s);
            }
        }
    }
    // persist walker state, fold the kept-sample sums of this launch
    if (own0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) xstate[((size_t)q * p.nvox + v) * W + wown0] = x0s[q];
        if constexpr (SCREEN == 0) lpstate[(size_t)v * W + wown0] = lp0;
    }
    if constexpr (RB) {
        if (own1) {
#pragma unroll
            for (int q = 0; q < NV; ++q) xstate[((size_t)q * p.nvox + v) * W + wown1] = x1s[q];
            if constexpr (SCREEN == 0) lpstate[(size_t)v * W + wown1] = lp1;
        }
    }
    if (live) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double t1 = own0 ? sv1[wown0 * NV + j] : 0.0, t2 = own0 ? sv2[wown0 * NV + j] : 0.0;
            if (own1) { t1 += sv1[wown1 * NV + j]; t2 += sv2[wown1 * NV + j]; }
            if (t1 != 0.0) atomicAdd(&sum[(size_t)j * p.nvox + v], t1);
            if (t2 != 0.0) atomicAdd(&sumsq[(size_t)j * p.nvox + v], t2);
        }
    }
    unsigned int wsum = nacc;
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if ((threadIdx.x & 31) == 0 && wsum) atomicAdd(p.n_acc, (unsigned long long)wsum);
}

// Metropolis-Hastings, one thread per voxel (mcmc.m:144-167).  NV =
// parameters + noise at compile time (the state in registers); the voxel's
// measurements are read from [nm][nvox] with coalesced loads, once into
// registers when the acceptance is screened (SCREEN).  A step's draws do not
// depend on the state, so those of step k + 1 are made while step k's
// proposal is evaluated: with few voxels a step is one dependent chain, and
// the draws fill its latencies.
template <int MODEL, int NV, int SCREEN>
__global__ void mh_kernel(McmcParams p, int rr, int k0, int k1, int init, float* xstate,
                          double* lpstate, double* sum, double* sumsq) {
    __shared__ DevProtocol s_P;
    stage_protocol(p.P, &s_P);
    __shared__ __align__(16) unsigned char s_nodes[kIsNexi<MODEL> ? sizeof(NexiNodes) : 16];
    if constexpr (kIsNexi<MODEL>) stage_nodes(p.nodes, reinterpret_cast<NexiNodes*>(s_nodes));
    __syncthreads();
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    bool live = v < p.nvox;
    const int nm = p.nm;
    const float* yv = p.data + (live ? v : 0);
    const float* wv = p.weights ? p.weights + (live ? v : 0) : nullptr;
    float b1 = (live && p.b1) ? p.b1[v] : 1.0f;
    float sa[MODEL == kR1R2S ? kMaxFA : 1], ca[MODEL == kR1R2S ? kMaxFA : 1];
    if (MODEL == kR1R2S)
        for (int f = 0; f < p.P.n_fa; ++f) sincosf(b1 * p.P.fa_rad[f], &sa[f], &ca[f]);
    VoxAux va{b1, sa, ca, 1};
    if constexpr (kIsNexi<MODEL>) va.nodes = reinterpret_cast<const NexiNodes*>(s_nodes);
    float x[NV];
    double lp = 0.0;
    Screen cs{0.0f, 0.0f};
    float yr[SCREEN > 0 ? SCREEN : 1];
    double s1[NV], s2[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) { s1[q] = 0.0; s2[q] = 0.0; x[q] = 0.0f; }
    unsigned int nacc = 0;
    // the draws of step k: normals for the proposal and the acceptance uniform
    constexpr int ND = (NV + 3) / 4 * 4;
    auto draws = [&](int k, float (&nrm)[ND], float& u) {
        const uint32_t tag = kTagMhMove | ((uint32_t)rr << 16);
#pragma unroll
        for (int j = 0; j * 4 < NV; ++j) {
            U4 r = philox((uint32_t)v, (uint32_t)k, (uint32_t)j, tag, p.seed);
            box_muller(r.x, r.y, nrm[4 * j], nrm[4 * j + 1]);
            box_muller(r.z, r.w, nrm[4 * j + 2], nrm[4 * j + 3]);
        }
        u = u01(philox((uint32_t)v, (uint32_t)k, 8u, tag, p.seed).x);
    };
    if (live) {
        if (init) {
#pragma unroll
            for (int q = 0; q < NV; ++q)
                x[q] = fminf(fmaxf(p.x0[(size_t)q * p.nvox + v], p.lb[q]), p.ub[q]);
            if constexpr (SCREEN == 0) lp = log_prob_t<MODEL, NV>(nm, s_P, x, yv, p.nvox, wv, p.nvox, va);
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q) x[q] = xstate[(size_t)q * p.nvox + v];
            if constexpr (SCREEN == 0) lp = lpstate[v];
        }
        if constexpr (SCREEN > 0) {
#pragma unroll
            for (int m = 0; m < SCREEN; ++m) yr[m] = m < nm ? yv[(size_t)m * p.nvox] : 0.0f;
            cs = screen_eval(p.P, nm, x, yr);
        }
        int kept_k = first_kept(p, k0);
        float nrm[ND], u;
        draws(k0, nrm, u);
        for (int k = k0; k <= k1; ++k) {
            float xp[NV];
            bool oob = false;
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                float t = x[q] + p.xstep[q] * nrm[q];
                oob |= (t < p.lb[q]) || (t > p.ub[q]);
                xp[q] = fminf(fmaxf(t, p.lb[q]), p.ub[q]);
            }
            const float uk = u;
            bool acc;
            if constexpr (SCREEN > 0) {
                const Screen cp = screen_eval(p.P, nm, xp, yr);
                draws(k + 1, nrm, u);
                int d = screen_decide(nm, cs, cp, 0.0f, 1.0f, uk);
                if (d < 0 && !oob)
                    d = exact_accept(s_P, nm, x[0], x[1], x[2], xp[0], xp[1], xp[2], yv, p.nvox, 0.0f, 1.0f, uk);
                acc = !oob && d > 0;
                if (acc) cs = cp;
            } else {
                const double lpp = log_prob_t<MODEL, NV>(nm, s_P, xp, yv, p.nvox, wv, p.nvox, va);
                draws(k + 1, nrm, u);
                acc = !oob && (lpp - lp) > (double)logf(uk);
                if (acc) lp = lpp;
            }
            if (acc) {
#pragma unroll
                for (int q = 0; q < NV; ++q) x[q] = xp[q];
                ++nacc;
            }
            if (k == kept_k) {
                kept_k += p.thinning;
                const int c = kept_index(p, k);
                if (c >= 0)
#pragma unroll
                    for (int j = 0; j < NV; ++j) {
                        double d = (double)x[j] - (double)p.shift[(size_t)j * p.nvox + v];
                        s1[j] += d;
                        s2[j] += d * d;
                        if (p.posterior)
                            p.posterior[(((size_t)j * p.repetition + rr) * p.ns + c) * p.nvox + v] = x[j];
                    }
            }
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) xstate[(size_t)q * p.nvox + v] = x[q];
        if constexpr (SCREEN == 0) lpstate[v] = lp;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            sum[(size_t)j * p.nvox + v] += s1[j];
            sumsq[(size_t)j * p.nvox + v] += s2[j];
        }
    }
    unsigned int wsum = nacc;
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if ((threadIdx.x & 31) == 0 && wsum) atomicAdd(p.n_acc, (unsigned long long)wsum);
}

// ---------------------------------------------------------------------------
// Metropolis-Hastings for few voxels (screened R2*).  With a warp or less a
// scheduler a chain is bound by its own latencies, and half of a step's
// instructions are its draws, which no state enters.  A CTA takes 32 voxels:
// warps 1-3 make the draws of the next kMhBatch steps into one of two shared
// buffers while warp 0 runs the chains through the other, one barrier a batch.
// Same draws, same decisions as mh_kernel.  Seven drawing warps measured
// slower (2.8 against 2.6 ms below).
// Whole call, 12 echoes, mh_kernel -> this one: 1000 voxels x 10,000 steps
// 5.9 -> 2.3 ms, 4096 x 10,000 6.25 -> 2.6, 10,000 x 10,000 6.6 -> 3.8,
// 20,000 x 4000 4.25 -> 3.55, 40,000 x 3000 6.64 -> 6.70: six chain warps an
// SM are the line; beyond, the chains fill each other's latencies anyway.
// ---------------------------------------------------------------------------
constexpr int kMhBatch = 16;
constexpr int kMhBatchVoxels = 148 * 6 * 32;

template <int MAXM>
__global__ void __launch_bounds__(128)
mh_batch_kernel(McmcParams p, int rr, int k0, int k1, int init, float* xstate, double* sum, double* sumsq) {
    constexpr int NV = 3;
    __shared__ DevProtocol s_P;
    __shared__ float4 s_draw[2][kMhBatch][32];  // three normals, the acceptance uniform
    stage_protocol(p.P, &s_P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v = blockIdx.x * 32 + lane;
    const bool live = v < p.nvox;
    const int nm = p.nm;
    auto make = [&](int first, float4 (*buf)[32]) {  // steps first, first + 1, .. of a batch, by warps 1-3
        const uint32_t tag = kTagMhMove | ((uint32_t)rr << 16);
        for (int i = warp - 1; i < kMhBatch && first + i <= k1; i += 3) {
            const uint32_t k = (uint32_t)(first + i);
            const U4 r = philox((uint32_t)v, k, 0u, tag, p.seed);
            float n0, n1, n2, n3;
            box_muller(r.x, r.y, n0, n1);
            box_muller(r.z, r.w, n2, n3);
            buf[i][lane] = make_float4(n0, n1, n2, u01(philox((uint32_t)v, k, 8u, tag, p.seed).x));
        }
    };
    float x[NV], yr[MAXM];
    double s1[NV], s2[NV];
    Screen cs{0.0f, 0.0f};
    unsigned int nacc = 0;
    int kept_k = 0;
    const float* yv = p.data + (live ? v : 0);
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            s1[q] = s2[q] = 0.0;
            // a lane without a voxel runs along on a harmless state and writes nothing
            x[q] = !live ? 1.0f
                   : init ? fminf(fmaxf(p.x0[(size_t)q * p.nvox + v], p.lb[q]), p.ub[q])
                          : xstate[(size_t)q * p.nvox + v];
        }
#pragma unroll
        for (int m = 0; m < MAXM; ++m) yr[m] = m < nm ? yv[(size_t)m * p.nvox] : 0.0f;
        cs = screen_eval(p.P, nm, x, yr);
        kept_k = first_kept(p, k0);
    } else {
        make(k0, s_draw[0]);
    }
    __syncthreads();
    for (int kb = k0, b = 0; kb <= k1; kb += kMhBatch, b ^= 1) {
        if (warp > 0) {
            make(kb + kMhBatch, s_draw[b ^ 1]);
        } else {
            const int n = min(kMhBatch, k1 - kb + 1);
            float4 d = s_draw[b][0][lane];
            for (int i = 0; i < n; ++i) {
                const float4 dn = s_draw[b][min(i + 1, n - 1)][lane];
                const float nrm[NV] = {d.x, d.y, d.z}, uk = d.w;
                float xp[NV];
                bool oob = false;
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    float t = x[q] + p.xstep[q] * nrm[q];
                    oob |= (t < p.lb[q]) || (t > p.ub[q]);
                    xp[q] = fminf(fmaxf(t, p.lb[q]), p.ub[q]);
                }
                const Screen cp = screen_eval(p.P, nm, xp, yr);
                int dec = screen_decide(nm, cs, cp, 0.0f, 1.0f, uk);
                if (dec < 0 && !oob && live)
                    dec = exact_accept(s_P, nm, x[0], x[1], x[2], xp[0], xp[1], xp[2], yv, p.nvox, 0.0f, 1.0f, uk);
                const bool acc = !oob && dec > 0;
                if (acc) {
                    cs = cp;
                    ++nacc;
                }
#pragma unroll
                for (int q = 0; q < NV; ++q) x[q] = acc ? xp[q] : x[q];
                if (kb + i == kept_k) {
                    kept_k += p.thinning;
                    const int c = kept_index(p, kb + i);
                    if (c >= 0 && live)
#pragma unroll
                        for (int j = 0; j < NV; ++j) {
                            double e = (double)x[j] - (double)p.shift[(size_t)j * p.nvox + v];
                            s1[j] += e;
                            s2[j] += e * e;
                            if (p.posterior)
                                p.posterior[(((size_t)j * p.repetition + rr) * p.ns + c) * p.nvox + v] = x[j];
                        }
                }
                d = dn;
            }
        }
        __syncthreads();
    }
    if (warp > 0) return;
    if (live) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            xstate[(size_t)q * p.nvox + v] = x[q];
            sum[(size_t)q * p.nvox + v] += s1[q];
            sumsq[(size_t)q * p.nvox + v] += s2[q];
        }
    } else {
        nacc = 0;
    }
    for (int o = 16; o > 0; o >>= 1) nacc += __shfl_xor_sync(0xffffffffu, nacc, o);
    if (lane == 0 && nacc) atomicAdd(p.n_acc, (unsigned long long)nacc);
}

// ---------------------------------------------------------------------------
// goodman_weare_wglobal_constant (mcmc.m:385-578) and gw_global_block
// (:581-626).  One iteration = a local stretch move per (voxel, walker) with
// the walker's globals held (z^(NND-1)), then a global stretch move per walker
// with the locals held (z^(NGlobal-1)), accepted on the log-likelihood
// difference summed over all voxels in FP64.  The voxel sum is a grid-wide
// dependency, so an iteration is two launches (four with red-black):
//   gwg_step_kernel    apply the previous global decision to the cached logP,
//                      local block, kept local samples, and the logP of the
//                      global proposal with per-CTA partial sums;
//   gwg_accept_kernel  one CTA per walker: partial sums in a fixed order,
//                      accept / reject, kept global samples.
// The step kernel's first CTA publishes each global proposal (with its
// stretch factor, acceptance uniform and bounds flag); the accept kernel reads
// it, so no CTA reads a global value another CTA of the same launch updates.
// ---------------------------------------------------------------------------
enum GwgFlags { kGwgInit = 1, kGwgApply = 2, kGwgLocal = 4, kGwgEval = 8 };

// Row of the global partner table and the Philox tag bits of one global block.
__device__ __forceinline__ int gwg_row(const McmcParams& p, int rr, int k, int warm) {
    return rr * p.nsteps_g + (warm ? p.iteration + k - 1 : k - 1);
}

__device__ __forceinline__ bool gwg_active(int half, int w, int W) {
    return half < 0 || (half == 0 ? w < W / 2 : w >= W / 2);
}

// Global proposal of walker w: g(anchor) + (g(w) - g(anchor)) * z, clamped;
// g(walker, q) = g[walker * nvar + q].  Returns true when out of bounds.
__device__ bool gwg_proposal(const McmcParams& p, int rr, int k, int warm, int w, const float* g, float* out,
                             float& zz, float& lu) {
    const int q0 = p.gpartner[(size_t)gwg_row(p, rr, k, warm) * p.nwalker + w];
    uint32_t tag = kTagGwGMove | ((uint32_t)rr << 16) | (warm ? kTagWarmup : 0u) | (p.update ? kTagRedBlack : 0u);
    U4 u = philox((uint32_t)w, (uint32_t)k, 0u, tag, p.seed);
    float t = (p.a - 1.0f) * u01(u.x) + 1.0f;
    zz = t * t / p.a;
    lu = logf(u01(u.y));
    bool oob = false;
    const int nvar = p.nvar;
    for (int q = 0; q < nvar; ++q) {
        if (!p.is_global[q]) { out[q] = 0.0f; continue; }
        float gq = g[q0 * nvar + q];
        float val = gq + (g[w * nvar + q] - gq) * zz;
        oob |= (val < p.lb[q]) || (val > p.ub[q]);
        out[q] = fminf(fmaxf(val, p.lb[q]), p.ub[q]);
    }
    return oob;
}

// Start value of global q for walker w: uniform over [lb, ub] (mcmc.m:488).
__device__ __forceinline__ float gwg_global_init(const McmcParams& p, int w, int q) {
    U4 u = philox((uint32_t)w, (uint32_t)(q >> 2), 0u, kTagGwGInit, p.seed);
    uint32_t r = (q & 3) == 0 ? u.x : (q & 3) == 1 ? u.y : (q & 3) == 2 ? u.z : u.w;
    return p.lb[q] + (p.ub[q] - p.lb[q]) * u01(r);
}

// One thread per (voxel, walker); blockDim = vpb * W.  NV = parameters +
// noise at compile time (per-thread vectors in registers).
template <int MODEL, int NV>
__global__ void gwg_step_kernel(McmcParams p, int rr, int k, int warm, int flags, int half, float* xstate,
                                double* lpstate) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ DevProtocol s_P;
    stage_protocol(p.P, &s_P);
    constexpr int nvar = NV;
    const int W = p.nwalker, nm = p.nm, h = W / 2;
    const int vpb = blockDim.x / W;
    const int vl = threadIdx.x / W, w = threadIdx.x % W;
    const int v = blockIdx.x * vpb + vl;
    const bool live = v < p.nvox;
    double* s_red = reinterpret_cast<double*>(smem_raw);          // [vpb][W]
    float* xs = reinterpret_cast<float*>(s_red + vpb * W);         // [vpb][W][nvar] locals
    float* s_g = xs + vpb * W * nvar;                              // [W][nvar] globals
    float* s_gp = s_g + W * nvar;                                  // [W][nvar] global proposals
    float* ys = s_gp + W * nvar;                                   // [vpb][nm]
    float* ws = ys + vpb * nm;                                     // [vpb][nm]
    float* xv = xs + vl * W * nvar;
    const float* yv = ys + vl * nm;
    const float* wv = p.weights ? ws + vl * nm : nullptr;
    if (live)
        for (int m = w; m < nm; m += W) {
            ys[vl * nm + m] = p.data[(size_t)m * p.nvox + v];
            if (p.weights) ws[vl * nm + m] = p.weights[(size_t)m * p.nvox + v];
        }
    for (int i = threadIdx.x; i < W * nvar; i += blockDim.x) {
        int ww = i / nvar, q = i % nvar;
        float gv = 0.0f;
        if (p.is_global[q]) gv = (flags & kGwgInit) ? gwg_global_init(p, ww, q) : p.gstate[(size_t)q * W + ww];
        s_g[i] = gv;
        if ((flags & kGwgInit) && blockIdx.x == 0 && p.is_global[q]) p.gstate[(size_t)q * W + ww] = gv;
    }
    float b1 = (live && p.b1) ? p.b1[v] : 1.0f;
    float sa[MODEL == kR1R2S ? kMaxFA : 1], ca[MODEL == kR1R2S ? kMaxFA : 1];
    if (MODEL == kR1R2S)
        for (int f = 0; f < p.P.n_fa; ++f) sincosf(b1 * p.P.fa_rad[f], &sa[f], &ca[f]);
    VoxAux va{b1, sa, ca, 1};
    if constexpr (kIsNexi<MODEL>)
        if (p.node_smem) {
            NexiNodes* s_nodes = reinterpret_cast<NexiNodes*>(
                smem_raw + ((sizeof(double) * vpb * W + sizeof(float) * (vpb * W * nvar + 2 * W * nvar + 2 * vpb * nm) + 15) &
                            ~(size_t)15));
            stage_nodes(p.nodes, s_nodes);
            va.nodes = s_nodes;
        }
    float x[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) x[q] = 0.0f;
    if (live) {
        if (flags & kGwgInit) {
            // locals: x0 + (ub-lb)*startRange*randn, clamped (mcmc.m:483-484), goodman_weare's stream
            float xi[NV];
            gw_walker_start<NV>(p, v, w, xi);
#pragma unroll
            for (int q = 0; q < NV; ++q)
                if (!p.is_global[q]) x[q] = xi[q];
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q)
                if (!p.is_global[q]) x[q] = xstate[((size_t)q * p.nvox + v) * W + w];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) xv[w * NV + q] = x[q];
    }
    __syncthreads();
    // parameter vector of (this voxel, walker ww) with globals gsrc
    auto compose = [&](const float (&loc)[NV], const float* gsrc, float (&out)[NV]) {
#pragma unroll
        for (int q = 0; q < NV; ++q) out[q] = p.is_global[q] ? gsrc[q] : loc[q];
    };
    double lp = 0.0;
    if (live) {
        if (flags & kGwgInit) {
            float xx[NV];
            compose(x, s_g + w * nvar, xx);
            lp = log_prob_t<MODEL, NV>(nm, s_P, xx, yv, 1, wv, 1, va);
        } else {
            lp = lpstate[(size_t)v * W + w];
            if ((flags & kGwgApply) && p.gacc[w]) lp = p.lpg[(size_t)v * W + w];
        }
    }
    unsigned int nacc = 0;
    if (flags & kGwgLocal) {
        const int* pt = p.partner + ((size_t)rr * p.iteration + (k - 1)) * W;
        const float expo = (float)(p.nnd - 1);
        for (int s = 0; s < (p.update == 0 ? 1 : 2); ++s) {
            const bool act = live && (p.update == 0 || (s == 0 ? w < h : w >= h));
            float xn[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) xn[q] = 0.0f;
            bool acc = false;
            double lpp = 0.0;
            if (act) {
                int q0 = pt[w];
                uint32_t tag = kTagGwMove | ((uint32_t)rr << 16) | (p.update ? kTagRedBlack : 0u);
                U4 u = philox((uint32_t)v, (uint32_t)w, (uint32_t)k, tag, p.seed);
                float t = (p.a - 1.0f) * u01(u.x) + 1.0f;
                float zz = t * t / p.a;
                bool oob = false;
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    if (p.is_global[q]) { xn[q] = 0.0f; continue; }
                    float xq = xv[q0 * nvar + q];
                    float xp = xq + (xv[w * nvar + q] - xq) * zz;
                    oob |= (xp < p.lb[q]) || (xp > p.ub[q]);
                    xn[q] = fminf(fmaxf(xp, p.lb[q]), p.ub[q]);
                }
                float xx[NV];
                compose(xn, s_g + w * nvar, xx);
                lpp = log_prob_t<MODEL, NV>(nm, s_P, xx, yv, 1, wv, 1, va);
                double lr = (double)expo * (double)logf(zz) + (lpp - lp);
                acc = !oob && lr > (double)logf(u01(u.y));
            }
            __syncthreads();  // the (half-)ensemble was read before any walker moves
            if (act && acc) {
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    x[q] = xn[q];
                    xv[w * NV + q] = xn[q];
                }
                lp = lpp;
                ++nacc;
            }
            __syncthreads();
        }
        // kept local samples: per voxel, summed over walkers in order (no atomics)
        int c = warm ? -1 : kept_index(p, k);
        if (c >= 0 && live) {
            for (int q = w; q < nvar; q += W) {
                if (p.is_global[q]) continue;
                double sh = (double)p.shift[(size_t)q * p.nvox + v], s1 = 0.0, s2 = 0.0;
                for (int ww = 0; ww < W; ++ww) {
                    double d = (double)xv[ww * nvar + q] - sh;
                    s1 += d;
                    s2 += d * d;
                }
                p.sum[(size_t)q * p.nvox + v] += s1;
                p.sumsq[(size_t)q * p.nvox + v] += s2;
            }
            if (p.posterior)
#pragma unroll
                for (int q = 0; q < NV; ++q)
                    if (!p.is_global[q])
                        p.posterior[((((size_t)q * p.repetition + rr) * p.ns + c) * W + w) * p.nvox + v] = x[q];
        }
    }
    if (flags & kGwgEval) {
        for (int ww = threadIdx.x; ww < W; ww += blockDim.x) {
            if (!gwg_active(half, ww, W)) continue;
            float zz, lu;
            bool oob = gwg_proposal(p, rr, k, warm, ww, s_g, s_gp + ww * nvar, zz, lu);
            if (blockIdx.x == 0) {  // published for the accept kernel
                for (int q = 0; q < nvar; ++q) p.gprop[(size_t)q * W + ww] = s_gp[ww * nvar + q];
                p.gzz[ww] = zz;
                p.glu[ww] = lu;
                p.goob[ww] = oob ? 1 : 0;
            }
        }
        __syncthreads();
        const bool act = gwg_active(half, w, W);
        double d = 0.0;
        if (live && act) {
            float xx[NV];
            compose(x, s_gp + w * nvar, xx);
            double lpg = log_prob_t<MODEL, NV>(nm, s_P, xx, yv, 1, wv, 1, va);
            p.lpg[(size_t)v * W + w] = lpg;
            d = lpg - lp;
        }
        s_red[vl * W + w] = d;
        __syncthreads();
        if (vl == 0 && act) {
            double t = 0.0;
            for (int j = 0; j < vpb; ++j) t += s_red[j * W + w];
            p.partial[(size_t)w * gridDim.x + blockIdx.x] = t;
        }
    }
    if (live) {
#pragma unroll
        for (int q = 0; q < NV; ++q)
            if (!p.is_global[q]) xstate[((size_t)q * p.nvox + v) * W + w] = x[q];
        lpstate[(size_t)v * W + w] = lp;
    }
    unsigned int wsum = nacc;
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if ((threadIdx.x & 31) == 0 && wsum) atomicAdd(p.n_acc, (unsigned long long)wsum);
}

// One CTA per walker (grid = W).  c >= 0: record the kept global sample c.
__global__ void gwg_accept_kernel(McmcParams p, int rr, int k, int warm, int half, int c, int nparts) {
    __shared__ double red[256];
    __shared__ float s_g[kMaxParam];
    const int w = blockIdx.x, W = p.nwalker;
    const bool act = gwg_active(half, w, W);
    double t = 0.0;
    if (act)
        for (int i = threadIdx.x; i < nparts; i += blockDim.x) t += p.partial[(size_t)w * nparts + i];
    red[threadIdx.x] = t;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int acc = 0;
        float gp[kMaxParam];
        if (act) {
            // the proposal the step kernel evaluated (mcmc.m:598-603)
            for (int q = 0; q < p.nvar; ++q) gp[q] = p.gprop[(size_t)q * W + w];
            double lr = (double)(p.ng - 1) * (double)logf(p.gzz[w]) + red[0];
            acc = !p.goob[w] && lr > (double)p.glu[w];
            if (acc) {
                for (int q = 0; q < p.nvar; ++q)
                    if (p.is_global[q]) p.gstate[(size_t)q * W + w] = gp[q];
                atomicAdd(p.n_gacc, 1ull);
            }
        }
        p.gacc[w] = acc;
        for (int q = 0; q < p.nvar; ++q) s_g[q] = p.gstate[(size_t)q * W + w];
        if (c >= 0)
            for (int q = 0; q < p.nvar; ++q)
                if (p.is_global[q]) {
                    double d = (double)s_g[q] - (double)p.shift[(size_t)q * p.nvox];
                    p.gsum[(size_t)q * W + w] += d;
                    p.gsumsq[(size_t)q * W + w] += d * d;
                }
    }
    __syncthreads();
    if (c >= 0 && p.posterior)
        for (int q = 0; q < p.nvar; ++q)
            if (p.is_global[q])
                for (int v = threadIdx.x; v < p.nvox; v += blockDim.x)
                    p.posterior[((((size_t)q * p.repetition + rr) * p.ns + c) * W + w) * p.nvox + v] = s_g[q];
}

// mean / std of the global parameters over W * ns * rep samples (unfilled
// slots count as zeros, as for the locals), repeated for every voxel.
__global__ void gwg_finalize_kernel(McmcParams p, int missing, float* mean, float* stdv) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= p.nvox) return;
    const int W = p.nwalker;
    double N = (double)W * p.ns * p.repetition;
    for (int q = 0; q < p.nvar; ++q) {
        if (!p.is_global[q]) continue;
        double sh = (double)p.shift[(size_t)q * p.nvox];
        double s1 = 0.0, s2 = 0.0;
        for (int w = 0; w < W; ++w) {
            s1 += p.gsum[(size_t)q * W + w];
            s2 += p.gsumsq[(size_t)q * W + w];
        }
        double nz = (double)missing * W * p.repetition;
        s1 += nz * (-sh);
        s2 += nz * sh * sh;
        double md = s1 / N;
        double var = N > 1.0 ? (s2 - s1 * md) / (N - 1.0) : 0.0;
        if (mean) mean[(size_t)q * p.nvox + v] = (float)(sh + md);
        if (stdv) stdv[(size_t)q * p.nvox + v] = (float)sqrt(fmax(var, 0.0));
    }
}

// shift = clamp(x0): the running sums are taken about the start value.
__global__ void mcmc_shift_kernel(McmcParams p) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= p.nvox) return;
    for (int q = 0; q < p.nvar; ++q)
        p.shift[(size_t)q * p.nvox + v] = fminf(fmaxf(p.x0[(size_t)q * p.nvox + v], p.lb[q]), p.ub[q]);
}

// mean / std (N-1) over W*ns*rep samples; slots the reference preallocates
// but never fills stay zero and are counted (res2out, mcmc.m:806-862).
__global__ void mcmc_finalize_kernel(McmcParams p, int missing, float* mean, float* stdv) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= p.nvox) return;
    int W = p.algorithm == 1 ? p.nwalker : 1;
    double N = (double)W * p.ns * p.repetition;
    for (int q = 0; q < p.nvar; ++q) {
        size_t i = (size_t)q * p.nvox + v;
        double sh = (double)p.shift[i];
        double s1 = p.sum[i], s2 = p.sumsq[i];
        double nz = (double)missing * W * p.repetition;
        s1 += nz * (-sh);
        s2 += nz * sh * sh;
        double md = s1 / N;
        double var = N > 1.0 ? (s2 - s1 * md) / (N - 1.0) : 0.0;
        if (mean) mean[i] = (float)(sh + md);
        if (stdv) stdv[i] = (float)sqrt(fmax(var, 0.0));
    }
}

cudaError_t launch_mcmc_partners(const McmcParams& p, int* partner, cudaStream_t s) {
    int n = p.repetition * p.iteration;
    int block = 128;
    gw_partner_kernel<<<(n + block - 1) / block, block, 0, s>>>(p, partner, p.iteration, 0);
    ++g_kernel_launches;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || p.ng == 0) return e;
    n = p.repetition * p.nsteps_g;
    gw_partner_kernel<<<(n + block - 1) / block, block, 0, s>>>(p, const_cast<int*>(p.gpartner), p.nsteps_g, 1);
    ++g_kernel_launches;
    return cudaGetLastError();
}

// Goodman-Weare launch shape for a block hint (threads): whole voxels of
// tpv threads (one walker, or one walker of each half) per CTA.
static void gw_shape(const McmcParams& p, int block_hint, int* vpb, int* block, size_t* smem) {
    const int W = p.nwalker, h = W / 2;
    const int tpv = p.update == 0 ? W : W - h;
    const int target = block_hint > 0 ? block_hint : 128;
    *vpb = target / tpv > 0 ? target / tpv : 1;
    *block = *vpb * tpv;
    *smem = sizeof(double) * 2 * (size_t)(*vpb) * W * p.nvar +
            sizeof(float) * ((size_t)(*vpb) * W * p.nvar + 2 * (size_t)(*vpb) * p.nm);
}

// The screen's bound holds for a sum of squares (no weights) and for noises
// (clamped to their bounds in every state) in its range; its measurements are
// held in registers.
static bool screened(const McmcParams& p) {
    return p.weights == nullptr && p.nm <= kScreenM && p.lb[p.nvar - 1] >= kScreenMinNoise &&
           p.ub[p.nvar - 1] <= kScreenMaxNoise;
}

bool mcmc_screened(const McmcParams& p, int model) { return model == kR2S && screened(p); }

bool mcmc_batched(const McmcParams& p, int model) {
    return p.algorithm == 0 && mcmc_screened(p, model) && p.nvox <= kMhBatchVoxels;
}

template <int MODEL>
static decltype(&mh_kernel<MODEL, ModelNP<MODEL>::value + 1, 0>) mh_kernel_fn(const McmcParams& p) {
    constexpr int NV = ModelNP<MODEL>::value + 1;
    if constexpr (MODEL == kR2S)
        if (screened(p))
            return p.nm <= 8 ? mh_kernel<MODEL, NV, 8> : p.nm <= 12 ? mh_kernel<MODEL, NV, 12> : mh_kernel<MODEL, NV, 16>;
    return mh_kernel<MODEL, NV, 0>;
}

// Threads per block of a Metropolis-Hastings launch: the chosen block up to what the
// kernel's registers leave (a chain does not depend on its block).
template <class K>
static cudaError_t mh_block_of(K kernel, int block_hint, int* block) {
    *block = block_hint > 0 ? block_hint : 128;
    if (*block <= 512 || *block > 1024) return cudaSuccess;  // always fits; refused by the launch
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e == cudaSuccess) *block = std::min(*block, fa.maxThreadsPerBlock / 32 * 32);
    return e;
}

int mcmc_mh_block(const McmcParams& p, int model, int block_hint) {
    int block = block_hint;
    if (mcmc_batched(p, model) && block_hint <= 0) return 128;
    switch (model) {
    case kR2S: mh_block_of(mh_kernel_fn<kR2S>(p), block_hint, &block); break;
    case kR1R2S: mh_block_of(mh_kernel_fn<kR1R2S>(p), block_hint, &block); break;
    case kNEXI: mh_block_of(mh_kernel_fn<kNEXI>(p), block_hint, &block); break;
    default: mh_block_of(mh_kernel_fn<kNEXI2>(p), block_hint, &block); break;
    }
    return block;
}

// Steps [k0, k1] of repetition rr as one launch (init: the walkers start at k0 == 1).
template <int MODEL>
static cudaError_t mcmc_launch_steps(McmcParams p, int block_hint, int rr, int k0, int k1, float* xstate,
                                     double* lpstate, double* sum, double* sumsq, cudaStream_t s) {
    constexpr int NV = ModelNP<MODEL>::value + 1;  // the model's parameters and the noise sigma
    if (p.nvar != NV) return cudaErrorInvalidValue;
    if (p.algorithm == 1) {
        int vpb, block;
        size_t smem;
        gw_shape(p, block_hint, &vpb, &block, &smem);
        const int nb = (p.nvox + vpb - 1) / vpb;
        auto k = p.update == 0 ? gw_kernel<MODEL, NV, false, 0> : gw_kernel<MODEL, NV, true, 0>;
        if constexpr (MODEL == kR2S)
            if (screened(p))
                k = p.nm <= 8    ? (p.update == 0 ? gw_kernel<MODEL, NV, false, 8> : gw_kernel<MODEL, NV, true, 8>)
                    : p.nm <= 12 ? (p.update == 0 ? gw_kernel<MODEL, NV, false, 12> : gw_kernel<MODEL, NV, true, 12>)
                                 : (p.update == 0 ? gw_kernel<MODEL, NV, false, 16> : gw_kernel<MODEL, NV, true, 16>);
        if (kIsNexi<MODEL>) p.node_smem = nodes_fit(&smem);
        if (smem + sizeof(DevProtocol) > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
        k<<<nb, block, smem, s>>>(p, rr, k0, k1, k0 == 1 ? 1 : 0, xstate, lpstate, sum, sumsq);
    } else {
        if constexpr (MODEL == kR2S)
            if (block_hint <= 0 && mcmc_batched(p, MODEL)) {
                auto kb = p.nm <= 8 ? mh_batch_kernel<8> : p.nm <= 12 ? mh_batch_kernel<12> : mh_batch_kernel<16>;
                kb<<<(p.nvox + 31) / 32, 128, 0, s>>>(p, rr, k0, k1, k0 == 1 ? 1 : 0, xstate, sum, sumsq);
                ++g_kernel_launches;
                return cudaGetLastError();
            }
        auto k = mh_kernel_fn<MODEL>(p);
        int block;
        const cudaError_t e = mh_block_of(k, block_hint, &block);
        if (e != cudaSuccess) return e;
        const int nb = (p.nvox + block - 1) / block;
        k<<<nb, block, 0, s>>>(p, rr, k0, k1, k0 == 1 ? 1 : 0, xstate, lpstate, sum, sumsq);
    }
    ++g_kernel_launches;
    return cudaGetLastError();
}

// Steps per launch: a bounded kernel duration (below a second for a million
// walkers), and enough steps that few walkers do not spend their time on
// launches, each of which reloads the state.
int mcmc_steps_per_launch(const McmcParams& p) {
    const size_t walkers = (size_t)p.nvox * (p.algorithm == 1 ? p.nwalker : 1);
    return (int)std::min<size_t>(5000, std::max<size_t>(250, 250000000 / walkers));
}

template <int MODEL>
static cudaError_t mcmc_run_model(const McmcParams& p, int block_hint, cudaStream_t s,
                                  float* xstate, double* lpstate) {
    const int chunk = mcmc_steps_per_launch(p);
    for (int rr = 0; rr < p.repetition; ++rr)
        for (int k0 = 1; k0 <= p.iteration; k0 += chunk) {
            int k1 = k0 + chunk - 1 < p.iteration ? k0 + chunk - 1 : p.iteration;
            cudaError_t e = mcmc_launch_steps<MODEL>(p, block_hint, rr, k0, k1, xstate, lpstate, p.sum, p.sumsq, s);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

int mcmc_block_candidates(const McmcParams& p, int* out, int maxn) {
    int n = 0;
    if (p.algorithm == 1) {
        const int W = p.nwalker, tpv = p.update == 0 ? W : W - W / 2;
        for (int vpb = 1; vpb <= 32 && n < maxn; vpb *= 2) {
            const int block = vpb * tpv;
            if (block > 1024) break;
            if (block < 32 && vpb < 32) continue;  // at least one warp
            out[n++] = block;
        }
    } else {
        for (int b = 32; b <= 512 && n < maxn; b *= 2) out[n++] = b;
    }
    return n;
}

cudaError_t launch_mcmc_trial(const McmcParams& p, int model, int block_hint, int k1, float* xstate,
                              double* lpstate, double* sum, double* sumsq, cudaStream_t s) {
    switch (model) {
    case kR2S: return mcmc_launch_steps<kR2S>(p, block_hint, 0, 1, k1, xstate, lpstate, sum, sumsq, s);
    case kR1R2S: return mcmc_launch_steps<kR1R2S>(p, block_hint, 0, 1, k1, xstate, lpstate, sum, sumsq, s);
    case kNEXI: return mcmc_launch_steps<kNEXI>(p, block_hint, 0, 1, k1, xstate, lpstate, sum, sumsq, s);
    default: return mcmc_launch_steps<kNEXI2>(p, block_hint, 0, 1, k1, xstate, lpstate, sum, sumsq, s);
    }
}

int kept_index_host(const McmcParams& p, int k) {
    if (k <= p.nburnin) return -1;
    int j = k - p.nburnin + 1;
    if (j % p.thinning) return -1;
    int c = j / p.thinning - (p.thinning == 1 ? 1 : 0) - 1;
    return c < p.ns ? c : -1;
}

void gwg_launch_shape(const McmcParams& p, int block_hint, int* vpb, int* block, int* nblocks, size_t* smem) {
    const int W = p.nwalker;
    int target = block_hint > 0 ? block_hint : 256;
    *vpb = target / W > 0 ? target / W : 1;
    *block = *vpb * W;
    *nblocks = (p.nvox + *vpb - 1) / *vpb;
    *smem = sizeof(double) * (size_t)(*vpb) * W +
            sizeof(float) * ((size_t)(*vpb) * W * p.nvar + 2 * (size_t)W * p.nvar + 2 * (size_t)(*vpb) * p.nm);
}

template <int MODEL>
static cudaError_t mcmc_run_global(McmcParams p, int block_hint, cudaStream_t s, float* xstate,
                                   double* lpstate) {
    if (p.nvar != ModelNP<MODEL>::value + 1) return cudaErrorInvalidValue;
    int vpb, block, nb;
    size_t smem;
    gwg_launch_shape(p, block_hint, &vpb, &block, &nb, &smem);
    if (kIsNexi<MODEL>) p.node_smem = nodes_fit(&smem);
    if (smem + sizeof(DevProtocol) > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(gwg_step_kernel<MODEL, ModelNP<MODEL>::value + 1>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    auto A = [&](int rr, int k, int warm, int flags, int half) {
        gwg_step_kernel<MODEL, ModelNP<MODEL>::value + 1><<<nb, block, smem, s>>>(p, rr, k, warm, flags, half,
                                                                                  xstate, lpstate);
        ++g_kernel_launches;
    };
    auto B = [&](int rr, int k, int warm, int half, int c) {
        gwg_accept_kernel<<<p.nwalker, 256, 0, s>>>(p, rr, k, warm, half, c, nb);
        ++g_kernel_launches;
    };
    for (int rr = 0; rr < p.repetition; ++rr) {
        bool first = true;
        for (int kw = 1; kw <= p.global_warmup; ++kw) {
            int f = (first ? kGwgInit : kGwgApply) | kGwgEval;
            first = false;
            if (p.update == 0) {
                A(rr, kw, 1, f, -1);
                B(rr, kw, 1, -1, -1);
            } else {
                A(rr, kw, 1, f, 0);
                B(rr, kw, 1, 0, -1);
                A(rr, kw, 1, kGwgApply | kGwgEval, 1);
                B(rr, kw, 1, 1, -1);
            }
        }
        for (int k = 1; k <= p.iteration; ++k) {
            int f = (first ? kGwgInit : kGwgApply) | kGwgLocal | kGwgEval;
            first = false;
            int c = kept_index_host(p, k);
            if (p.update == 0) {
                A(rr, k, 0, f, -1);
                B(rr, k, 0, -1, c);
            } else {
                A(rr, k, 0, f, 0);
                B(rr, k, 0, 0, -1);
                A(rr, k, 0, kGwgApply | kGwgEval, 1);
                B(rr, k, 0, 1, c);
            }
            if ((k & 63) == 0) {
                cudaError_t e = cudaGetLastError();
                if (e != cudaSuccess) return e;
            }
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_mcmc(const McmcParams& p, int model, int block, float* xstate, double* lpstate, cudaStream_t s) {
    mcmc_shift_kernel<<<(p.nvox + 127) / 128, 128, 0, s>>>(p);
    ++g_kernel_launches;
    if (p.ng > 0) {
        switch (model) {
        case kR2S: return mcmc_run_global<kR2S>(p, block, s, xstate, lpstate);
        case kR1R2S: return mcmc_run_global<kR1R2S>(p, block, s, xstate, lpstate);
        case kNEXI: return mcmc_run_global<kNEXI>(p, block, s, xstate, lpstate);
        default: return mcmc_run_global<kNEXI2>(p, block, s, xstate, lpstate);
        }
    }
    switch (model) {
    case kR2S: return mcmc_run_model<kR2S>(p, block, s, xstate, lpstate);
    case kR1R2S: return mcmc_run_model<kR1R2S>(p, block, s, xstate, lpstate);
    case kNEXI: return mcmc_run_model<kNEXI>(p, block, s, xstate, lpstate);
    default: return mcmc_run_model<kNEXI2>(p, block, s, xstate, lpstate);
    }
}

int mcmc_missing_slots(const McmcParams& p) {
    // kept = #k in (nburnin, iteration] with (k - nburnin + 1) % thinning == 0
    int kept = 0;
    for (int k = p.nburnin + 1; k <= p.iteration; ++k)
        if ((k - p.nburnin + 1) % p.thinning == 0) ++kept;
    int missing = p.ns - kept;
    return missing < 0 ? 0 : missing;
}

cudaError_t launch_mcmc_finalize(const McmcParams& p, float* mean, float* stdv, cudaStream_t s) {
    const int missing = mcmc_missing_slots(p);
    mcmc_finalize_kernel<<<(p.nvox + 127) / 128, 128, 0, s>>>(p, missing, mean, stdv);
    ++g_kernel_launches;
    if (p.ng > 0) {
        gwg_finalize_kernel<<<(p.nvox + 127) / 128, 128, 0, s>>>(p, missing, mean, stdv);
        ++g_kernel_launches;
    }
    return cudaGetLastError();
}

}  // namespace gx
