// askadam_fused.cu -- multi-epoch askAdam kernels without spatial coupling for
// the configuration that most fits run: MSE, sigmoid transform, Adam, no prior.
//
//   fused_r2s_kernel    R2*, up to 16 echoes, one voxel a thread: measurements in
//                       registers, echo constants in the constant bank, the
//                       echoes unrolled.  For few voxels, where an epoch is one
//                       dependent chain.
//   fused_r2s_pairs     R2*, two voxels a thread in FP32x2 pair instructions.
//   fused_r1r2s_pairs   joint R1-R2*, two flip angles, up to 16 echoes, two
//                       voxels a thread.
//
// Per voxel each evaluates the operations of fused_kernel (askadam_kernels.cu),
// with the same roundings, so that the parameters are the same bit for bit;
// loss sums go through HistorySums.  Reference: utils/askadam.m:23-117,673-691.
#include "gx_history.cuh"

namespace gx {

namespace {

// The echoes of a protocol within a compile-time bound: without a test when
// the protocol fills it.
template <int MAXM, class F>
__device__ __forceinline__ void each_echo(int n, F&& f) {
    if (n == MAXM) {
#pragma unroll
        for (int m = 0; m < MAXM; ++m) f(m);
    } else {
#pragma unroll
        for (int m = 0; m < MAXM; ++m)
            if (m < n) f(m);
    }
}

__device__ __forceinline__ int first_checkpoint(const AdamParams& a, int e_begin) {
    return a.ckpt_every > 0 ? (e_begin + a.ckpt_every - 1) / a.ckpt_every * a.ckpt_every : 0x7fffffff;
}

}  // namespace

// ---------------------------------------------------------------------------
// R2*, one voxel a thread.  Bound, for few voxels, by the chain of one epoch
// (transform, exponentials, sums, square root and reciprocals of the step): 720
// clocks.  4096 voxels, 12 echoes, 2000 epochs: 1.76 ms with measurements and
// constants in shared memory, a loop over the echoes and a block reduction every
// epoch -> 0.755 ms.
// ---------------------------------------------------------------------------
template <int MAXM, bool STATS>
__global__ void fused_r2s_kernel(AdamParams a, int e_begin, int e_end, int update_last, int record) {
    constexpr int NP = 2, NQ = STATS ? kHistW : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int vol = a.blk_vol[blockIdx.x];
    const DevVol& V = a.vols[vol];
    const bool valid = (v - V.off) < V.nvox;
    const int nm = a.nm;
    PrefLossAcc<kMSE, NP, MAXM> acc;
    acc.load(a.data + v, a.nvtot, nm);
    acc.w = nullptr; acc.ws = 0;
    acc.aux = LossAux{0.0f, 0.0f};
    acc.mse_scale = a.mse_scale; acc.hd = 0.0f;
    acc.res = nullptr; acc.rs = a.nvtot;
    float z[NP], m1[NP], m2[NP], zp[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const size_t i = (size_t)k * a.nvtot + v;
        z[k] = a.z[i];
        m1[k] = a.m1[i];
        m2[k] = a.m2[i];
        zp[k] = STATS ? a.zprev[i] : 0.0f;
    }
    const float normf = V.norm;
    const OptConst oc{kAdam, a.beta1, a.beta2, a.eps, 0.0f, 0.0f, 0.0f};
    const size_t slot = (size_t)3 * NP * a.nvtot;
    int next_ck = first_checkpoint(a, e_begin);
    HistorySums<NQ> sums(reinterpret_cast<double*>(smem_raw), a.hist + (size_t)vol * (a.niter + 1) * kHistW, V.normd, e_begin);
    float2 sc = e_begin <= update_last ? a.sched[e_begin] : make_float2(0.f, 0.f);
    for (int e = e_begin; e <= e_end; ++e) {
        const float2 sc_next = e < update_last ? a.sched[e + 1] : make_float2(0.f, 0.f);  // in flight over the epoch
        float th[NP], dth[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) th[k] = unscale(0, a.P.lb[k], a.P.ub[k], z[k], dth[k]);
        acc.total = 0.0f;
        acc.g[0] = acc.g[1] = 0.0f;
        R2sMseSums u;
        each_echo<MAXM>(nm, [&](int m) { u.echo(a.P.te[m], a.P.te_l2e[m], th[0], th[1], acc.meas(m)); });
        u.store(th[0], acc);
        if (a.res_out && e == e_end && valid)
            each_echo<MAXM>(nm, [&](int m) {
                R2sMseSums t;
                const float r = t.echo(a.P.te[m], a.P.te_l2e[m], th[0], th[1], acc.meas(m));
                a.res_out[(size_t)m * a.nvtot + v] = a.mse_scale * r * r;
            });
        acc.finish();
        float gz[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) gz[k] = acc.g[k] * normf * dth[k];
        if (record) {
            float q[NQ];
            q[0] = valid ? acc.total : 0.0f;
            if constexpr (STATS) {
                float g2 = 0.f, z2 = 0.f, d2 = 0.f;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    g2 += gz[k] * gz[k];
                    z2 += z[k] * z[k];
                    d2 += (z[k] - zp[k]) * (z[k] - zp[k]);
                }
                q[1] = 0.0f;
                q[2] = valid ? g2 : 0.f;
                q[3] = valid ? z2 : 0.f;
                q[4] = valid ? d2 : 0.f;
            }
            sums.add(q, e_end);
        }
        if (e <= update_last) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                if (STATS) zp[k] = z[k];
                opt_step(oc, sc, z[k], m1[k], m2[k], gz[k]);
            }
            if (e == next_ck) {
                next_ck += a.ckpt_every;
                float* c = a.ckpt + (size_t)(e / a.ckpt_every) * slot;
                if (valid)
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        c[(size_t)k * a.nvtot + v] = z[k];
                        c[(size_t)(NP + k) * a.nvtot + v] = m1[k];
                        c[(size_t)(2 * NP + k) * a.nvtot + v] = m2[k];
                    }
            }
        }
        sc = sc_next;
    }
    if (record) sums.finish(e_end);
    if (valid) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const size_t i = (size_t)k * a.nvtot + v;
            a.z[i] = z[k];
            a.m1[i] = m1[k];
            a.m2[i] = m2[k];
            if (STATS) a.zprev[i] = zp[k];
        }
    }
}

// ---------------------------------------------------------------------------
// Pair kernels.  Bound: the SFU (per voxel-epoch an exponential an echo and four
// operations a parameter, 61 % of the epoch at R1-R2*, whose epoch took three
// times the instructions with one voxel a thread).  1.26 M voxels in six volumes, joint
// R1-R2*, 12 echoes x 2 angles, 400 epochs: 8.38 -> 4.93 ms (110 registers
// uncapped: 5.06, 64: 5.36); with stopping statistics (68 bytes spilled) one volume
// of as many voxels, whole call, 9.6 -> 6.6 ms.  R2*, 12 echoes, 500 epochs of 640,000 voxels:
// 2.21 ms one voxel a thread -> 1.73 ms.
// Two voxels a thread: thread t of a block takes voxels base + 64 (t / 32) +
// t % 32 and that + 32, lane .x and .y of the pair instructions.
// ---------------------------------------------------------------------------
namespace {

template <int NP, bool STATS>
struct PairState {
    float2 z[NP], m1[NP], m2[NP], zp[STATS ? NP : 1];
    int v0;            // second voxel at v0 + 32
    bool ok0, ok1;

    __device__ __forceinline__ void load(const AdamParams& a, const DevVol& V) {
        v0 = blockIdx.x * (blockDim.x * 2) + ((threadIdx.x >> 5) << 6) + (threadIdx.x & 31);
        ok0 = v0 - V.off < V.nvox;
        ok1 = v0 + 32 - V.off < V.nvox;
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const size_t i = (size_t)k * a.nvtot + v0;
            z[k] = make_float2(a.z[i], a.z[i + 32]);
            m1[k] = make_float2(a.m1[i], a.m1[i + 32]);
            m2[k] = make_float2(a.m2[i], a.m2[i + 32]);
            if constexpr (STATS) zp[k] = make_float2(a.zprev[i], a.zprev[i + 32]);
        }
    }
    // [z, m1, m2] rows of `p` (a checkpoint slot, or the three state arrays)
    __device__ __forceinline__ void put(float* p, size_t i, float2 x) const {
        if (ok0) p[i] = x.x;
        if (ok1) p[i + 32] = x.y;
    }
    __device__ __forceinline__ void checkpoint(float* c, size_t n) const {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            put(c, (size_t)k * n + v0, z[k]);
            put(c, (size_t)(NP + k) * n + v0, m1[k]);
            put(c, (size_t)(2 * NP + k) * n + v0, m2[k]);
        }
    }
    __device__ __forceinline__ void store(const AdamParams& a) const {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const size_t i = (size_t)k * a.nvtot + v0;
            put(a.z, i, z[k]);
            put(a.m1, i, m1[k]);
            put(a.m2, i, m2[k]);
            if constexpr (STATS) put(a.zprev, i, zp[k]);
        }
    }
    // loss and stopping statistics of both voxels (the first voxel's terms first)
    template <int NQ>
    __device__ __forceinline__ void quantities(float2 total, const float2 (&gz)[NP], float (&q)[NQ]) const {
        q[0] = (ok0 ? total.x : 0.0f) + (ok1 ? total.y : 0.0f);
        if constexpr (STATS) {
            float2 g2 = make_float2(0.f, 0.f), z2 = g2, d2 = g2;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                g2 = fma2(gz[k], gz[k], g2);
                z2 = fma2(z[k], z[k], z2);
                const float2 d = sub2(z[k], zp[k]);
                d2 = fma2(d, d, d2);
            }
            q[1] = 0.0f;
            q[2] = (ok0 ? g2.x : 0.0f) + (ok1 ? g2.y : 0.0f);
            q[3] = (ok0 ? z2.x : 0.0f) + (ok1 ? z2.y : 0.0f);
            q[4] = (ok0 ? d2.x : 0.0f) + (ok1 ? d2.y : 0.0f);
        }
    }
};

// The epochs of a pair kernel.  eval(th, total, g): the model's loss and
// derivatives (MSE sums before mse_finish's factors); resid(th, write): the
// residuals, write(m, r) for both voxels.
template <int NP, bool STATS, class Eval, class Resid>
__device__ __forceinline__ void pair_epochs(const AdamParams& a, const FusedPairConsts& k, const DevVol& V, int vol,
                                            PairState<NP, STATS>& s, double* shared, int e_begin, int e_end,
                                            int update_last, int record, Eval&& eval, Resid&& resid) {
    constexpr int NQ = STATS ? kHistW : 1;
    const float2 norm = bcast2(V.norm);
    const size_t slot = (size_t)3 * NP * a.nvtot;
    int next_ck = first_checkpoint(a, e_begin);
    HistorySums<NQ> sums(shared, a.hist + (size_t)vol * (a.niter + 1) * kHistW, V.normd, e_begin);
    float2 sc = e_begin <= update_last ? a.sched[e_begin] : make_float2(0.f, 0.f);
    for (int e = e_begin; e <= e_end; ++e) {
        const float2 sc_next = e < update_last ? a.sched[e + 1] : make_float2(0.f, 0.f);
        float2 th[NP], dth[NP], g[NP], gz[NP], total;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const float2 x = mul2(s.z[i], k.nl2e);
            const float2 den = add2(k.one, make_float2(ex2_ftz(x.x), ex2_ftz(x.y)));
            const float2 sg = make_float2(rcp_ftz(den.x), rcp_ftz(den.y));
            dth[i] = mul2(mul2(k.rng[i], sg), sub2(k.one, sg));
            th[i] = fma2(k.rng[i], sg, k.lb[i]);
        }
        eval(th, total, g);
        if (a.res_out && e == e_end)
            resid(th, [&](int m, float2 r) {
                if (s.ok0) a.res_out[(size_t)m * a.nvtot + s.v0] = a.mse_scale * r.x * r.x;
                if (s.ok1) a.res_out[(size_t)m * a.nvtot + s.v0 + 32] = a.mse_scale * r.y * r.y;
            });
        total = mul2(total, k.mse);
#pragma unroll
        for (int i = 0; i < NP; ++i) gz[i] = mul2(mul2(mul2(g[i], k.s2), norm), dth[i]);
        if (record) {
            float q[NQ];
            s.template quantities<NQ>(total, gz, q);
            sums.add(q, e_end);
        }
        if (e <= update_last) {
            const float2 nscx = bcast2(-sc.x), scy = bcast2(sc.y);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                if constexpr (STATS) s.zp[i] = s.z[i];
                s.m1[i] = fma2(k.b1, s.m1[i], mul2(k.omb1, gz[i]));
                s.m2[i] = fma2(k.b2, s.m2[i], mul2(mul2(k.omb2, gz[i]), gz[i]));
                const float2 w = mul2(s.m2[i], scy);
                const float2 den = add2(make_float2(fast_sqrt0(w.x), fast_sqrt0(w.y)), k.eps);
                s.z[i] = fma2(mul2(nscx, s.m1[i]), make_float2(rcp_ftz(den.x), rcp_ftz(den.y)), s.z[i]);
            }
            if (e == next_ck) {
                next_ck += a.ckpt_every;
                s.checkpoint(a.ckpt + (size_t)(e / a.ckpt_every) * slot, a.nvtot);
            }
        }
        sc = sc_next;
    }
    if (record) sums.finish(e_end);
    s.store(a);
}

}  // namespace

// R2*: both voxels' measurements in registers.
template <int MAXM, bool STATS>
__global__ void fused_r2s_pairs(AdamParams a, FusedPairConsts k, int e_begin, int e_end, int update_last, int record) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int vol = a.blk_vol[blockIdx.x];
    const DevVol& V = a.vols[vol];
    PairState<2, STATS> s;
    s.load(a, V);
    const int nm = a.nm;
    float2 ny[MAXM];  // minus the measurements
#pragma unroll
    for (int m = 0; m < MAXM; ++m)
        ny[m] = m < nm ? make_float2(-a.data[(size_t)m * a.nvtot + s.v0], -a.data[(size_t)m * a.nvtot + s.v0 + 32])
                       : make_float2(0.f, 0.f);
    const float2 zero = make_float2(0.f, 0.f);
    auto echo = [&](int m, float2 M0, float2 R2, float2& E) {
        const float2 x = mul2(a.P.nl2e_pair[m], R2);
        E = make_float2(ex2_ftz(x.x), ex2_ftz(x.y));
        return fma2(M0, E, ny[m]);
    };
    pair_epochs<2, STATS>(
        a, k, V, vol, s, reinterpret_cast<double*>(smem_raw), e_begin, e_end, update_last, record,
        [&](const float2 (&th)[2], float2& total, float2 (&g)[2]) {
            float2 sse = zero, g0 = zero, g1 = zero;
            each_echo<MAXM>(nm, [&](int m) {
                float2 E;
                const float2 r = echo(m, th[0], th[1], E);
                sse = fma2(r, r, sse);
                const float2 q = mul2(r, E);
                g0 = add2(g0, q);
                g1 = fma2(a.P.te_pair[m], q, g1);
            });
            total = sse;
            g[0] = g0;
            g[1] = fma2(make_float2(-th[0].x, -th[0].y), g1, zero);
        },
        [&](const float2 (&th)[2], auto&& write) {
            each_echo<MAXM>(nm, [&](int m) {
                float2 E;
                write(m, echo(m, th[0], th[1], E));
            });
        });
}

// Joint R1-R2* with two flip angles.  The measurements lie in shared memory,
// negated, one 16-byte access for both angles of both voxels at an echo time:
// [echo][thread] = (y_0(v0), y_0(v1), y_1(v0), y_1(v1)).
template <int MAXT, bool STATS>
__global__ void __maxnreg__(96) fused_r1r2s_pairs(AdamParams a, FusedPairConsts k, int e_begin, int e_end,
                                                         int update_last, int record) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int vol = a.blk_vol[blockIdx.x];
    const DevVol& V = a.vols[vol];
    PairState<3, STATS> s;
    s.load(a, V);
    const int T = blockDim.x, tid = threadIdx.x, nte = a.P.n_te;
    double* shared = reinterpret_cast<double*>(smem_raw);
    float4* sy = reinterpret_cast<float4*>(shared + HistorySums<STATS ? kHistW : 1>::buf_doubles(T >> 5)) + tid;
    for (int t = 0; t < nte; ++t) {
        const float* y0 = a.data + (size_t)t * a.nvtot + s.v0;
        const float* y1 = a.data + (size_t)(t + nte) * a.nvtot + s.v0;
        sy[t * T] = make_float4(-y0[0], -y0[32], -y1[0], -y1[32]);
    }
    float sa[2][2], ca[2][2];  // [angle][voxel]
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float b1 = a.b1 ? a.b1[s.v0 + 32 * h] : 1.0f;
#pragma unroll
        for (int f = 0; f < 2; ++f) sincosf(b1 * a.P.fa_rad[f], &sa[f][h], &ca[f][h]);
    }
    const float2 zero = make_float2(0.f, 0.f);
    // the steady-state factor of both voxels at an angle, and its derivative
    auto angle = [&](int f, float2 E1, float2& A, float2& dA) {
        r1r2s_angle(sa[f][0], ca[f][0], a.P.tr, E1.x, A.x, dA.x);
        r1r2s_angle(sa[f][1], ca[f][1], a.P.tr, E1.y, A.y, dA.y);
    };
    pair_epochs<3, STATS>(
        a, k, V, vol, s, shared, e_begin, e_end, update_last, record,
        [&](const float2 (&th)[3], float2& total, float2 (&g)[3]) {
            const float2 E1 = make_float2(__expf(-a.P.tr * th[1].x), __expf(-a.P.tr * th[1].y));
            float2 A0, A1, dA0, dA1;
            angle(0, E1, A0, dA0);
            angle(1, E1, A1, dA1);
            const float2 AM0 = mul2(A0, th[0]), AM1 = mul2(A1, th[0]);
            float2 sse = zero, Sq0 = zero, Sq1 = zero, St0 = zero, St1 = zero;
            each_echo<MAXT>(nte, [&](int t) {
                const float2 x = mul2(a.P.nl2e_pair[t], th[2]);
                const float2 E2 = make_float2(ex2_ftz(x.x), ex2_ftz(x.y));
                const float4 y = sy[t * T];
                const float2 r0 = fma2(AM0, E2, make_float2(y.x, y.y));
                sse = fma2(r0, r0, sse);
                const float2 q0 = mul2(r0, E2);
                Sq0 = add2(Sq0, q0);
                St0 = fma2(a.P.te_pair[t], q0, St0);
                const float2 r1 = fma2(AM1, E2, make_float2(y.z, y.w));
                sse = fma2(r1, r1, sse);
                const float2 q1 = mul2(r1, E2);
                Sq1 = add2(Sq1, q1);
                St1 = fma2(a.P.te_pair[t], q1, St1);
            });
            total = sse;
            g[0] = fma2(A1, Sq1, fma2(A0, Sq0, zero));
            g[1] = fma2(th[0], fma2(dA1, Sq1, fma2(dA0, Sq0, zero)), zero);
            g[2] = fma2(make_float2(-th[0].x, -th[0].y), fma2(A1, St1, fma2(A0, St0, zero)), zero);
        },
        [&](const float2 (&th)[3], auto&& write) {
            const float2 E1 = make_float2(__expf(-a.P.tr * th[1].x), __expf(-a.P.tr * th[1].y));
            float2 A0, A1, d;
            angle(0, E1, A0, d);
            angle(1, E1, A1, d);
            const float2 AM0 = mul2(A0, th[0]), AM1 = mul2(A1, th[0]);
            each_echo<MAXT>(nte, [&](int t) {
                const float2 x = mul2(a.P.nl2e_pair[t], th[2]);
                const float2 E2 = make_float2(ex2_ftz(x.x), ex2_ftz(x.y));
                const float4 y = sy[t * T];
                write(t, fma2(AM0, E2, make_float2(y.x, y.y)));
                write(t + nte, fma2(AM1, E2, make_float2(y.z, y.w)));
            });
        });
}

namespace {

FusedPairConsts pair_consts(const AdamParams& a) {
    auto pr = [](float x) { return make_float2(x, x); };
    FusedPairConsts k;
    k.nl2e = pr(-kLog2e);
    k.one = pr(1.0f);
    for (int i = 0; i < 3; ++i) {
        k.rng[i] = pr(a.P.ub[i] - a.P.lb[i]);
        k.lb[i] = pr(a.P.lb[i]);
    }
    k.b1 = pr(a.beta1);
    k.omb1 = pr(1.0f - a.beta1);
    k.b2 = pr(a.beta2);
    k.omb2 = pr(1.0f - a.beta2);
    k.eps = pr(a.eps);
    k.mse = pr(a.mse_scale);
    k.s2 = pr(2.0f * a.mse_scale);
    return k;
}

template <class K, class... Args>
cudaError_t launch_with(K kernel, int nblocks, int threads, size_t smem, cudaStream_t s, Args... args) {
    if (smem > 40 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kernel<<<nblocks, threads, smem, s>>>(args...);
    ++g_kernel_launches;
    return cudaGetLastError();
}

}  // namespace

// Which kernel takes a fused fit of `block` voxels a CTA.
//   R2*: pairs from kPairVoxels voxels on (2000 epochs: 40,000 voxels 1.16 ms in
//   pairs, 1.00 ms one a thread, whose chain is shorter; 80,000: 1.46, 1.51;
//   160,000: 2.19, 2.53).
//   R1-R2*: pairs.
// More than 512 voxels a CTA, blocks that are not whole 64-voxel chunks and the
// other configurations take the general kernel.
FusedKind fused_kind(const AdamParams& a, int model, int loss, int block) {
    if (loss != kMSE || a.transform != 0 || a.optimiser != kAdam || a.prior_mu) return kFusedGeneral;
    if (block > 512) return kFusedGeneral;  // threads x registers
    if (model == kR2S && a.nm <= kPairTE) {
        const bool pairs = a.nvtot >= kPairVoxels && block % 64 == 0;
        return pairs ? kFusedR2sPairs : kFusedR2s;
    }
    if (model == kR1R2S && a.P.n_fa == 2 && a.P.n_te <= kPairTE && block % 64 == 0) return kFusedR1r2sPairs;
    return kFusedGeneral;
}

cudaError_t launch_fused_std(FusedKind kind, const AdamParams& a, bool stats, int e_begin, int e_end, int update_last,
                             bool record, int block, int nblocks, cudaStream_t s) {
    const int rec = record ? 1 : 0;
    const int threads = kind == kFusedR2s ? block : block / 2;
    const size_t hist = sizeof(double) * (stats ? HistorySums<kHistW>::buf_doubles(threads / 32)
                                                : HistorySums<1>::buf_doubles(threads / 32));
    const FusedPairConsts k = pair_consts(a);
#define GX_ONE(M)                                                                                             \
    (stats ? launch_with(fused_r2s_kernel<M, true>, nblocks, threads, hist, s, a, e_begin, e_end, update_last, rec) \
           : launch_with(fused_r2s_kernel<M, false>, nblocks, threads, hist, s, a, e_begin, e_end, update_last, rec))
#define GX_TWO(K, M, SMEM)                                                                                    \
    (stats ? launch_with(K<M, true>, nblocks, threads, SMEM, s, a, k, e_begin, e_end, update_last, rec)        \
           : launch_with(K<M, false>, nblocks, threads, SMEM, s, a, k, e_begin, e_end, update_last, rec))
    if (kind == kFusedR2s) {
        if (a.nm <= 8) return GX_ONE(8);
        if (a.nm <= 12) return GX_ONE(12);
        return GX_ONE(16);
    }
    if (kind == kFusedR2sPairs) {
        if (a.nm <= 8) return GX_TWO(fused_r2s_pairs, 8, hist);
        if (a.nm <= 12) return GX_TWO(fused_r2s_pairs, 12, hist);
        return GX_TWO(fused_r2s_pairs, 16, hist);
    }
    const size_t smem = hist + sizeof(float4) * (size_t)a.P.n_te * threads;
    if (a.P.n_te <= 8) return GX_TWO(fused_r1r2s_pairs, 8, smem);
    if (a.P.n_te <= 12) return GX_TWO(fused_r1r2s_pairs, 12, smem);
    return GX_TWO(fused_r1r2s_pairs, 16, smem);
#undef GX_ONE
#undef GX_TWO
}

}  // namespace gx
