// dictionary.cu -- dictionary matching for likelihood starting points
// (gpuNEXI.likelihood, NEXI/gpuNEXI.m:813-836): for every voxel the first
// dictionary entry j minimising
//     sse_j = sum_m wt_m (S0_m - c_j S_jm)^2,   c_j = (S0 . S_j) / (S_j . S_j).
//
// Expanded per (voxel i, entry j):  sse = A_i - 2 c B_ij + c^2 C_j with
// D_ij = S0_i . S_j, B_ij = sum_m wt_m S0_im S_jm, A_i = sum_m wt_m S0_im^2,
// E_j = S_j . S_j, C_j = sum_m wt_m S_jm^2 and c = D_ij / E_j (unit weights:
// sse = A_i - D_ij^2 / E_j).  The expanded form is evaluated in FP64: for a good
// match sse / A is ~1e-3, so it loses about three digits to cancellation,
// which an FP32 decision cannot afford.
//
// Unit weights (dict_tensor_kernel): sse is least where |D| / |S_j| is largest,
// so the tensor cores compute every pair's d = (S0 / |S0|) . (S_j / |S_j|) with
// a bound on its error, and only the runs of 32 entries whose largest |d| lies
// within the bound of the voxel's best are scored in FP64 (1.5 of 313 runs at
// 10^4 NEXI entries), by the expression of the FP64 kernel: the same entry, the
// same score.
// Weighted, few entries or many measurements (dict_match_kernel): every pair in
// FP64, a register-tiled GEMM over dictionary tiles with a running argmin in
// the epilogue.
#include <cuda_bf16.h>

#include <algorithm>

#include "gx_internal.h"

namespace gx {

namespace {

constexpr int kTile = 64;   // voxels and entries per CTA tile
constexpr int kThreads = 256;
constexpr int kFewLeft = 4 * 148;  // voxels left by the tensor-core kernel that dict_scan_kernel takes

// Splitting of a value of magnitude at most 1 into three bf16 parts on fixed
// grids: x1 a multiple of 2^-7, x2 of 2^-15 (|x2| <= 2^-8), x3 the rest
// (|x3| <= 2^-16, rounded at 2^-25).
__device__ __forceinline__ void split3(double x, __nv_bfloat16 (&p)[3]) {
    const double x1 = rint(x * 128.0) * 0.0078125;
    const double r1 = x - x1;
    const double x2 = rint(r1 * 32768.0) * 3.0517578125e-05;
    p[0] = __double2bfloat16(x1);
    p[1] = __double2bfloat16(x2);
    p[2] = __double2bfloat16(r1 - x2);
}

// Operand tile of 128 rows (voxels or entries): chunks of 8 measurements, a
// chunk's 128 rows of 16 bytes together (the 8-row, 16-byte core matrices of
// the tensor core's K-major layout without swizzle: 128 bytes from one 8-row
// group to the next, 2048 bytes from one chunk to the next); the three parts'
// chunks after one another, measurements padded with zeros to a
// multiple of 8 (at least 16).
constexpr int kRows = 128;
constexpr int kChunkBytes = kRows * 16;
__host__ __device__ constexpr int chunks_of(int nm) { return nm <= 16 ? 2 : (nm + 7) / 8; }
__host__ __device__ constexpr size_t tile_bytes(int nm) { return (size_t)3 * chunks_of(nm) * kChunkBytes; }

// Row `row` of an operand tile: x(m) * scale split into its parts (zeros when !on).
template <class F>
__device__ __forceinline__ void write_operand(unsigned char* tile, int row, int nm, bool on, double scale, F&& x) {
    const int nc = chunks_of(nm);
    for (int c = 0; c < nc; ++c) {
        __align__(16) __nv_bfloat16 q[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            __nv_bfloat16 p[3];
            split3(on && c * 8 + e < nm ? x(c * 8 + e) * scale : 0.0, p);
#pragma unroll
            for (int b = 0; b < 3; ++b) q[b][e] = p[b];
        }
#pragma unroll
        for (int b = 0; b < 3; ++b)
            *reinterpret_cast<uint4*>(tile + (size_t)(b * nc + c) * kChunkBytes + row * 16) =
                *reinterpret_cast<const uint4*>(q[b]);
    }
}

// Per entry: 1 / (S_j . S_j) and sum_m wt_m S_jm^2 (double); with op, the
// entry's row of its operand tile (whole tiles: the rows past ndict are zero),
// and the first entry whose norm is a positive number (stat->first holds ndict
// minus it).
__global__ void dict_entry_kernel(const float* dict, int ndict, int nm, const float* wt, double* invE,
                                  double* C, unsigned char* op, DictStat* stat) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    double e = 0.0, c = 0.0;
    if (j < ndict) {
        for (int m = 0; m < nm; ++m) {
            double s = (double)dict[(size_t)m * ndict + j];
            e = fma(s, s, e);
            c = fma(wt ? (double)wt[m] * s : s, s, c);
        }
        invE[j] = 1.0 / e;   // E = 0: inf, and the pair scores NaN, which never wins
        C[j] = c;
    } else if (!op || j >= (ndict + kRows - 1) / kRows * kRows) {
        return;
    }
    if (!op) return;
    const bool on = j < ndict && e > 0.0 && isfinite(e);
    if (on) atomicMax(&stat->first, ndict - j);
    write_operand(op + (size_t)(j / kRows) * tile_bytes(nm), j % kRows, nm, on, on ? 1.0 / sqrt(e) : 0.0,
                  [&](int m) { return (double)dict[(size_t)m * ndict + j]; });
}

// Lexicographic (sse, j): smaller sse, then smaller j (MATLAB min's first index).
__device__ __forceinline__ bool better(double s1, int j1, double s0, int j0) {
    return s1 < s0 || (s1 == s0 && j1 < j0);
}

template <bool WEIGHTED>
__global__ void __launch_bounds__(kThreads)
dict_match_kernel(const float* signals, int nvox, const float* dict, int ndict, int nm, const float* wt,
                  const double* invE, const double* Cj, int* best, float* best_sse, const int* list,
                  const DictStat* stat) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sv = reinterpret_cast<double*>(smem_raw);      // [nm][64] voxel signals
    double* sd = sv + (size_t)nm * kTile;                  // [nm][64] dictionary tile
    double* sw = sd + (size_t)nm * kTile;                  // [nm][64] wt * voxel signals (weighted)
    __shared__ double s_A[kTile], s_ie[kTile], s_c[kTile];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    // list: the voxels that the tensor-core kernel left (count in stat)
    const int n = list ? min(stat->n_left, nvox) : nvox;
    if (list && n <= kFewLeft) return;  // dict_scan_kernel's
    // 64-bit: with a grid over all voxels the step passes 2^31 from 2^30 voxels on
    for (long long at = (long long)blockIdx.x * kTile; at < n; at += (long long)gridDim.x * kTile) {
    const int i0 = (int)at;
    __syncthreads();  // the previous voxels' tile is consumed
    for (int q = tid; q < nm * kTile; q += kThreads) {
        int m = q / kTile, v = q % kTile;
        double x = (i0 + v < n) ? (double)signals[(size_t)m * nvox + (list ? list[i0 + v] : i0 + v)] : 0.0;
        sv[q] = x;
        if (WEIGHTED) sw[q] = (double)wt[m] * x;
    }
    __syncthreads();
    if (tid < kTile) {
        double a = 0.0;
        for (int m = 0; m < nm; ++m) a = fma(WEIGHTED ? sw[m * kTile + tid] : sv[m * kTile + tid], sv[m * kTile + tid], a);
        s_A[tid] = a;
    }
    double bs[4];
    int bj[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) { bs[a] = INFINITY; bj[a] = 0x7fffffff; }

    for (int j0 = 0; j0 < ndict; j0 += kTile) {
        __syncthreads();  // the previous tile is consumed
        for (int q = tid; q < nm * kTile; q += kThreads) {
            int m = q / kTile, e = q % kTile;
            sd[q] = (j0 + e < ndict) ? (double)dict[(size_t)m * ndict + j0 + e] : 0.0;
        }
        if (tid < kTile) {
            bool ok = j0 + tid < ndict;
            s_ie[tid] = ok ? invE[j0 + tid] : 0.0;
            s_c[tid] = ok ? Cj[j0 + tid] : 0.0;
        }
        __syncthreads();
        double D[4][4], B[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) { D[a][b] = 0.0; B[a][b] = 0.0; }
        for (int m = 0; m < nm; ++m) {
            double x[4], y[4], xw[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                x[a] = sv[m * kTile + ty + 16 * a];
                if (WEIGHTED) xw[a] = sw[m * kTile + ty + 16 * a];
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) y[b] = sd[m * kTile + tx + 16 * b];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    D[a][b] = fma(x[a], y[b], D[a][b]);
                    if (WEIGHTED) B[a][b] = fma(xw[a], y[b], B[a][b]);
                }
        }
        // epilogue: entries in increasing j per thread, strict improvement
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int e = tx + 16 * b, j = j0 + e;
            if (j >= ndict) continue;
            const double ie = s_ie[e], cc = s_c[e];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double c = D[a][b] * ie;
                const double sse = WEIGHTED ? s_A[ty + 16 * a] - c * (2.0 * B[a][b] - c * cc)
                                            : s_A[ty + 16 * a] - c * D[a][b];
                if (sse < bs[a]) { bs[a] = sse; bj[a] = j; }
            }
        }
    }
    // fold the 16 threads that share each voxel (lanes with equal ty)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        double s = bs[a];
        int j = bj[a];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            double s2 = __shfl_xor_sync(0xffffffffu, s, o);
            int j2 = __shfl_xor_sync(0xffffffffu, j, o);
            if (better(s2, j2, s, j)) { s = s2; j = j2; }
        }
        const int il = i0 + ty + 16 * a;
        if (tx == 0 && il < n) {
            const int i = list ? list[il] : il;
            best[i] = j == 0x7fffffff ? -1 : j;
            if (best_sse) best_sse[i] = (float)s;
        }
    }
    }
}

// ---------------------------------------------------------------------------
// Tensor-core matching (unit weights).
//
// One CTA holds 128 voxels (rows of operand A, normalised by |S0|) and streams
// the dictionary's operand tiles (128 normalised entries) through two shared
// buffers by bulk copies.  Per tile, with the parts x = x1 + x2 + x3 of both
// operands, 8 products accumulate in two FP32 accumulators in tensor memory:
//   hi = x1 y1 + x1 y2 + x2 y1,
//   lo = x2 y2 + x1 y3 + x3 y1 + x2 y3 + x3 y2,   d = hi + lo.
// hi's products are multiples of 2^-22 and its partial sums stay below 2, so
// FP32 accumulates it without error; lo is below 2^-8, and its roundings
// together below 2^-24.  Left out are x3 y3 (nm 2^-32) and the parts' own
// roundings, at most sqrt(nm) 2^-25 for each operand; with the rounding of
// hi + lo, |d error| <= (sqrt(nm) + 4) 2^-24 <= (nm + 16) 2^-25 (1.2e-6 at
// nm = 24).  A product of the tensor core takes two chunks of 8 measurements; a
// schedule made on the host pairs them (the second chunk at any larger
// offset), so that 24 measurements take 13 products of 16, not 16.
// The 16 warps read the accumulators (a thread has one voxel and 32 columns),
// take the largest |d| of the 32 entries, and keep the runs of 32 within twice
// the bound of the largest so far.  At the end the runs within it of the
// voxel's best are scored in FP64, a warp to a run.  A voxel with more than kKeep
// such runs in one quarter of the columns (a dictionary of near-identical
// entries) is left to the FP64 kernels.
//
// Bound: latencies around the tensor pipe.  At nm = 24 a tile's 13 products take
// 806 clocks, the wait for them 350 more and the epilogue 800, the FP64 scores
// 60 k clocks of a block's 240 k; two CTAs share an SM so that one works under
// the other's waits.  500,000 voxels x 10^4 entries x 24 measurements: 14.6 ms
// (FP64 pipe 47 %, operands from shared memory) -> 2.4 ms; 20,000 x 2000:
// 0.11 ms; 1000 x 10^4: 0.17 ms; 200,000 x 10^4 x 64 (280 bytes spilled): 13.7
// -> 2.7 ms.  The products are unrolled with descriptors
// known at compile time: with descriptors loaded in a loop the issuing thread
// took 126 clocks a product, unrolled it takes the pipe's 62.
// ---------------------------------------------------------------------------
constexpr int kMaxTensorNm = 64;
constexpr int kKeep = 8;               // runs kept by a thread
constexpr int kRun = 32;
constexpr int kTensorThreads = 512;
constexpr int kParts = kTensorThreads / kRows;  // columns' quarters
constexpr int kMaxMma = 32;            // products of 16 measurements a tile, at most (8 chunks)

// Product of 16 measurements: first and second chunk of both operands.
struct MmaStep {
    int a, a2, b, b2;
};
struct MmaPlan {
    int n, n_hi;  // the first n_hi go to hi
    MmaStep s[kMaxMma];
};

// The chunk products of hi and lo in pairs, the second at larger chunk offsets
// in both operands: a product of parts (p, q) takes its chunks two by two; with
// an odd count it leaves out chunk `out`, and the chunks left out pair with one
// another (0 of x1 y1 with 1 of x1 y2, and so on), the one without a partner
// with the chunk of zeros behind operand A.
__host__ __device__ constexpr MmaPlan make_plan(int nc) {
    struct Term { int p, q, out, partner; };  // partner: the next term (1), the previous one (-1) or zeros (0)
    constexpr Term terms[2][5] = {{{0, 0, 0, 1}, {0, 1, 1, -1}, {1, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}},
                                  {{0, 2, 0, 1}, {1, 2, 1, -1}, {2, 0, 0, 1}, {2, 1, 1, -1}, {1, 1, 0, 0}}};
    MmaPlan plan{};
    for (int acc = 0; acc < 2; ++acc) {
        if (acc) plan.n_hi = plan.n;
        for (int i = 0; i < (acc ? 5 : 3); ++i) {
            const Term t = terms[acc][i];
            int held = -1;
            for (int k = 0; k < nc; ++k) {
                if (nc % 2 && k == t.out) continue;
                if (held < 0) held = k;
                else {
                    plan.s[plan.n++] = MmaStep{t.p * nc + held, t.p * nc + k, t.q * nc + held, t.q * nc + k};
                    held = -1;
                }
            }
            if (nc % 2 == 0 || t.partner < 0) continue;
            const int a = t.p * nc + t.out, b = t.q * nc + t.out;
            if (t.partner > 0) {
                const Term u = terms[acc][i + 1];
                plan.s[plan.n++] = MmaStep{a, u.p * nc + u.out, b, u.q * nc + u.out};
            } else {
                plan.s[plan.n++] = MmaStep{a, 3 * nc, b, b + 1};
            }
        }
    }
    return plan;
}

constexpr long long kWaitCycles = 4000000000LL;  // bound of every wait: about 2 s (DictWait may shorten it)

__device__ __forceinline__ unsigned int smem_addr(const void* p) { return (unsigned int)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool bar_wait(unsigned long long* bar, unsigned int parity, long long limit = kWaitCycles) {
    const long long t0 = clock64();
    do {
        unsigned int done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(smem_addr(bar)), "r"(parity) : "memory");
        if (done) return true;
    } while (clock64() - t0 < limit);
    return false;
}

// The same, ending early once another thread has raised err (looked at, with
// the clock, every 16 tries).
__device__ __forceinline__ bool bar_wait_or_err(unsigned long long* bar, unsigned int parity, volatile int* err,
                                                long long limit) {
    const long long t0 = clock64();
    do {
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            unsigned int done;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done) : "r"(smem_addr(bar)), "r"(parity) : "memory");
            if (done) return true;
        }
    } while (!*err && clock64() - t0 < limit);
    return false;
}

// Shared-memory matrix descriptors (K-major core matrices without swizzle, 128
// bytes between 8-row groups): the low word holds the address and the distance
// of the two chunks of K, in 16-byte units; an operand's low word at chunk 0
// and the chunks of a product, known at compile time, make it by one addition.
constexpr unsigned int kDescHigh = (128u >> 4) | (1u << 14);
__host__ __device__ constexpr unsigned int desc_low(int first, int second) {
    return (unsigned int)(first * (kChunkBytes >> 4)) + ((unsigned int)((second - first) * (kChunkBytes >> 4)) << 16);
}

// Instruction descriptor: D in FP32, A and B in bf16, both K-major, 128 x 128.
constexpr unsigned int kMmaDesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

template <bool ADD>
__device__ __forceinline__ void mma_bf16(unsigned int d, unsigned int a, unsigned int b) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                 "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
                 :: "r"(d), "r"(a), "r"(b), "n"(kDescHigh), "n"(kMmaDesc), "n"(ADD ? 1 : 0));
}

// All products of a tile, unrolled; a, b: the operands' low words.
template <int NC, int Q = 0>
__device__ __forceinline__ void mma_tile(unsigned int tmem, unsigned int a, unsigned int b) {
    constexpr MmaPlan plan = make_plan(NC);
    if constexpr (Q < plan.n) {
        constexpr MmaStep s = plan.s[Q];
        mma_bf16<(Q != 0 && Q != plan.n_hi)>(tmem + (Q < plan.n_hi ? 0u : 128u), a + desc_low(s.a, s.a2),
                                             b + desc_low(s.b, s.b2));
        mma_tile<NC, Q + 1>(tmem, a, b);
    }
}

// 16 columns of the calling warp's 32 lanes
__device__ __forceinline__ void tmem_load16(unsigned int addr, float (&r)[16]) {
    unsigned int u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(addr));
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(u[i]);
}

struct TensorSmem {
    unsigned long long full[2], done;   // operand tile arrived; products finished
    unsigned long long drain;           // after a wait that ran out: all products finished
    unsigned int tmem;
    int err;
    int scan[kRows];                    // end of each voxel's items
    double A[kRows];
    float best[kTensorThreads];
    unsigned char nkeep[kTensorThreads];  // runs kept; kKeep + 1: too many
    float val[kKeep][kTensorThreads];   // largest |d| of a kept run
    int run[kKeep][kTensorThreads];
};

// Dynamic shared memory: operand A, a chunk of zeros, two buffers of operand B;
// afterwards the items and their scores, and the voxels' measurements.
template <int NC>
__global__ void __launch_bounds__(kTensorThreads, 2)
dict_tensor_kernel(const float* signals, int nvox, const float* dict, int ndict, int nm, const double* invE,
                   const unsigned char* op, int* best, float* best_sse, int* list, DictStat* stat, DictWait wait) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TensorSmem S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr unsigned int tb = 3 * NC * kChunkBytes;
    unsigned char* opA = smem_raw;
    unsigned char* opB = smem_raw + tb + kChunkBytes;
    const int ntile = (ndict + kRows - 1) / kRows;
    const int i0 = blockIdx.x * kRows;
    const float slack = 2.0f * (float)(nm + 16) * 2.98023223876953125e-08f;
    if (tid == 0) {
        for (int b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" :: "r"(smem_addr(&S.full[b])) : "memory");
        asm volatile("mbarrier.init.shared.b64 [%0], %1;" :: "r"(smem_addr(&S.done)), "r"(1 + wait.extra) : "memory");
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" :: "r"(smem_addr(&S.drain)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    auto fetch = [&](int t) {  // operand tile t into buffer t & 1 (one thread)
        unsigned long long* bar = &S.full[t & 1];
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" :: "r"(smem_addr(bar)), "r"(tb) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(smem_addr(opB + (size_t)(t & 1) * tb)), "l"(op + (size_t)t * tb), "r"(tb), "r"(smem_addr(bar))
                     : "memory");
    };
    int fetched = 0;  // tiles requested (thread 0)
    if (tid == 0) {
        for (; fetched < min(2, ntile); ++fetched) fetch(fetched);
        S.err = *(volatile int*)&stat->err;  // an earlier CTA's wait ran out: the call has failed, no long waits here
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" :: "r"(smem_addr(&S.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid < kRows) {
        const int i = i0 + tid;
        double a = 0.0;
        if (i < nvox)
            for (int m = 0; m < nm; ++m) {
                const double x = (double)signals[(size_t)m * nvox + i];
                a = fma(x, x, a);
            }
        S.A[tid] = a;
        const bool on = i < nvox && a > 0.0 && isfinite(a);
        write_operand(opA, tid, nm, on, on ? 1.0 / sqrt(a) : 0.0,
                      [&](int m) { return (double)signals[(size_t)m * nvox + i]; });
        *reinterpret_cast<uint4*>(smem_raw + tb + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // operand A, for the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned int tmem = S.tmem;

    // this thread: voxel row (lane of the warp's quarter of the lanes), 32 columns
    const int part = warp >> 2;
    const unsigned int acc_addr = tmem + ((unsigned int)((warp & 3) * 32) << 16) + (unsigned int)(part * kRun);
    float top = 0.0f;
    int kept = 0;
    for (int t = 0; t < ntile; ++t) {
        if (tid == 0) {
            if (!bar_wait(&S.full[t & 1], (unsigned int)(t >> 1) & 1u, wait.limit)) S.err = 1;
            else {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                mma_tile<NC>(tmem, smem_addr(opA) >> 4, smem_addr(opB + (size_t)(t & 1) * tb) >> 4);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             :: "r"(smem_addr(&S.done)) : "memory");
            }
        }
        const bool ok = __all_sync(0xffffffffu, bar_wait_or_err(&S.done, (unsigned int)t & 1u, &S.err, wait.limit));
        if (!ok) S.err = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (ok) {
            if (tid == 0 && fetched < ntile) fetch(fetched++);  // the products of tile t have read its buffer
            __syncwarp();
            float m = 0.0f;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                float h[16], l[16];
                tmem_load16(acc_addr + 16u * g, h);
                tmem_load16(acc_addr + 128u + 16u * g, l);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < 16; e += 2) m = fmaxf(m, fmaxf(fabsf(h[e] + l[e]), fabsf(h[e + 1] + l[e + 1])));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (m >= top - slack) {
                top = fmaxf(top, m);
                if (kept == kKeep) {  // drop the runs that a later one has left behind
                    int n = 0;
                    for (int k = 0; k < kKeep; ++k)
                        if (S.val[k][tid] >= top - slack) {
                            S.val[n][tid] = S.val[k][tid];
                            S.run[n][tid] = S.run[k][tid];
                            ++n;
                        }
                    kept = n < kKeep ? n : kKeep + 1;
                }
                if (kept < kKeep) {
                    S.val[kept][tid] = m;
                    S.run[kept][tid] = t * (kRows / kRun) + part;
                    ++kept;
                }
            }
        }
        if (__syncthreads_or(!ok)) break;  // the accumulators are read; a wait that ran out ends the loop
    }
    S.best[tid] = top;
    S.nkeep[tid] = (unsigned char)kept;
    if (tid == 0 && S.err) {  // copies and products in flight, before the buffers and the tensor memory are let go
        for (int t = max(0, fetched - 2); t < fetched; ++t) bar_wait(&S.full[t & 1], (unsigned int)(t >> 1) & 1u);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                     :: "r"(smem_addr(&S.drain)) : "memory");
        bar_wait(&S.drain, 0u);
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" :: "r"(tmem));
    if (S.err) {
        if (tid == 0) stat->err = 1;
        return;
    }

    // items: the kept runs within the bound of the voxel's best, in a row per
    // voxel, and their scores; the voxels' measurements [voxel][nm] (odd stride)
    constexpr int kItems = kParts * kKeep * kRows;
    int* item = reinterpret_cast<int*>(smem_raw);
    int* entry = item + kItems;
    double* score = reinterpret_cast<double*>(entry + kItems);
    const double A = tid < kRows ? S.A[tid] : 0.0;
    const bool scored = tid < kRows && i0 + tid < nvox && A > 0.0 && isfinite(A);
    bool left = false;
    float floor_d = 0.0f;
    if (scored)
        for (int h = 0; h < kParts; ++h) {
            left |= S.nkeep[tid + h * kRows] > kKeep;
            floor_d = fmaxf(floor_d, S.best[tid + h * kRows]);
        }
    floor_d -= slack;
    auto each_run = [&](auto&& f) {
        if (scored && !left)
            for (int h = 0; h < kParts; ++h)
                for (int k = 0; k < S.nkeep[tid + h * kRows]; ++k)
                    if (S.val[k][tid + h * kRows] >= floor_d) f(S.run[k][tid + h * kRows]);
    };
    int mine = 0;
    each_run([&](int) { ++mine; });
    if (tid < kRows) S.scan[tid] = mine;
    __syncthreads();
    if (warp == 0) {  // running sums, 4 voxels a lane
        int c[4], n = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) { n += S.scan[lane * 4 + e]; c[e] = n; }
        int before = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += u;
        }
        before -= n;
#pragma unroll
        for (int e = 0; e < 4; ++e) S.scan[lane * 4 + e] = before + c[e];
    }
    __syncthreads();
    const int total = S.scan[kRows - 1];
    int at = tid < kRows ? S.scan[tid] - mine : 0;
    const int first = at;
    each_run([&](int r) { item[at++] = (tid << 24) | r; });
    __syncthreads();
    // an item's loads in flight together: one of the voxel's measurements a
    // lane, the entries' in registers
    for (int q = warp; q < total; q += kTensorThreads / 32) {
        const int v = (item[q] >> 24) & 0x7f, j = (item[q] & 0xffffff) * kRun + lane;
        const int jc = min(j, ndict - 1);
        const float* y = dict + jc;
        double D = 0.0;
        const double ie = invE[jc];
#pragma unroll
        for (int m0 = 0; m0 < NC * 8; m0 += 24) {
            const float xl = m0 + lane < nm && lane < 24 ? signals[(size_t)(m0 + lane) * nvox + i0 + v] : 0.0f;
            float ys[24];
#pragma unroll
            for (int e = 0; e < 24; ++e)
                if (m0 + e < NC * 8) ys[e] = y[(size_t)min(m0 + e, nm - 1) * ndict];
#pragma unroll
            for (int e = 0; e < 24; ++e)
                if (m0 + e < NC * 8) {
                    const double x = (double)__shfl_sync(0xffffffffu, xl, e);
                    if (m0 + e < nm) D = fma(x, (double)ys[e], D);
                }
        }
        double s = INFINITY;
        int js = 0x7fffffff;
        if (j < ndict) {
            const double c = D * ie;
            const double sse = S.A[v] - c * D;
            if (sse < s) { s = sse; js = j; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
            const int j2 = __shfl_xor_sync(0xffffffffu, js, o);
            if (better(s2, j2, s, js)) { s = s2; js = j2; }
        }
        if (lane == 0) { score[q] = s; entry[q] = js; }
    }
    __syncthreads();
    if (tid < kRows && i0 + tid < nvox) {
        if (left) {
            list[atomicAdd(&stat->n_left, 1)] = i0 + tid;
            return;
        }
        // a zero voxel scores 0 against every entry with a norm: the first of
        // them; a voxel that is not a number matches nothing
        double s = INFINITY;
        int js = 0x7fffffff;
        if (A == 0.0 && stat->first > 0) { s = 0.0; js = ndict - stat->first; }
        for (int q = first; q < first + mine; ++q)
            if (better(score[q], entry[q], s, js)) { s = score[q]; js = entry[q]; }
        best[i0 + tid] = js == 0x7fffffff ? -1 : js;
        if (best_sse) best_sse[i0 + tid] = (float)s;
    }
}

// The voxels left by dict_tensor_kernel when they are few: a CTA to a voxel,
// every entry in FP64 (dict_match_kernel would keep one CTA busy with 64 of
// them for as long as with a whole dictionary: 0.63 ms at 10^4 entries).
__global__ void __launch_bounds__(kThreads)
dict_scan_kernel(const float* signals, int nvox, const float* dict, int ndict, int nm, const double* invE, int* best,
                 float* best_sse, const int* list, const DictStat* stat) {
    __shared__ double s_x[kMaxTensorNm], s_s[kThreads / 32];
    __shared__ int s_j[kThreads / 32];
    const int n = stat->n_left, tid = threadIdx.x;
    if (n > kFewLeft) return;
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int i = list[q];
        __syncthreads();
        for (int m = tid; m < nm; m += kThreads) s_x[m] = (double)signals[(size_t)m * nvox + i];
        __syncthreads();
        double A = 0.0;
        for (int m = 0; m < nm; ++m) A = fma(s_x[m], s_x[m], A);
        double s = INFINITY;
        int js = 0x7fffffff;
        for (int j = tid; j < ndict; j += kThreads) {
            double D = 0.0;
#pragma unroll 8
            for (int m = 0; m < nm; ++m) D = fma(s_x[m], (double)dict[(size_t)m * ndict + j], D);
            const double c = D * invE[j];
            const double sse = A - c * D;
            if (sse < s) { s = sse; js = j; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
            const int j2 = __shfl_xor_sync(0xffffffffu, js, o);
            if (better(s2, j2, s, js)) { s = s2; js = j2; }
        }
        if ((tid & 31) == 0) { s_s[tid >> 5] = s; s_j[tid >> 5] = js; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kThreads / 32; ++w)
                if (better(s_s[w], s_j[w], s, js)) { s = s_s[w]; js = s_j[w]; }
            best[i] = js == 0x7fffffff ? -1 : js;
            if (best_sse) best_sse[i] = (float)s;
        }
    }
}

}  // namespace

size_t dict_match_smem(int nm, bool weighted) {
    return sizeof(double) * (size_t)nm * kTile * (weighted ? 3 : 2);
}

// The tensor-core kernel takes unit weights, up to 64 measurements (three
// operand tiles in shared memory) and dictionaries whose runs fit an item's 24
// bits, from the number of entries on at which it wins over dict_match_kernel:
// its launches, operand tiles and FP64 scores take 55-110 us whatever the
// dictionary, which the other kernel's time is proportional to.  us, FP64 kernel /
// tensor cores, 2000 voxels: 24 measurements, 600 entries 58 / 74, 1000: 79 /
// 82, 2000: 132 / 95, 10,000: 547 / 171; 64 measurements, 1000: 133 / 132,
// 2000: 235 / 146; 8 measurements, 1000: 53 / 70, 2000: 81 / 78, 5000: 169 /
// 105.  60,000 voxels: 24 measurements, 300 entries 93 / 132, 600: 155 / 143; 8
// measurements, 600: 87 / 110, 1000: 122 / 121; 48 measurements, 600: 253 / 269,
// 1000: 388 / 294.
// A dictionary so fine that most voxels overflow the kept runs (entries on a
// curve of one parameter in random order, or all alike) pays for both kernels:
// 200,000 voxels x 10,000 x 24, 6.1 / 6.9-7.2 ms, 2000 x 2000: 0.13 / 0.25; in
// order of the parameter 6.1 / 1.2 ms.
bool dict_tensor_ok(int nvox, int ndict, int nm, bool weighted) {
    const bool many = nvox >= 40000;
    const int least = nm < 16 ? (many ? 1024 : 1536) : (many && nm <= 32 ? 600 : 1024);
    return !weighted && nm <= kMaxTensorNm && ndict >= least && ndict / kRun < (1 << 24);
}

size_t dict_operand_bytes(int ndict, int nm) { return (size_t)((ndict + kRows - 1) / kRows) * tile_bytes(nm); }

cudaError_t launch_dictionary_match(const float* signals, int nvox, const float* dict, int ndict, int nm,
                                    const float* wt, double* invE, double* Cj, int* best, float* best_sse,
                                    unsigned char* op, int* list, DictStat* stat, DictWait wait, cudaStream_t s) {
    if (wait.limit <= 0) wait.limit = kWaitCycles;
    const bool tensor = op != nullptr;
    const int nentry = tensor ? (ndict + kRows - 1) / kRows * kRows : ndict;
    cudaError_t e = cudaSuccess;
    if (tensor) {
        e = cudaMemsetAsync(stat, 0, sizeof(DictStat), s);
        if (e != cudaSuccess) return e;
    }
    // few entries a block: the operand rows are written by as many SMs as can be
    dict_entry_kernel<<<(nentry + 63) / 64, 64, 0, s>>>(dict, ndict, nm, wt, invE, Cj, op, stat);
    ++g_kernel_launches;
    if (tensor) {
        // operands, or the items with their scores; two CTAs share an SM's tensor memory (256 of 512
        // columns each), and the threads of a third do not fit
        const size_t items = (size_t)kParts * kKeep * kRows * (2 * sizeof(int) + sizeof(double));
        const size_t smem = std::max(3 * tile_bytes(nm) + kChunkBytes, items);
        static decltype(&dict_tensor_kernel<2>) const kernels[] = {
            dict_tensor_kernel<2>, dict_tensor_kernel<3>, dict_tensor_kernel<4>, dict_tensor_kernel<5>,
            dict_tensor_kernel<6>, dict_tensor_kernel<7>, dict_tensor_kernel<8>};
        auto kt = kernels[chunks_of(nm) - 2];
        e = cudaFuncSetAttribute(kt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kt<<<(nvox - 1) / kRows + 1, kTensorThreads, smem, s>>>(signals, nvox, dict, ndict, nm, invE, op, best,
                                                                    best_sse, list, stat, wait);
        dict_scan_kernel<<<kFewLeft, kThreads, 0, s>>>(signals, nvox, dict, ndict, nm, invE, best, best_sse, list, stat);
        g_kernel_launches += 2;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const bool weighted = wt != nullptr;
    const size_t smem = dict_match_smem(nm, weighted);
    auto k = weighted ? dict_match_kernel<true> : dict_match_kernel<false>;
    // the kernel also holds static shared arrays, so opt in for every size
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // after the tensor-core kernel: the voxels it left (none as a rule)
    const int blocks = (nvox - 1) / kTile + 1;
    k<<<tensor ? std::min(blocks, 4 * 148) : blocks, kThreads, smem, s>>>(signals, nvox, dict, ndict, nm, wt, invE, Cj, best,
                                                          best_sse, tensor ? list : nullptr, stat);
    ++g_kernel_launches;
    return cudaGetLastError();
}

}  // namespace gx
