// cg_common.cuh -- device helpers shared by the CG kernels (kernels.cu: the
// memory-resident solve; cg_group.cu: the solve of blobs that fit on chip):
// warp sums, double-float sums, the 3x3 block product, the CG transition and
// the coarse space's row operators.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace ffea {
namespace {

constexpr unsigned int kSpinLimit = 1u << 24;  // ~1 s of 64 ns sleeps, then give up
constexpr int kMaxRestarts = 4;

template <typename A>
__device__ __forceinline__ A warp_sum(A v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// SELL-32 value index of component k (0..8 row-major 3x3) of entry `off`
__device__ __forceinline__ size_t sell_vidx(int off, int k)
{
    return (size_t)(off & ~31) * 9 + (size_t)k * 32 + (off & 31);
}

// Double-float accumulation (Knuth's TwoSum, error-free in FP32): sums with
// ~48-bit precision on the FP32 pipes, which on GB300 run many times faster
// than FP64.
struct DF {
    float hi, lo;
};

__device__ __forceinline__ DF df_add(DF a, DF b)
{
    const float s = a.hi + b.hi;
    const float bb = s - a.hi;
    float err = (a.hi - (s - bb)) + (b.hi - bb);
    err += a.lo + b.lo;
    const float hi = s + err;
    return DF{hi, err - (hi - s)};
}

// Vector of 4 T: the published copy of u in the CG kernel (x, y, z, 0), one
// 16-byte (FP32) load per neighbour instead of three 4-byte loads that each
// touch the same sectors.
struct alignas(16) Dbl4 {
    double x, y, z, w;
};

template <typename T> struct Vec4T;
template <> struct Vec4T<float> { using type = float4; };
template <> struct Vec4T<double> { using type = Dbl4; };

// One 3x3 block times a difference vector, added with explicit FMAs so that
// every code path gives the same bits.
template <typename T>
__device__ __forceinline__ void block_fma(const T K[9], T d0, T d1, T d2, T &a0, T &a1, T &a2)
{
    a0 = fma(K[2], d2, fma(K[1], d1, fma(K[0], d0, a0)));
    a1 = fma(K[5], d2, fma(K[4], d1, fma(K[3], d0, a1)));
    a2 = fma(K[8], d2, fma(K[7], d1, fma(K[6], d0, a2)));
}

__device__ __forceinline__ DF df_warp_sum(DF v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        DF w{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = df_add(v, w);
    }
    return v;
}

// Sum of N values per lane over a warp (N a power of two, 2..32) by a
// transposed butterfly: at offsets 16, 8, ... each lane keeps half of its
// values and adds its partner's copy of that half (N/2 + N/4 + ... shuffles),
// then the remaining offsets add whole values.  Returns this lane's total of
// value index idx; every lane holding the same idx holds the same bits, which
// are those of warp_sum (the same tree).
template <int N, typename A>
__device__ __forceinline__ A warp_sum_multi(A (&v)[N], int &idx)
{
    static_assert(N >= 2 && N <= 32 && (N & (N - 1)) == 0, "N must be a power of two in [2, 32]");
    const int lane = threadIdx.x & 31;
    idx = 0;
    int o = 16;
#pragma unroll
    for (int h = N / 2; h >= 1; h /= 2, o /= 2) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const A send = upper ? v[k] : v[k + h];
            const A keep = upper ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (upper) idx += h;
    }
    A x = v[0];
#pragma unroll
    for (; o > 0; o /= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// One CG transition of a blob from its three sums:
//   ACTIVE   sums r.u, w.u, r.r: stop test, then alpha / beta of the next update
//   VERIFY   sums r.u, -, |b - A x|^2: converged, or restart from that residual
//   RESTART  sums r.u, w.u, -: alpha of the first restarted update, beta = 0
// Returns true when the blob stops (cg.state is then CONVERGED or FAILED) and
// sets *fail_bits to the failure bits (0 if none).
//
// FP64 precision runs the recurrence in FP64: alpha = r.u / (w.u - beta r.u /
// alpha_prev), beta = r.u / r.u_prev, stop when r.r / f.f < eps^2.  Mixed
// precision (`fast`) applies alpha and beta in FP32 anyway and runs it in
// FP32 as alpha = r.u / p.Ap with p.Ap = w.u - beta^2 (p.Ap)_prev (the same
// recurrence), stop when r.r < eps^2 f.f: FP64 arithmetic and conversions run
// at 1/64 of the FP32 rate and would sit on the critical path of every
// iteration.  VERIFY (once per solve) stays in FP64.
__device__ __forceinline__ bool transition_core(CgScalars &cg, const BlobParams &bp, const DF sums[3],
                                                int *fail_bits, bool fast)
{
    const int limit = bp.solver == SOLVER_MASS ? bp.max_iter - 1 : bp.max_iter;
    int finish = 0, bits = 0;
    if (cg.state == CG_ACTIVE) {
        bool conv, nan, breakdown = false, at_floor = false;
        if (fast) {
            const float g = sums[0].hi + sums[0].lo, dl = sums[1].hi + sums[1].lo, rr = sums[2].hi + sums[2].lo;
            conv = rr < cg.stop_f;
            nan = !(rr == rr) || !(g == g) || !(dl == dl);
            if (!(cg.iters > 0 && conv) && !nan && cg.iters < limit) {
                const float beta = cg.iters == 0 ? 0.f : g / cg.gamma_f;
                const float pap = cg.iters == 0 ? dl : fmaf(-beta * beta, cg.pap_f, dl);
                if (!(pap > 0.f) || !(g > 0.f)) {
                    // the FP32 recurrence broke down (p.Ap or r.u not
                    // positive, so alpha would not be finite).  Below the
                    // floor this is the precision limit of FP32 vectors
                    // (an epsilon tighter than FP32 can reach): stop there;
                    // above it, it is a failure.
                    breakdown = true;
                    at_floor = rr < cg.floor_f;
                } else {
                    cg.beta_f = beta;
                    cg.pap_f = pap;
                    cg.alpha_f = g / pap;
                    cg.gamma_f = g;
                }
            }
        } else {
            const double g = (double)sums[0].hi + (double)sums[0].lo, dl = (double)sums[1].hi + (double)sums[1].lo;
            const double rr = (double)sums[2].hi + (double)sums[2].lo;
            cg.rr = rr;
            const double res = (cg.ff == 0.0) ? 0.0 : rr / cg.ff;
            conv = res < bp.epsilon2;
            nan = !(res == res) || !(g == g) || !(dl == dl);
            if (!(cg.iters > 0 && conv) && !nan && cg.iters < limit) {
                if (cg.iters == 0) {
                    cg.beta = 0.0;
                    cg.alpha = g / dl;
                } else {
                    const double beta = g / cg.gamma;
                    cg.alpha = g / (dl - beta * g / cg.alpha);
                    cg.beta = beta;
                }
                cg.gamma = g;
            }
        }
        if ((cg.iters > 0 && conv) || (breakdown && at_floor)) {
            // with the true-residual check on, the FP64 b - A x decides
            // (converged, or a restart from it)
            if (bp.true_residual) cg.state = CG_VERIFY;
            else finish = CG_CONVERGED;
        } else if (breakdown) {
            finish = CG_FAILED;
            bits = BLOB_FAIL_CG;
        } else if (nan) {
            finish = CG_FAILED;
            bits = BLOB_FAIL_CG | BLOB_FAIL_NAN;
        } else if (cg.iters >= limit) {
            finish = CG_FAILED;
            bits = BLOB_FAIL_CG;
        } else {
            cg.iters += 1;
        }
    } else if (cg.state == CG_VERIFY) {
        const double tr = (double)sums[2].hi + (double)sums[2].lo;
        cg.true_relres2 = (cg.ff == 0.0) ? 0.0 : tr / cg.ff;
        if (cg.true_relres2 < bp.epsilon2) {
            finish = CG_CONVERGED;
        } else if (cg.restarts >= kMaxRestarts || cg.iters >= limit) {
            finish = CG_FAILED;
            bits = BLOB_FAIL_CG;
        } else {
            cg.restarts += 1;
            cg.gamma = (double)sums[0].hi + (double)sums[0].lo;
            cg.gamma_f = sums[0].hi + sums[0].lo;
            cg.state = CG_RESTART;
        }
    } else if (cg.state == CG_RESTART) {
        // r.u of the restarted u (phase B of the restart step recomputes it,
        // with the coarse correction where there is one)
        cg.state = CG_ACTIVE;
        cg.iters += 1;
        bool nan;
        if (fast) {
            cg.gamma_f = sums[0].hi + sums[0].lo;
            cg.beta_f = 0.f;
            cg.pap_f = sums[1].hi + sums[1].lo;
            cg.alpha_f = cg.gamma_f / cg.pap_f;
            nan = !(cg.alpha_f == cg.alpha_f);
        } else {
            cg.gamma = (double)sums[0].hi + (double)sums[0].lo;
            cg.beta = 0.0;
            cg.alpha = cg.gamma / ((double)sums[1].hi + (double)sums[1].lo);
            nan = !(cg.alpha == cg.alpha);
        }
        if (nan) {
            finish = CG_FAILED;
            bits = BLOB_FAIL_CG | BLOB_FAIL_NAN;
        }
    }
    if (finish) cg.state = finish;
    *fail_bits = bits;
    return finish != 0;
}

// The coefficients of the next update in the arithmetic type of the vectors.
template <typename T>
__device__ __forceinline__ void cg_coefs(const CgScalars &cg, T &alpha, T &beta);

template <>
__device__ __forceinline__ void cg_coefs<float>(const CgScalars &cg, float &alpha, float &beta)
{
    alpha = cg.alpha_f;
    beta = cg.beta_f;
}

template <>
__device__ __forceinline__ void cg_coefs<double>(const CgScalars &cg, double &alpha, double &beta)
{
    alpha = cg.alpha;
    beta = cg.beta;
}

// The iteration's reduced sums (r.u, w.u, r.r) as the transition received
// them, kept per blob for inspection of the reduction's accuracy.
__device__ __forceinline__ void record_sums(const DeviceBatch &d, int b, const DF sums[3])
{
#pragma unroll
    for (int i = 0; i < 3; i++) d.last_sums[3 * (size_t)b + i] = (double)sums[i].hi + (double)sums[i].lo;
}

// Phi_p^T v = (v, d_p x v) into ex[0..5] for the rest offset f.xyz of row p
template <typename T>
__device__ __forceinline__ void restrict6_of(const float4 f, const T v[3], float *ex)
{
    const float v0 = (float)v[0], v1 = (float)v[1], v2 = (float)v[2];
    ex[0] = v0;
    ex[1] = v1;
    ex[2] = v2;
    ex[3] = f.y * v2 - f.z * v1;
    ex[4] = f.z * v0 - f.x * v2;
    ex[5] = f.x * v1 - f.y * v0;
}

// u = omega D^-1 r + Phi_p c for row p (f = rest offset and omega, c = its
// segment's coarse correction)
template <typename T>
__device__ __forceinline__ void coarse_u_of(const float4 f, const float *c, const T dinv[3], const T r[3], T u[3])
{
    const float cx = c[3], cy = c[4], cz = c[5];
    const T pc[3] = {(T)(c[0] + cy * f.z - cz * f.y), (T)(c[1] + cz * f.x - cx * f.z), (T)(c[2] + cx * f.y - cy * f.x)};
#pragma unroll
    for (int k = 0; k < 3; k++) u[k] = (T)f.w * dinv[k] * r[k] + pc[k];
}

}  // namespace
}  // namespace ffea
