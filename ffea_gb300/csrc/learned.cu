// learned.cu -- the learned part of the two-level preconditioner: a mesh
// message-passing network that sets the per-node weight omega_p of the
// Jacobi term of M = diag(omega) D^-1 + P A_c^-1 P^T, its training gradient,
// and the loss it is trained on.
//
// Network (FP32 weights, BF16 stored activations, FP32 accumulation):
//   h0_p = features of row p (8, see k_features)
//   h(l+1)_p = ReLU(Ws_l h(l)_p + Wn_l mean_{q ~ p} h(l)_q + b_l),  l = 0, 1, 2,
//              hidden width 32, q ~ p the rows sharing a mesh edge with p
//   omega_p = 2 sigmoid(wo . h3_p + bo)  in (0, 2)
// Loss of one (rhs f, solution x) pair of the NoMass solve, on the matrix A
// and coarse inverse X of that solve: the A-norm error of the best multiple
// of one preconditioner application z = M f (one preconditioned steepest-
// descent step), relative to |x|_A:
//   L = min_tau |x - tau z|_A^2 / |x|_A^2 = 1 - (f.z)^2 / ((z.Az)(x.f)),
// invariant to the scale of M, as CG is (x.f = x.Ax).  With a = f.z,
// b = z.Az, c = x.f: dL/dz = (2a/(bc)) ((a/b) Az - f), and z_p depends on
// omega_p through omega_p (D^-1 f)_p, so dL/d omega_p = k1 (Az.v)_p - k2
// (f.v)_p with v = D^-1 f, k1 = 2a^2/(b^2 c), k2 = 2a/(bc); then the network
// backward.
// Every sum over rows is a fixed-order reduction (per-CTA partials, then a
// CTA-ordered sum): results do not depend on scheduling.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <vector>

#include "kernels.h"

namespace ffea {

namespace {

constexpr int kHid = MPNN_HIDDEN, kFin = MPNN_FEATURES;
constexpr int kRowThreads = 128;   // rows per CTA of the kernels with a thread per row
constexpr int kFwdRows = 32;       // rows per CTA of a forward layer: four threads gather a row
constexpr int kBwdRows = 64;       // rows per CTA of a backward layer, four threads a row
constexpr int kNbrBatch = 8;       // neighbours whose loads are in flight together
static_assert(kBwdRows == MPNN_BWD_ROWS && kRowThreads == MPNN_LOSS_ROWS, "sizes of the partial sums");

struct MpnnLayout {
    int ws[3], wn[3], b[3], wo, bo, total;
};

__host__ __device__ constexpr MpnnLayout mpnn_layout()
{
    MpnnLayout L{};
    int off = 0;
    for (int l = 0; l < 3; l++) {
        const int din = l == 0 ? kFin : kHid;
        L.ws[l] = off;
        off += kHid * din;
        L.wn[l] = off;
        off += kHid * din;
        L.b[l] = off;
        off += kHid;
    }
    L.wo = off;
    off += kHid;
    L.bo = off;
    off += 1;
    L.total = off;
    return L;
}
static_assert(mpnn_layout().total == MPNN_NUM_PARAMS, "parameter count");

__device__ __forceinline__ bool free_nomass_row(const DeviceBatch &d, int row, int &blob)
{
    if (row >= d.nl_pad) return false;
    blob = d.seg_of_row[row] >= 0 ? d.seg_blob[d.seg_of_row[row]] : -1;
    if (blob < 0) return false;
    const BlobParams &bp = d.bp[blob];
    return bp.solver == SOLVER_NOMASS && !(d.flags[row] & NODE_PINNED);
}

template <typename T>
__device__ __forceinline__ void load_K(const DeviceBatch &d, int base, int j, int lane, float K[9])
{
    const T *val = static_cast<const T *>(d.sell_val);
    const size_t vb = (size_t)(base + 32 * j) * 9 + lane;
#pragma unroll
    for (int k = 0; k < 9; k++) K[k] = (float)val[vb + 32 * k];
}

// Eight scale-free features of row p from the current matrix and the coarse
// layout: drag / stiffness, neighbours in other segments, distance from the
// segment centroid, degree, off-diagonal weight, pinned neighbours,
// anisotropy of the diagonal block, and a constant.
template <typename T>
__global__ void __launch_bounds__(kRowThreads) k_features(DeviceBatch d, float *x0)
{
    const int row = blockIdx.x * kRowThreads + threadIdx.x;
    if (row >= d.nl_pad) return;
    float f[kFin] = {0, 0, 0, 0, 0, 0, 0, 0};
    int b;
    if (free_nomass_row(d, row, b)) {
        const BlobParams &bp = d.bp[b];
        const int sl = row >> 5, lane = row & 31;
        const int L = d.slice_len[sl], base = d.slice_ptr[sl];
        const int seg = d.seg_of_row[row];
        float S[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, off = 0.f;
        int deg = 0, other = 0, pinned = 0;
        for (int j0 = 0; j0 < L; j0 += kNbrBatch) {
            int q[kNbrBatch], sg[kNbrBatch];
            float K[kNbrBatch][9];
            uint32_t fl[kNbrBatch];
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                q[u] = row;
                if (j0 + u < L) {
                    q[u] = d.sell_col[base + 32 * (j0 + u) + lane];
                    load_K<T>(d, base, j0 + u, lane, K[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                sg[u] = d.seg_of_row[q[u]];
                fl[u] = d.flags[q[u]];
            }
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                if (q[u] == row) continue;
                float n2 = 0.f;
#pragma unroll
                for (int m = 0; m < 9; m++) {
                    S[m] -= K[u][m];
                    n2 += K[u][m] * K[u][m];
                }
                off += sqrtf(n2);
                deg++;
                other += sg[u] != seg;
                pinned += (fl[u] & NODE_PINNED) != 0;
            }
        }
        const float z = bp.calc_stokes == 1 ? (float)d.drag[row] : 0.f;
        S[0] += z;
        S[4] += z;
        S[8] += z;
        const float tr = fmaxf((S[0] + S[4] + S[8]) / 3.f, 1e-30f);
        const float4 ph = d.phi[row];
        const float od = sqrtf(S[1] * S[1] + S[2] * S[2] + S[3] * S[3] + S[5] * S[5] + S[6] * S[6] + S[7] * S[7]);
        const float inv = deg > 0 ? 1.f / deg : 0.f;
        f[0] = z / tr;
        f[1] = other * inv;
        f[2] = sqrtf(ph.x * ph.x + ph.y * ph.y + ph.z * ph.z);
        f[3] = deg / 16.f;
        f[4] = off / (3.f * tr);
        f[5] = pinned * inv;
        f[6] = od / tr;
        f[7] = 1.f;
    }
    float4 *o = reinterpret_cast<float4 *>(x0) + 2 * (size_t)row;
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
}

// Channels of a row's activations that one of its four threads holds: 8 BF16
// of the hidden width (one 16-byte load), 2 floats of the features (8 bytes)
template <int DIN>
struct Part;
template <>
struct Part<kHid> {
    using Act = __nv_bfloat16;
    uint4 raw;
    __device__ __forceinline__ void load(const Act *h, int row, int part)
    {
        raw = reinterpret_cast<const uint4 *>(h)[(size_t)row * 4 + part];
    }
    __device__ __forceinline__ void get(float (&f)[kHid / 4]) const
    {
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            f[2 * k] = __uint_as_float(w[k] << 16);
            f[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
        }
    }
};
template <>
struct Part<kFin> {
    using Act = float;
    float2 raw;
    __device__ __forceinline__ void load(const Act *h, int row, int part)
    {
        raw = reinterpret_cast<const float2 *>(h)[(size_t)row * 4 + part];
    }
    __device__ __forceinline__ void get(float (&f)[kFin / 4]) const
    {
        f[0] = raw.x;
        f[1] = raw.y;
    }
};

// columns j0 .. j0 + kNbrBatch - 1 of a row, the row itself past its end
__device__ __forceinline__ void batch_columns(const DeviceBatch &d, int row, int L, int base, int j0,
                                              int (&q)[kNbrBatch])
{
#pragma unroll
    for (int u = 0; u < kNbrBatch; u++) q[u] = j0 + u < L ? d.sell_col[base + 32 * (j0 + u) + (row & 31)] : row;
}

// One message-passing layer: out = bf16(ReLU(Ws h + Wn mean(h_nbr) + b)).
// Bound by the latency of the gather, not by its bytes (a row's neighbours,
// 64 bytes each, come from L2): one thread per row left an SM four warps and
// read a neighbour as sixteen 4-byte loads, one neighbour after another (28
// us a layer for 8.7 k rows).  Here a CTA takes the 32 rows of a SELL slice;
// four threads a row read 16 bytes of each neighbour, eight neighbours in
// flight, and sum them in slot order; then each warp computes 8 of the 32
// outputs of the 32 rows, its weights one broadcast read for all lanes.
// LAST adds the output layer: omega = 2 sigmoid(wo . h3 + bo) from the
// rounded activations, written to the smoother weight of free NoMass rows
// (other rows keep weight 1).
template <int DIN, bool LAST>
__global__ void __launch_bounds__(4 * kFwdRows) k_layer(DeviceBatch d, const float *theta, int ws, int wn, int bo,
                                                        const typename Part<DIN>::Act *hin, __nv_bfloat16 *hout,
                                                        float *omega, int write_phi)
{
    constexpr int C = DIN / 4, O = kHid / 4;
    __shared__ __align__(16) float sWs[kHid * DIN], sWn[kHid * DIN];
    __shared__ float sb[kHid], sh[kFwdRows][DIN + 1], sm[kFwdRows][DIN + 1];
    __shared__ float so[LAST ? kFwdRows : 1][kHid + 1];
    const int t = threadIdx.x;
    for (int k = t; k < kHid * DIN; k += 4 * kFwdRows) {
        sWs[k] = theta[ws + k];
        sWn[k] = theta[wn + k];
    }
    if (t < kHid) sb[t] = theta[bo + t];
    {
        const int r = t >> 2, part = t & 3, row = blockIdx.x * kFwdRows + r;
        const int L = d.slice_len[blockIdx.x], base = d.slice_ptr[blockIdx.x];
        Part<DIN> own;
        own.load(hin, row, part);
        float m[C], v[C];
        int deg = 0;
#pragma unroll
        for (int k = 0; k < C; k++) m[k] = 0.f;
        for (int j0 = 0; j0 < L; j0 += kNbrBatch) {
            int q[kNbrBatch];
            Part<DIN> nb[kNbrBatch];
            batch_columns(d, row, L, base, j0, q);
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) nb[u].load(hin, q[u], part);
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                if (q[u] == row) continue;
                nb[u].get(v);
#pragma unroll
                for (int k = 0; k < C; k++) m[k] += v[k];
                deg++;
            }
        }
        const float inv = deg > 0 ? 1.f / deg : 0.f;
        own.get(v);
#pragma unroll
        for (int k = 0; k < C; k++) {
            sh[r][C * part + k] = v[k];
            sm[r][C * part + k] = m[k] * inv;
        }
    }
    __syncthreads();
    const int r = t & 31, i0 = O * (t >> 5), row = blockIdx.x * kFwdRows + r;
    float a[O];
#pragma unroll
    for (int i = 0; i < O; i++) a[i] = sb[i0 + i];
#pragma unroll
    for (int k = 0; k < DIN; k += 4) {
        float h[4], m[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            h[c] = sh[r][k + c];
            m[c] = sm[r][k + c];
        }
#pragma unroll
        for (int i = 0; i < O; i++) {
            const float4 w = *reinterpret_cast<const float4 *>(&sWs[(i0 + i) * DIN + k]);
            const float4 n = *reinterpret_cast<const float4 *>(&sWn[(i0 + i) * DIN + k]);
            a[i] = fmaf(w.x, h[0], fmaf(n.x, m[0], a[i]));
            a[i] = fmaf(w.y, h[1], fmaf(n.y, m[1], a[i]));
            a[i] = fmaf(w.z, h[2], fmaf(n.z, m[2], a[i]));
            a[i] = fmaf(w.w, h[3], fmaf(n.w, m[3], a[i]));
        }
    }
    alignas(16) __nv_bfloat162 o[O / 2];  // (stored as one 16-byte word)
#pragma unroll
    for (int i = 0; i < O; i += 2) o[i / 2] = __floats2bfloat162_rn(fmaxf(a[i], 0.f), fmaxf(a[i + 1], 0.f));
    reinterpret_cast<uint4 *>(hout)[(size_t)row * 4 + (t >> 5)] = *reinterpret_cast<const uint4 *>(o);
    if constexpr (LAST) {
#pragma unroll
        for (int i = 0; i < O; i += 2) {
            const float2 v = __bfloat1622float2(o[i / 2]);
            so[r][i0 + i] = v.x;
            so[r][i0 + i + 1] = v.y;
        }
        __syncthreads();
        if (t >= kFwdRows) return;
        constexpr MpnnLayout P = mpnn_layout();
        int b;
        float w = 1.f;
        if (free_nomass_row(d, row, b)) {
            float s = theta[P.bo];
#pragma unroll
            for (int i = 0; i < kHid; i++) s = fmaf(theta[P.wo + i], so[r][i], s);
            w = 2.f / (1.f + expf(-s));
            if (write_phi) d.phi[row].w = w;
        }
        omega[row] = w;
    }
}

// ---------------------------------------------------------------- loss
// P^T f per segment (one CTA of CG_SEG_MAX_ROWS threads per segment) and
// v = D^-1 f per row
template <typename T>
__global__ void __launch_bounds__(CG_SEG_MAX_ROWS) k_loss_restrict(DeviceBatch d, float4 *v, float *gvec)
{
    __shared__ float red[6][32];
    const int s = blockIdx.x, t = threadIdx.x;
    const int b = d.seg_blob[s];
    const BlobParams &bp = d.bp[b];
    const int row = d.seg_row0[s] + t;
    float ex[6] = {0, 0, 0, 0, 0, 0};
    if (t < d.seg_rows[s]) {
        float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!(d.flags[row] & NODE_PINNED) && bp.solver == SOLVER_NOMASS) {
            const float f0 = (float)d.rhs[3 * (size_t)row], f1 = (float)d.rhs[3 * (size_t)row + 1],
                        f2 = (float)d.rhs[3 * (size_t)row + 2];
            const T *di = static_cast<const T *>(d.dinv) + 3 * (size_t)row;
            vv = make_float4((float)di[0] * f0, (float)di[1] * f1, (float)di[2] * f2, 0.f);
            const float4 ph = d.phi[row];
            ex[0] = f0;
            ex[1] = f1;
            ex[2] = f2;
            ex[3] = ph.y * f2 - ph.z * f1;
            ex[4] = ph.z * f0 - ph.x * f2;
            ex[5] = ph.x * f1 - ph.y * f0;
        }
        v[row] = vv;
    }
    const int lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int l = 0; l < 6; l++) {
        float x = ex[l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[l][warp] = x;
    }
    __syncthreads();
    if (t < 6) {
        float x = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) x += red[t][w];
        gvec[bp.coarse_off + 6 * (s - bp.seg_off) + t] = x;
    }
}

// c = X g for the six coarse rows of a segment (a warp each), then
// z = M f = omega v + Phi_p c for its rows.  A thread per coarse row of a
// blob left 7 CTAs to read X, 85 us for the 2.3 MB of a 15 nm sphere.
constexpr int kApplyThreads = 256;
__global__ void __launch_bounds__(kApplyThreads) k_loss_apply(DeviceBatch d, const float *gvec, const float4 *v,
                                                              const float *omega, float4 *z)
{
    __shared__ float c[6];
    const int s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const BlobParams &bp = d.bp[d.seg_blob[s]];
    const bool nomass = bp.solver == SOLVER_NOMASS;
    if (nomass && warp < 6) {
        const int n = bp.coarse_n;
        const float *X = d.coarse_X + bp.coarse_xoff + (size_t)(6 * (s - bp.seg_off) + warp) * n;
        const float *g = gvec + bp.coarse_off;
        float a = 0.f;
#pragma unroll 8
        for (int j = lane; j < n; j += 32) a = fmaf(X[j], g[j], a);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) c[warp] = a;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < d.seg_rows[s]; t += kApplyThreads) {
        const int row = d.seg_row0[s] + t;
        float4 zv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (nomass && !(d.flags[row] & NODE_PINNED)) {
            const float4 ph = d.phi[row], vv = v[row];
            const float w = omega[row];
            zv.x = w * vv.x + c[0] + c[4] * ph.z - c[5] * ph.y;
            zv.y = w * vv.y + c[1] + c[5] * ph.x - c[3] * ph.z;
            zv.z = w * vv.z + c[2] + c[3] * ph.y - c[4] * ph.x;
        }
        z[row] = zv;
    }
}

// A z per row (difference form); per row (Az.v, f.v) for the omega
// gradient; per CTA the sums f.z, z.Az, x.f
template <typename T>
__global__ void __launch_bounds__(kRowThreads) k_loss_products(DeviceBatch d, const float4 *z, const float4 *v,
                                                               float2 *gw, double *cta_sums)
{
    __shared__ double red[3][kRowThreads / 32];
    const int row = blockIdx.x * kRowThreads + threadIdx.x;
    double fz = 0.0, zaz = 0.0, xf = 0.0;
    int b;
    if (free_nomass_row(d, row, b)) {
        const BlobParams &bp = d.bp[b];
        const int sl = row >> 5, lane = row & 31;
        const int L = d.slice_len[sl], base = d.slice_ptr[sl];
        const float4 zp = z[row];
        const float zeta = bp.calc_stokes == 1 ? (float)d.drag[row] : 0.f;
        float a0 = zeta * zp.x, a1 = zeta * zp.y, a2 = zeta * zp.z;
        for (int j0 = 0; j0 < L; j0 += kNbrBatch) {
            int q[kNbrBatch];
            float K[kNbrBatch][9];
            float4 zq[kNbrBatch];
            batch_columns(d, row, L, base, j0, q);
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                if (j0 + u < L) load_K<T>(d, base, j0 + u, lane, K[u]);
                zq[u] = z[q[u]];
            }
#pragma unroll
            for (int u = 0; u < kNbrBatch; u++) {
                if (q[u] == row) continue;
                const float d0 = zq[u].x - zp.x, d1 = zq[u].y - zp.y, d2 = zq[u].z - zp.z;
                a0 += K[u][0] * d0 + K[u][1] * d1 + K[u][2] * d2;
                a1 += K[u][3] * d0 + K[u][4] * d1 + K[u][5] * d2;
                a2 += K[u][6] * d0 + K[u][7] * d1 + K[u][8] * d2;
            }
        }
        const float4 vv = v[row];
        const double f0 = d.rhs[3 * (size_t)row], f1 = d.rhs[3 * (size_t)row + 1], f2 = d.rhs[3 * (size_t)row + 2];
        gw[row] = make_float2(a0 * vv.x + a1 * vv.y + a2 * vv.z, (float)(f0 * vv.x + f1 * vv.y + f2 * vv.z));
        fz = f0 * zp.x + f1 * zp.y + f2 * zp.z;
        zaz = (double)zp.x * a0 + (double)zp.y * a1 + (double)zp.z * a2;
        const T *x = static_cast<const T *>(d.x) + 3 * (size_t)row;
        xf = (double)x[0] * f0 + (double)x[1] * f1 + (double)x[2] * f2;
    } else if (row < d.nl_pad) {
        gw[row] = make_float2(0.f, 0.f);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
        zaz += __shfl_xor_sync(0xffffffffu, zaz, o);
        xf += __shfl_xor_sync(0xffffffffu, xf, o);
    }
    if (lane == 0) {
        red[0][warp] = fz;
        red[1][warp] = zaz;
        red[2][warp] = xf;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double s = 0.0;
        for (int w = 0; w < kRowThreads / 32; w++) s += red[threadIdx.x][w];
        cta_sums[3 * blockIdx.x + threadIdx.x] = s;
    }
}

// a = f.z, b = z.Az, c = x.f: a warp each over the CTAs' sums, in a fixed
// order; scal = (loss, k1, k2) with loss = 1 - a^2/(bc), k1 = 2a^2/(b^2 c),
// k2 = 2a/(bc)
__global__ void __launch_bounds__(96) k_loss_total(const double *cta_sums, int n, double *scal)
{
    __shared__ double sums[3];
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += cta_sums[3 * i + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sums[k] = s;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double a = sums[0], b = sums[1], c = sums[2];
    const bool ok = b > 0.0 && c > 0.0;
    scal[0] = ok ? 1.0 - a * a / (b * c) : 0.0;
    scal[1] = ok ? 2.0 * a * a / (b * b * c) : 0.0;
    scal[2] = ok ? 2.0 * a / (b * c) : 0.0;
}

// ---------------------------------------------------------------- backward
// Backward of one layer, 64 rows to a CTA.  dh_out, the gradient of the
// layer's output:
//   TOP: dL/d omega = k1 gw.x - k2 gw.y, dL/ds = dL/d omega * omega (1 -
//        omega / 2), dh_out = dL/ds wo, and the partials of dwo and dbo;
//   else the adjoint of the layer above: its self part plus the sum over the
//        neighbours p of t[p] (the edge graph is symmetric).
// da = dh_out * (h_out > 0).  Partials of dWs, dWn and db per CTA, at
// partial[cta * MPNN_NUM_PARAMS + ...]; unless the layer is the first, the
// self part of dh_in (Ws^T da) and t = Wn^T da / deg for the layer below.
// Latency-bound like the forward layers: with a thread per row and 64
// threads a CTA an SM had three warps, each walking its row's neighbours one
// at a time in 4-byte loads and reading the weights from global memory, with
// the gather in a kernel of its own (61 + 37 us a layer for 8.7 k rows).
// Four threads a row gather t and h together, eight neighbours in flight;
// the products run from shared memory: Ws^T da and Wn^T da on tiles of 8
// channels with broadcast weights, the outer products on DIN/8 x 2 tiles.
template <int DIN, bool TOP>
__global__ void __launch_bounds__(4 * kBwdRows) k_layer_bwd(DeviceBatch d, const float *theta, int ws, int wn, int bo,
                                                            const typename Part<DIN>::Act *hin,
                                                            const __nv_bfloat16 *hout, const float *omega,
                                                            const float2 *gw, const double *scal,
                                                            const float *self_above, const float *t_above,
                                                            float *dh_in_self, float *tbuf, float *partial)
{
    constexpr MpnnLayout P = mpnn_layout();
    constexpr int T = 4 * kBwdRows, C = DIN / 4, O = kHid / 4, W = 2 * DIN;
    constexpr bool FIRST = DIN == kFin;
    __shared__ __align__(16) float sda[kBwdRows][kHid + 4], shm[kBwdRows][W + 4];
    __shared__ __align__(16) float sWs[FIRST ? 4 : kHid * DIN], sWn[FIRST ? 4 : kHid * DIN];
    __shared__ float sds[kBwdRows], sinv[kBwdRows];
    const int t = threadIdx.x, row0 = blockIdx.x * kBwdRows;
    if (!FIRST)
        for (int k = t; k < kHid * DIN; k += T) {
            sWs[k] = theta[ws + k];
            sWn[k] = theta[wn + k];
        }
    {
        const int r = t >> 2, part = t & 3, row = row0 + r;
        float dh[O], m[C], v[C], inv = 0.f;
#pragma unroll
        for (int i = 0; i < O; i++) dh[i] = 0.f;
#pragma unroll
        for (int k = 0; k < C; k++) m[k] = v[k] = 0.f;
        if (row < d.nl_pad) {
            const int L = d.slice_len[row >> 5], base = d.slice_ptr[row >> 5];
            Part<DIN> own;
            Part<kHid> ho;
            own.load(hin, row, part);
            ho.load(hout, row, part);
            if (TOP) {
                const float w = omega[row];
                const float2 g = gw[row];
                const float ds = ((float)scal[1] * g.x - (float)scal[2] * g.y) * w * (1.f - 0.5f * w);
                if (part == 0) sds[r] = ds;
#pragma unroll
                for (int i = 0; i < O; i++) dh[i] = ds * theta[P.wo + O * part + i];
            } else {
                const float4 *p = reinterpret_cast<const float4 *>(self_above) + (size_t)row * (kHid / 4) + 2 * part;
                const float4 x = p[0], y = p[1];
                dh[0] = x.x, dh[1] = x.y, dh[2] = x.z, dh[3] = x.w;
                dh[4] = y.x, dh[5] = y.y, dh[6] = y.z, dh[7] = y.w;
            }
            int deg = 0;
            for (int j0 = 0; j0 < L; j0 += kNbrBatch) {
                int q[kNbrBatch];
                Part<DIN> nb[kNbrBatch];
                float4 x[TOP ? 1 : kNbrBatch], y[TOP ? 1 : kNbrBatch];
                batch_columns(d, row, L, base, j0, q);
#pragma unroll
                for (int u = 0; u < kNbrBatch; u++) {
                    nb[u].load(hin, q[u], part);
                    if (!TOP) {
                        const float4 *p =
                            reinterpret_cast<const float4 *>(t_above) + (size_t)q[u] * (kHid / 4) + 2 * part;
                        x[u] = p[0];
                        y[u] = p[1];
                    }
                }
#pragma unroll
                for (int u = 0; u < kNbrBatch; u++) {
                    if (q[u] == row) continue;
                    nb[u].get(v);
#pragma unroll
                    for (int k = 0; k < C; k++) m[k] += v[k];
                    if (!TOP) {
                        dh[0] += x[u].x, dh[1] += x[u].y, dh[2] += x[u].z, dh[3] += x[u].w;
                        dh[4] += y[u].x, dh[5] += y[u].y, dh[6] += y[u].z, dh[7] += y[u].w;
                    }
                    deg++;
                }
            }
            inv = deg > 0 ? 1.f / deg : 0.f;
            float o[O];
            ho.get(o);
#pragma unroll
            for (int i = 0; i < O; i++) dh[i] = o[i] > 0.f ? dh[i] : 0.f;
            own.get(v);
        } else if (TOP && part == 0) {
            sds[r] = 0.f;
        }
        if (part == 0) sinv[r] = inv;
#pragma unroll
        for (int i = 0; i < O; i++) sda[r][O * part + i] = dh[i];
#pragma unroll
        for (int k = 0; k < C; k++) {
            shm[r][C * part + k] = v[k];
            shm[r][DIN + C * part + k] = m[k] * inv;
        }
    }
    __syncthreads();
    const int warp = t >> 5, lane = t & 31;
    if (!FIRST) {
        const int r = 32 * (warp & 1) + lane, k0 = O * (warp >> 1), row = row0 + r;
        float a[O], n[O];
#pragma unroll
        for (int k = 0; k < O; k++) a[k] = n[k] = 0.f;
#pragma unroll 2
        for (int i = 0; i < kHid; i += 4) {
            const float4 da4 = *reinterpret_cast<const float4 *>(&sda[r][i]);
            const float da[4] = {da4.x, da4.y, da4.z, da4.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
#pragma unroll
                for (int k = 0; k < O; k += 4) {
                    const float4 w = *reinterpret_cast<const float4 *>(&sWs[(i + c) * DIN + k0 + k]);
                    const float4 x = *reinterpret_cast<const float4 *>(&sWn[(i + c) * DIN + k0 + k]);
                    a[k] = fmaf(w.x, da[c], a[k]);
                    a[k + 1] = fmaf(w.y, da[c], a[k + 1]);
                    a[k + 2] = fmaf(w.z, da[c], a[k + 2]);
                    a[k + 3] = fmaf(w.w, da[c], a[k + 3]);
                    n[k] = fmaf(x.x, da[c], n[k]);
                    n[k + 1] = fmaf(x.y, da[c], n[k + 1]);
                    n[k + 2] = fmaf(x.z, da[c], n[k + 2]);
                    n[k + 3] = fmaf(x.w, da[c], n[k + 3]);
                }
            }
        }
        if (row < d.nl_pad) {
            const float inv = sinv[r];
#pragma unroll
            for (int k = 0; k < O; k += 4) {
                const size_t o = ((size_t)row * DIN + k0 + k) / 4;
                reinterpret_cast<float4 *>(dh_in_self)[o] = make_float4(a[k], a[k + 1], a[k + 2], a[k + 3]);
                reinterpret_cast<float4 *>(tbuf)[o] =
                    make_float4(n[k] * inv, n[k + 1] * inv, n[k + 2] * inv, n[k + 3] * inv);
            }
        }
    }
    // dW[i][c] = sum_r da[r][i] hm[r][c], c over the DIN channels of h, then of the mean
    float *G = partial + (size_t)blockIdx.x * MPNN_NUM_PARAMS;
    constexpr int I = DIN / 8;
    const int i0 = I * (t / DIN), c0 = 2 * (t % DIN);
    float g[I][2];
#pragma unroll
    for (int i = 0; i < I; i++) g[i][0] = g[i][1] = 0.f;
#pragma unroll 8
    for (int r = 0; r < kBwdRows; r++) {
        const float2 x = *reinterpret_cast<const float2 *>(&shm[r][c0]);
        float da[I];
        if (I == 4) {
            const float4 q = *reinterpret_cast<const float4 *>(&sda[r][i0]);
            da[0] = q.x, da[I - 3 > 0 ? 1 : 0] = q.y, da[I - 2 > 0 ? 2 : 0] = q.z, da[I - 1] = q.w;
        } else {
            da[0] = sda[r][i0];
        }
#pragma unroll
        for (int i = 0; i < I; i++) {
            g[i][0] = fmaf(da[i], x.x, g[i][0]);
            g[i][1] = fmaf(da[i], x.y, g[i][1]);
        }
    }
#pragma unroll
    for (int i = 0; i < I; i++) {
        float *o = G + (c0 < DIN ? ws : wn) + (i0 + i) * DIN + c0 % DIN;
        o[0] = g[i][0];
        o[1] = g[i][1];
    }
    if (warp == 0) {
        float a = 0.f;
#pragma unroll 8
        for (int r = 0; r < kBwdRows; r++) a += sda[r][lane];
        G[bo + lane] = a;
    } else if (TOP && warp == 1) {
        float a = 0.f;
        const int n = min(kBwdRows, d.nl_pad - row0);
#pragma unroll 8
        for (int r = 0; r < n; r++) a = fmaf(sds[r], __bfloat162float(hout[(size_t)(row0 + r) * kHid + lane]), a);
        G[P.wo + lane] = a;
    } else if (TOP && t == 64) {
        float a = 0.f;
#pragma unroll 8
        for (int r = 0; r < kBwdRows; r++) a += sds[r];
        G[P.bo] = a;
    }
}

// grad[e] = sum over CTAs of partial[cta][e] (parameter e): eight strided
// sums, then those in order
__global__ void __launch_bounds__(256) k_sum_partials(const float *partial, int nctas, float *grad)
{
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
    float a = 0.f;
    if (e < MPNN_NUM_PARAMS) {
#pragma unroll 8
        for (int c = warp; c < nctas; c += 8) a += partial[(size_t)c * MPNN_NUM_PARAMS + e];
    }
    part[warp][lane] = a;
    __syncthreads();
    if (warp != 0 || e >= MPNN_NUM_PARAMS) return;
    for (int w = 1; w < 8; w++) a += part[w][lane];
    grad[e] = a;
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

}  // namespace

int mpnn_forward(const DeviceBatch &d, MpnnBuffers &B, const float *theta_dev, bool write_phi, cudaStream_t s)
{
    constexpr MpnnLayout L = mpnn_layout();
    const int nr = cdiv(d.nl_pad, kRowThreads), nf = d.nl_pad / kFwdRows;
    if (d.precision == PREC_FP64)
        k_features<double><<<nr, kRowThreads, 0, s>>>(d, B.x0);
    else
        k_features<float><<<nr, kRowThreads, 0, s>>>(d, B.x0);
    k_layer<kFin, false><<<nf, 4 * kFwdRows, 0, s>>>(d, theta_dev, L.ws[0], L.wn[0], L.b[0], B.x0, B.h[0], nullptr, 0);
    k_layer<kHid, false><<<nf, 4 * kFwdRows, 0, s>>>(d, theta_dev, L.ws[1], L.wn[1], L.b[1], B.h[0], B.h[1], nullptr,
                                                     0);
    k_layer<kHid, true><<<nf, 4 * kFwdRows, 0, s>>>(d, theta_dev, L.ws[2], L.wn[2], L.b[2], B.h[1], B.h[2], B.omega,
                                                    write_phi ? 1 : 0);
    count_launches(4);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int mpnn_loss(const DeviceBatch &d, MpnnBuffers &B, cudaStream_t s)
{
    const int nr = cdiv(d.nl_pad, kRowThreads);
    if (d.precision == PREC_FP64)
        k_loss_restrict<double><<<d.n_segs, CG_SEG_MAX_ROWS, 0, s>>>(d, B.v, B.gvec);
    else
        k_loss_restrict<float><<<d.n_segs, CG_SEG_MAX_ROWS, 0, s>>>(d, B.v, B.gvec);
    k_loss_apply<<<d.n_segs, kApplyThreads, 0, s>>>(d, B.gvec, B.v, B.omega, B.e);
    if (d.precision == PREC_FP64)
        k_loss_products<double><<<nr, kRowThreads, 0, s>>>(d, B.e, B.v, B.gw, B.cta_sums);
    else
        k_loss_products<float><<<nr, kRowThreads, 0, s>>>(d, B.e, B.v, B.gw, B.cta_sums);
    k_loss_total<<<1, 96, 0, s>>>(B.cta_sums, nr, B.scal);
    count_launches(4);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int mpnn_backward(const DeviceBatch &d, MpnnBuffers &B, const float *theta_dev, float *grad_dev, cudaStream_t s)
{
    constexpr MpnnLayout L = mpnn_layout();
    constexpr int T = 4 * kBwdRows;
    const int nb = cdiv(d.nl_pad, kBwdRows);
    k_layer_bwd<kHid, true><<<nb, T, 0, s>>>(d, theta_dev, L.ws[2], L.wn[2], L.b[2], B.h[1], B.h[2], B.omega, B.gw,
                                             B.scal, nullptr, nullptr, B.dself[0], B.tbuf[0], B.partial);
    k_layer_bwd<kHid, false><<<nb, T, 0, s>>>(d, theta_dev, L.ws[1], L.wn[1], L.b[1], B.h[0], B.h[1], nullptr, nullptr,
                                              nullptr, B.dself[0], B.tbuf[0], B.dself[1], B.tbuf[1], B.partial);
    k_layer_bwd<kFin, false><<<nb, T, 0, s>>>(d, theta_dev, L.ws[0], L.wn[0], L.b[0], B.x0, B.h[0], nullptr, nullptr,
                                              nullptr, B.dself[1], B.tbuf[1], nullptr, nullptr, B.partial);
    k_sum_partials<<<cdiv(MPNN_NUM_PARAMS, 32), 256, 0, s>>>(B.partial, nb, grad_dev);
    count_launches(4);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace ffea
