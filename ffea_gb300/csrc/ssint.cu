// ssint.cu -- surface-surface interactions of FFEA on the GPU.
//
// Replaces VdW_solver::solve for "vdw_type = lennard-jones"
// (src/VdW_solver.cpp:168-210, 237-330, 338-394, 664-752), "steric"
// (Steric_solver, src/VdW_solver.cpp:458-486), "ljsteric" (LJSteric_solver:
// steric where the faces' element tetrahedra overlap, Lennard-Jones
// elsewhere) and "gensoft" (GenSoftSSINT_solver, src/VdW_solver.cpp:488-563,
// 701-771), together with the nearest-neighbour grid they walk
// (NearestNeighbourLinkedListCube::build_nearest_neighbour_lookup,
// src/NearestNeighbourLinkedListCube.cpp:27-76) and the aggregation of face
// forces onto nodes (src/Blob.cpp:3841-3851).  The steric types first run,
// between steps 4 and 5 below, k_steric_find (the faces that have partners
// whose tetrahedra may overlap theirs) and k_steric (overlap volume of the two
// element tetrahedra by convex clipping, its forward-difference gradient and
// FFEA's barycentric weights) on those, whose force lands on the four nodes of
// each face's element; k_pairs then skips the pairs k_steric handled.
//
// GPU layout and passes (one stream, no host round trip between them):
//   1. k_face_geom   one thread per active face: gathers its three corners,
//                    computes area, unit normal and centroid as
//                    Face::calc_area_normal_centroid (src/Face.cpp:197-219),
//                    bins the centroid into a cell (floor(c/h), wrapped once,
//                    LinkedListCube::pbc) and counts the cell's faces.
//   2. k_scan_local / k_scan_blocks   exclusive scan of the cell counts.
//   3. k_scatter     places every face in its cell's segment.
//   4. k_sort_cells  sorts each segment by face index (deterministic order):
//      k_sort_large  a thread per face ranks it among its cell's where those
//                    are up to 64, a CTA per cell sorts up to 4096 (bitonic, in
//                    shared memory); a fuller cell makes the call an error (the
//                    grid is far too coarse).
//   5. k_pairs       one warp per face, in cell order so that neighbouring
//                    warps read the same cells: the lanes share the faces of
//                    the 27 cells around its own and integrate the LJ force
//                    of every partner the reference would pair with it; a
//                    fixed shuffle tree sums the lanes.  A pair (i, j) is evaluated
//                    from both sides, each side keeping only its own face's
//                    forces: twice the arithmetic of one evaluation, but no
//                    atomics on forces and a fixed summation order (the
//                    per-blob-pair energies use FP64 atomics, so their last
//                    bits may vary from run to run).  The pair
//                    is always evaluated with the lower pool index as FFEA's
//                    f1, so that both sides use the same point forces.
//   6. k_node_gather one thread per node: sums its faces' corner forces in
//                    face order (a CSR built at creation).
// The file is compiled with -fmad=false so that every product and sum rounds
// as in the reference's FP64 code where that decides something: cell binning,
// and the normal test, whose FP32 form decides only what is clear of its
// rounding.  The force of a pair differs from FFEA's at the rounding level
// (pot_pair; bound by the FP64 pipe): Gauss points and centroids are formed
// once a face, the point forces come from 1/r^2 with fused products (one
// reciprocal and, for Lennard-Jones, no square root a point pair), the nine
// weighted terms per corner are regrouped through column sums of the
// (symmetric) force matrix, and the weights follow once per face.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/ffea_gpu.h"

namespace ffea {
void set_last_error(const char *msg);  // api.cu
}

struct ffea_gpu_ssint {
    int num_nodes = 0, num_faces = 0, num_active = 0, num_types = 0, num_blobs = 0;
    int nx = 0, ny = 0, nz = 0, inc_self = 0;
    int type = FFEA_GPU_SSINT_LJ;
    double steric_factor = 0.0, steric_dr = 0.0;
    long long ncell = 0;
    int nblocks = 0;
    double h = 0.0;
    cudaStream_t stream = nullptr;
    // per active face, in the caller's face order
    int *d_corner = nullptr;    // 4 node indices: the corners, then the element's fourth node (-1: none)
    int *d_blob = nullptr;
    int *d_type = nullptr;
    double *d_geo = nullptr;    // 16 doubles: corners (9), unit normal (3), area, fourth node (3)
    double *d_gp = nullptr;     // 16 doubles: Gauss points (9), unit normal (3), area, centroid (3)
    float4 *d_nb = nullptr;     // the normal in FP32 and the blob (its bits)
    float4 *d_box = nullptr;    // steric types: two, the element tetrahedron's bounding box in FP32, rounded outwards
    int *d_cell = nullptr;      // -1: outside the box
    double *d_fforce = nullptr; // 12 doubles: force on each corner and on the fourth node
    double *d_corr = nullptr;   // periodic blob corrections (num_blobs^2 x 3), when set
    int has_corr = 0, sticky = 0;
    // steric types: per face its candidates (MAX_STERIC_PARTNERS kept), then the partners whose tetrahedra overlap
    int *d_stlist = nullptr;
    int *d_stcnt = nullptr;     // their number per face
    int *d_stwork = nullptr;    // the faces with candidates
    int sms = 0;
    // grid
    int *d_count = nullptr;     // ncell
    int *d_start = nullptr;     // ncell, block-local exclusive prefix
    int *d_block = nullptr;     // nblocks, global prefix of each block
    int *d_binned = nullptr;    // num_active faces by cell, in no order within a cell
    int *d_sorted = nullptr;    // num_active faces in cell order, each cell in face order
    // nodes
    int *d_node_ptr = nullptr;  // num_nodes + 1
    int *d_node_ent = nullptr;  // face * 4 + corner (3: the fourth node), face order
    double *d_emin = nullptr, *d_rmin = nullptr, *d_k0 = nullptr;
    double *d_pos = nullptr, *d_force = nullptr, *d_energy = nullptr;  // staging of the host entry point
    unsigned long long *d_stats = nullptr;  // [0] pairs, [1] out-of-box faces, [2] large cells, [3] oversized cells,
                                            // [4] faces with too many steric partners, [5] with steric candidates, [6] of those given out
    int *d_large = nullptr;                 // cells of more than kSortSmall faces (k_sort_large)
};

namespace {

constexpr int kScanBlock = 1024;
constexpr int kStats = 7;

int fail(const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    ffea::set_last_error(buf);
    return FFEA_GPU_ERROR;
}

#define SSINT_CUDA(call)                                                                    \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) return fail("%s: %s", #call, cudaGetErrorString(e_));        \
    } while (0)

// 3-point rule on a triangle (src/VdW_solver.cpp:61-71): weight kW, point k
// has barycentric coordinate eta(k, d).  Written as constant expressions so
// that, in the fully unrolled loops, products of constants such as
// kW * kW * eta fold at compile time (to the same double the reference
// computes at run time) instead of costing FP64 instructions per pair.
constexpr double kW = 0.333333333333333;
__host__ __device__ constexpr double eta(int k, int d) { return k == d ? 0.666666666666667 : 0.166666666666667; }

__device__ __forceinline__ int wrap(int x, int n)
{
    if (x < 0) return x + n;
    if (x >= n) return x - n;
    return x;
}

__global__ void k_face_geom(const double *__restrict__ pos, const int *__restrict__ corner, int nf, double h,
                            int nx, int ny, int nz, const int *__restrict__ fblob, double *__restrict__ geo,
                            double *__restrict__ gp, float4 *__restrict__ nb, float4 *__restrict__ box,
                            int *__restrict__ cell, int *__restrict__ count, unsigned long long *stats)
{
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    double v[3][3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int n = corner[4 * f + k];
#pragma unroll
        for (int d = 0; d < 3; d++) v[k][d] = pos[3 * (long long)n + d];
    }
    const int apex = corner[4 * f + 3];
    double a[3], b[3], nrm[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        a[d] = v[1][d] - v[0][d];
        b[d] = v[2][d] - v[0][d];
    }
    nrm[0] = a[1] * b[2] - a[2] * b[1];
    nrm[1] = a[2] * b[0] - a[0] * b[2];
    nrm[2] = a[0] * b[1] - a[1] * b[0];
    const double mag = sqrt(nrm[0] * nrm[0] + nrm[1] * nrm[1] + nrm[2] * nrm[2]);
    double *g = geo + 16 * (long long)f;
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int d = 0; d < 3; d++) g[3 * k + d] = v[k][d];
#pragma unroll
    for (int d = 0; d < 3; d++) g[9 + d] = nrm[d] / mag;
    g[12] = .5 * mag;
#pragma unroll
    for (int d = 0; d < 3; d++) g[13 + d] = apex >= 0 ? pos[3 * (long long)apex + d] : 0.0;
    // what the pair kernel reads of a face, formed once here instead of once
    // per pair
    double *q = gp + 16 * (long long)f;
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int d = 0; d < 3; d++) q[3 * k + d] = eta(k, 0) * v[0][d] + eta(k, 1) * v[1][d] + eta(k, 2) * v[2][d];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        q[9 + d] = g[9 + d];
        q[13 + d] = (1.0 / 3.0) * (v[0][d] + v[1][d] + v[2][d]);
    }
    q[12] = g[12];
    nb[f] = make_float4((float)g[9], (float)g[10], (float)g[11], __int_as_float(fblob[f]));
    if (box) {  // steric types: the element tetrahedron's bounding box, rounded outwards
        float b[6];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            b[d] = fminf(fminf(__double2float_rd(v[0][d]), __double2float_rd(v[1][d])),
                         fminf(__double2float_rd(v[2][d]), __double2float_rd(g[13 + d])));
            b[3 + d] = fmaxf(fmaxf(__double2float_ru(v[0][d]), __double2float_ru(v[1][d])),
                             fmaxf(__double2float_ru(v[2][d]), __double2float_ru(g[13 + d])));
        }
        box[2 * (long long)f] = make_float4(b[0], b[1], b[2], 0.f);
        box[2 * (long long)f + 1] = make_float4(b[3], b[4], b[5], 0.f);
    }
    int c[3];
    const int dims[3] = {nx, ny, nz};
    bool inside = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double fl = floor(q[13 + d] / h);
        // cells beyond int range (or a NaN centroid) are outside the box as well
        int x = (fl >= -2147483647.0 && fl <= 2147483647.0) ? (int)fl : -2147483647;
        x = (x < -dims[d] || x >= 2 * dims[d]) ? -1 : wrap(x, dims[d]);
        if (x < 0 || x >= dims[d]) inside = false;
        c[d] = x;
    }
    if (!inside) {
        cell[f] = -1;
        atomicAdd(&stats[1], 1ull);
        return;
    }
    const int id = (c[0] * ny + c[1]) * nz + c[2];
    cell[f] = id;
    atomicAdd(&count[id], 1);
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// block-local exclusive scan of kScanBlock cells; the block's total to block_sum
__global__ void __launch_bounds__(kScanBlock) k_scan_local(const int *__restrict__ count, long long ncell,
                                                           int *__restrict__ start, int *__restrict__ block_sum)
{
    __shared__ int warp_tot[kScanBlock / 32];
    const long long i = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = i < ncell ? count[i] : 0;
    const int incl = warp_incl_scan(v, lane);
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
        int t = warp_incl_scan(warp_tot[lane], lane);
        warp_tot[lane] = t;
    }
    __syncthreads();
    const int base = w ? warp_tot[w - 1] : 0;
    if (i < ncell) start[i] = base + incl - v;
    if (threadIdx.x == kScanBlock - 1) block_sum[blockIdx.x] = base + incl;
}

// exclusive scan of the block totals, in place, by one CTA
__global__ void __launch_bounds__(kScanBlock) k_scan_blocks(int *__restrict__ block, int nblocks)
{
    __shared__ int warp_tot[kScanBlock / 32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nblocks; base += kScanBlock) {
        const int i = base + threadIdx.x;
        const int v = i < nblocks ? block[i] : 0;
        const int incl = warp_incl_scan(v, lane);
        if (lane == 31) warp_tot[w] = incl;
        __syncthreads();
        if (w == 0) warp_tot[lane] = warp_incl_scan(warp_tot[lane], lane);
        __syncthreads();
        const int pre = (w ? warp_tot[w - 1] : 0) + incl - v;
        const int c = carry;
        if (i < nblocks) block[i] = c + pre;
        __syncthreads();
        if (threadIdx.x == kScanBlock - 1) carry = c + pre + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) block[nblocks] = carry;  // faces binned in all
}

__device__ __forceinline__ int cell_begin(const int *start, const int *block, long long c)
{
    return start[c] + block[c / kScanBlock];
}

// block[nblocks] holds the number of faces binned, the end of the last cell
__device__ __forceinline__ int cell_end(const int *start, const int *block, long long c, long long ncell,
                                        int nblocks)
{
    return c + 1 < ncell ? cell_begin(start, block, c + 1) : block[nblocks];
}

__global__ void k_scatter(const int *__restrict__ cell, int nf, const int *__restrict__ start,
                          const int *__restrict__ block, int *__restrict__ count, int *__restrict__ sorted)
{
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int c = cell[f];
    if (c < 0) return;
    const int slot = cell_begin(start, block, c) + atomicSub(&count[c], 1) - 1;
    sorted[slot] = f;
}

// Each cell's faces sorted by face index: a thread per face counts the faces
// of its cell with a lower index, which is its place (cells of at most
// kSortSmall faces; a thread per cell sorting by insertion took 43-54 us where
// this takes a few).  A larger cell, up to kSortMax faces, is copied and listed
// for k_sort_large (one CTA per cell); a cell above that is counted in stats[3]
// and makes the call an error, so that a grid far too coarse for the mesh
// fails at once.
constexpr int kSortSmall = 64;
constexpr int kSortMax = 4096;
constexpr int kSortLargeCtas = 256;

__global__ void k_sort_cells(long long ncell, int nblocks, const int *__restrict__ start,
                             const int *__restrict__ block, const int *__restrict__ cell,
                             const int *__restrict__ binned, int *__restrict__ sorted, int *__restrict__ large,
                             unsigned long long *stats)
{
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= block[nblocks]) return;
    const int f = binned[w];
    const long long c = cell[f];
    const int b = cell_begin(start, block, c);
    const int e = cell_end(start, block, c, ncell, nblocks);
    if (e - b > kSortSmall) {
        sorted[w] = f;
        if (w == b) {  // once per cell
            if (e - b > kSortMax) atomicAdd(&stats[3], 1ull);
            else large[atomicAdd(&stats[2], 1ull)] = (int)c;
        }
        return;
    }
    int place = b;
    for (int k = b; k < e; k++) place += binned[k] < f;
    sorted[place] = f;
}

// The listed large cells, one CTA each (grid-stride over the list): a
// bitonic sort in shared memory of the cell's face indices, padded to a
// power of two.
__global__ void __launch_bounds__(256) k_sort_large(long long ncell, int nblocks, const int *__restrict__ start,
                                                    const int *__restrict__ block, int *__restrict__ sorted,
                                                    const int *__restrict__ large,
                                                    const unsigned long long *__restrict__ stats)
{
    __shared__ int v[kSortMax];
    const int nl = (int)stats[2];
    for (int k = blockIdx.x; k < nl; k += gridDim.x) {
        const long long c = large[k];
        const int b = cell_begin(start, block, c);
        const int n = cell_end(start, block, c, ncell, nblocks) - b;  // kSortSmall < n <= kSortMax
        int m = 1;
        while (m < n) m <<= 1;
        for (int i = threadIdx.x; i < m; i += blockDim.x) v[i] = i < n ? sorted[b + i] : INT_MAX;
        __syncthreads();
        for (int size = 2; size <= m; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = threadIdx.x; i < m; i += blockDim.x) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const bool up = (i & size) == 0;
                        const int a = v[i], bb = v[j];
                        if ((a > bb) == up) {
                            v[i] = bb;
                            v[j] = a;
                        }
                    }
                }
                __syncthreads();
            }
        for (int i = threadIdx.x; i < n; i += blockDim.x) sorted[b + i] = v[i];
        __syncthreads();
    }
}

// The integrated point-pair potentials of one face pair (FFEA's f1 the face
// with the lower index):
//   POT_LJ    do_lj_interaction (src/VdW_solver.cpp:237-330) with
//             calc_lj_force_pair_matrix / calc_lj_factors (:664-699, :736-752);
//   POT_SOFT  do_gensoft_interaction (:488-563) with
//             calc_gensoft_force_pair_matrix / calc_gensoft_factors (:701-734, :754-771).
// own, oth: the Gauss points of the face whose force is summed and of its
// partner; lower: own is f1.  FFEA's matrix of point forces is symmetric by
// construction (the entry of points k < l of f1 and f2 stands for (l, k) too),
// so both faces' forces are weighted sums of its column sums
// S_l = sum_k fpm[k][l] (force1_j = sum_l W^2 eta_l[j] S_l, force2 = -force1),
// and with d = own - oth the own face's S has the same form on either side.
// Adds area product * S to S (the weights follow once per face) and returns
// the pair energy.  k0: the soft potential's k0 (unused by POT_LJ).
//
// FP64-bound: an FP64 instruction takes 64 issue slots on GB300, so the point
// forces are written with the fewest of them: fm (p - q) / r =
// 12 emin f6 (f6 - 1) / r^2 (p - q) needs one reciprocal and no square root,
// and products are fused (explicitly: the file is compiled without
// contraction).  About 200 instructions a pair and side, from about 600.
constexpr int POT_LJ = 0, POT_SOFT = 1;

template <int POT>
__device__ __forceinline__ double pot_pair(const double (&own)[9], const double (&oth)[9], double apaq, bool lower,
                                           double emin, double rmin, double k0, double (&S)[3][3])
{
    double T[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    const double r2m = rmin * rmin;
    const double r6 = r2m * r2m * r2m;
    const double c12 = 12 * emin;
    // soft potential: t = fm / r = s1 r^2 + s2 r + k0, e = e4 r^4 + e3 r^3 + k0/2 r^2 - emin
    double s1 = 0, s2 = 0, e4 = 0, e3 = 0;
    if constexpr (POT == POT_SOFT) {
        const double irm = 1. / rmin, irm2 = irm * irm, k0rm = k0 * rmin, k0rm2 = k0rm * rmin, eps = emin * irm;
        s1 = 2 * (k0rm - 6 * eps) * irm2 * irm;
        s2 = 3 * (4 * eps - k0rm) * irm2;
        e4 = (0.5 * k0rm2 - 3 * emin) * irm2 * irm2;
        e3 = (4 * emin - k0rm2) * irm2 * irm;
    }
    double energy = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int l = k; l < 3; l++) {
            // points k of f1 and l of f2
            double v[3];
#pragma unroll
            for (int d = 0; d < 3; d++)
                v[d] = (lower ? own[3 * k + d] : own[3 * l + d]) - (lower ? oth[3 * l + d] : oth[3 * k + d]);
            const double r2 = fma(v[0], v[0], fma(v[1], v[1], v[2] * v[2]));
            double t, e;
            if constexpr (POT == POT_LJ) {
                const double ri2 = __drcp_rn(r2);
                const double f6 = r6 * (ri2 * ri2 * ri2);
                t = c12 * f6 * (f6 - 1) * ri2;
                e = f6 * (f6 - 2);
            } else {
                const double r = sqrt(r2);
                t = fma(s1, r2, fma(s2, r, k0));
                e = fma(r2, fma(e4, r2, fma(e3, r, 0.5 * k0)), -emin);
            }
            energy = l == k ? energy + e : fma(2.0, e, energy);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                T[l][d] = fma(t, v[d], T[l][d]);
                if (l != k) T[k][d] = fma(t, v[d], T[k][d]);
            }
        }
    }
#pragma unroll
    for (int l = 0; l < 3; l++)
#pragma unroll
        for (int d = 0; d < 3; d++) S[l][d] = fma(apaq, T[l][d], S[l][d]);
    return (POT == POT_LJ ? kW * kW * emin : kW * kW) * energy * apaq;
}

// ---- steric: the overlap of two tetrahedra -------------------------------
// The overlap of tetrahedra A and B is clipped out of A by B's four
// half-spaces: each face polygon clipped in turn (Sutherland-Hodgman) and each
// cut closed by a cap polygon, its points ordered by angle.  Two tetrahedra
// intersect in at most 8 half-spaces, so the polyhedron has at most 8 faces
// of at most 7 vertices.  Its volume is a fan of tetrahedra from the mean of
// its vertices; its "centre" is what FFEA's volumeIntersectionII returns
// (findCM, src/VolumeIntersection.cpp:95-104): the mean of its distinct
// vertices.  Points closer than 1e-9 of the tetrahedra's extent are one.
constexpr int kStV = 8, kStF = 8, kStC = 16, kStU = 32;

struct StPolyh {
    int nf;
    int n[kStF];
    double v[kStF][kStV][3];
};

__device__ __forceinline__ double st_dot(const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

__device__ __forceinline__ double st_tet_volume(const double *a, const double *b, const double *c, const double *d)
{
    const double u0 = b[0] - a[0], u1 = b[1] - a[1], u2 = b[2] - a[2];
    const double v0 = c[0] - a[0], v1 = c[1] - a[1], v2 = c[2] - a[2];
    const double w0 = d[0] - a[0], w1 = d[1] - a[1], w2 = d[2] - a[2];
    const double x0 = v1 * w2 - v2 * w1, x1 = v2 * w0 - v0 * w2, x2 = v0 * w1 - v1 * w0;
    return (u0 * x0 + u1 * x1 + u2 * x2) / 6.0;
}

// x joins the n distinct points pts unless one is within sqrt(tol2) of it.
// org and far decide most comparisons in FP32: points whose FP32 offsets from
// org differ by more than far in a component are distinct (far is 1e-5 of the
// extent, a hundred FP32 roundings of an offset; the tolerance is 1e-9 of it).
__device__ __forceinline__ void st_add_unique(double (*pts)[3], float (*off)[3], int &n, int cap, const double *x,
                                              const double *org, float far, double tol2)
{
    const float f[3] = {(float)(x[0] - org[0]), (float)(x[1] - org[1]), (float)(x[2] - org[2])};
    for (int u = 0; u < n; u++) {
        const float g = fmaxf(fmaxf(fabsf(f[0] - off[u][0]), fabsf(f[1] - off[u][1])), fabsf(f[2] - off[u][2]));
        if (g > far) continue;
        const double e0 = x[0] - pts[u][0], e1 = x[1] - pts[u][1], e2 = x[2] - pts[u][2];
        if (e0 * e0 + e1 * e1 + e2 * e2 <= tol2) return;
    }
    if (n < cap) {
        for (int c = 0; c < 3; c++) {
            pts[n][c] = x[c];
            off[n][c] = f[c];
        }
        n++;
    }
}

// the sign of a double from its bits (-1, 0, 1), off the FP64 pipe; a NaN,
// which compares with nothing, has none of them
constexpr int kStNan = 2;
__device__ __forceinline__ int st_sign(double x)
{
    const int hi = __double2hiint(x), lo = __double2loint(x), mag = hi & 0x7fffffff;
    if ((mag | lo) == 0) return 0;
    if (mag > 0x7ff00000 || (mag == 0x7ff00000 && lo != 0)) return kStNan;
    return hi < 0 ? -1 : 1;
}

// increasing with atan2(y, x) over (-pi, pi], without its cost
__device__ __forceinline__ double st_angle(double y, double x)
{
    const double t = y / (fabs(x) + fabs(y));
    return __double2hiint(x) >= 0 ? t : copysign(2.0, y) - t;
}

__constant__ int c_tri[4][3] = {{1, 2, 3}, {0, 2, 3}, {0, 1, 3}, {0, 1, 2}};

// clip P by n . x <= off; false when nothing is left.  A vertex's distance is
// formed once and kept, and its sign read from its bits: comparisons run on
// the FP64 pipe too.  What a NaN decides is what it decides in comparisons
// (a distance from a node at infinity): it is not inside, starts no crossing,
// and as the first of the distances it leaves their range open.
__device__ bool st_clip(StPolyh &P, const double *nrm, double off, const double *org, float far, double tol2)
{
    double sd[kStF][kStV];
    bool neg = false, pos = false, open = false;
    for (int f = 0; f < P.nf; f++)
        for (int k = 0; k < P.n[f]; k++) {
            const double sv = st_dot(nrm, P.v[f][k]) - off;
            const int g = st_sign(sv);
            sd[f][k] = sv;
            neg |= g < 0;
            pos |= g == 1;
            open |= f == 0 && k == 0 && g == kStNan;
        }
    if (!neg && !open) {
        P.nf = 0;
        return false;
    }
    if (!pos && !open) return true;
    double cap[kStC][3];
    float capf[kStC][3];
    int nc = 0, nf = 0;
    for (int f = 0; f < P.nf; f++) {
        double out[kStV][3];
        int no = 0;
        const int m = P.n[f];
        for (int k = 0; k < m; k++) {
            const int kn = k + 1 < m ? k + 1 : 0;
            const double *a = P.v[f][k], *b = P.v[f][kn];
            const double sa = sd[f][k], sb = sd[f][kn];
            const int ga = st_sign(sa), gb = st_sign(sb);
            if (ga <= 0) {
                if (no < kStV) {
                    out[no][0] = a[0];
                    out[no][1] = a[1];
                    out[no][2] = a[2];
                    no++;
                }
                if (ga == 0) st_add_unique(cap, capf, nc, kStC, a, org, far, tol2);
            }
            if (ga * gb == -1) {
                const double t = sa / (sa - sb);
                double x[3];
                for (int c = 0; c < 3; c++) x[c] = a[c] + t * (b[c] - a[c]);
                if (no < kStV) {
                    out[no][0] = x[0];
                    out[no][1] = x[1];
                    out[no][2] = x[2];
                    no++;
                }
                st_add_unique(cap, capf, nc, kStC, x, org, far, tol2);
            }
        }
        if (no >= 3) {
            for (int k = 0; k < no; k++)
                for (int c = 0; c < 3; c++) P.v[nf][k][c] = out[k][c];
            P.n[nf++] = no;
        }
    }
    P.nf = nf;
    if (nf == 0) return false;
    if (nc >= 3 && nf < kStF) {
        double ctr[3] = {0, 0, 0};
        for (int k = 0; k < nc; k++)
            for (int d = 0; d < 3; d++) ctr[d] += cap[k][d];
        for (int d = 0; d < 3; d++) ctr[d] /= nc;
        int far = 0;
        double best = -1;
        for (int k = 0; k < nc; k++) {
            const double e0 = cap[k][0] - ctr[0], e1 = cap[k][1] - ctr[1], e2 = cap[k][2] - ctr[2];
            const double l = e0 * e0 + e1 * e1 + e2 * e2;
            if (l > best) {
                best = l;
                far = k;
            }
        }
        if (best > 0) {
            const double u[3] = {cap[far][0] - ctr[0], cap[far][1] - ctr[1], cap[far][2] - ctr[2]};
            const double w[3] = {nrm[1] * u[2] - nrm[2] * u[1], nrm[2] * u[0] - nrm[0] * u[2],
                                 nrm[0] * u[1] - nrm[1] * u[0]};
            double ang[kStC];
            for (int k = 0; k < nc; k++) {
                const double e[3] = {cap[k][0] - ctr[0], cap[k][1] - ctr[1], cap[k][2] - ctr[2]};
                ang[k] = st_angle(st_dot(e, w), st_dot(e, u));
            }
            for (int i = 1; i < nc; i++) {  // insertion sort by angle
                const double a = ang[i], v0 = cap[i][0], v1 = cap[i][1], v2 = cap[i][2];
                int j = i - 1;
                while (j >= 0 && ang[j] > a) {
                    ang[j + 1] = ang[j];
                    cap[j + 1][0] = cap[j][0];
                    cap[j + 1][1] = cap[j][1];
                    cap[j + 1][2] = cap[j][2];
                    j--;
                }
                ang[j + 1] = a;
                cap[j + 1][0] = v0;
                cap[j + 1][1] = v1;
                cap[j + 1][2] = v2;
            }
            const int nn = nc < kStV ? nc : kStV;
            for (int k = 0; k < nn; k++)
                for (int c = 0; c < 3; c++) P.v[P.nf][k][c] = cap[k][c];
            P.n[P.nf++] = nn;
        }
    }
    return true;
}

// overlap volume of tetrahedra A and B (4 x 3 each); with cm, FFEA's centre
__device__ __noinline__ double st_overlap(const double (*A)[3], const double (*B)[3], double *cm)
{
    double ext = 0.0;
    for (int i = 0; i < 4; i++)
        for (int d = 0; d < 3; d++) {
            ext = fmax(ext, fabs(A[i][d] - A[0][d]));
            ext = fmax(ext, fabs(B[i][d] - A[0][d]));
        }
    const double tol2 = (1e-9 * ext) * (1e-9 * ext);
    const double *org = A[0];
    const float far = 1e-5f * (float)ext;
    StPolyh P;
    P.nf = 4;
    for (int f = 0; f < 4; f++) {
        P.n[f] = 3;
        for (int k = 0; k < 3; k++)
            for (int c = 0; c < 3; c++) P.v[f][k][c] = A[c_tri[f][k]][c];
    }
    for (int f = 0; f < 4; f++) {
        // the half-space of B's face f (opposite vertex f) that holds B
        const double *t0 = B[c_tri[f][0]], *t1 = B[c_tri[f][1]], *t2 = B[c_tri[f][2]];
        const double u[3] = {t1[0] - t0[0], t1[1] - t0[1], t1[2] - t0[2]};
        const double v[3] = {t2[0] - t0[0], t2[1] - t0[1], t2[2] - t0[2]};
        double nrm[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
        double off = st_dot(nrm, t0);
        if (st_dot(nrm, B[f]) > off) {
            nrm[0] = -nrm[0];
            nrm[1] = -nrm[1];
            nrm[2] = -nrm[2];
            off = -off;
        }
        if (!st_clip(P, nrm, off, org, far, tol2)) {
            if (cm) cm[0] = cm[1] = cm[2] = 0.0;
            return 0.0;
        }
    }
    double o[3] = {0, 0, 0};
    int nv = 0;
    for (int f = 0; f < P.nf; f++)
        for (int k = 0; k < P.n[f]; k++) {
            for (int d = 0; d < 3; d++) o[d] += P.v[f][k][d];
            nv++;
        }
    for (int d = 0; d < 3; d++) o[d] /= nv;
    // six times the volume: a fan of tetrahedra per face, with the vertices'
    // offsets from o
    double vol6 = 0.0;
    for (int f = 0; f < P.nf; f++) {
        double u[3], v[3], w[3];
        for (int d = 0; d < 3; d++) {
            u[d] = P.v[f][0][d] - o[d];
            v[d] = P.v[f][1][d] - o[d];
        }
        for (int k = 2; k < P.n[f]; k++) {
            for (int d = 0; d < 3; d++) w[d] = P.v[f][k][d] - o[d];
            vol6 += fabs(u[0] * (v[1] * w[2] - v[2] * w[1]) + u[1] * (v[2] * w[0] - v[0] * w[2]) +
                         u[2] * (v[0] * w[1] - v[1] * w[0]));
            for (int d = 0; d < 3; d++) v[d] = w[d];
        }
    }
    const double vol = vol6 / 6.0;
    if (cm) {
        double uniq[kStU][3];
        float uniqf[kStU][3];
        int nu = 0;
        for (int f = 0; f < P.nf; f++)
            for (int k = 0; k < P.n[f]; k++) st_add_unique(uniq, uniqf, nu, kStU, P.v[f][k], org, far, tol2);
        cm[0] = cm[1] = cm[2] = 0.0;
        for (int u = 0; u < nu; u++)
            for (int d = 0; d < 3; d++) cm[d] += uniq[u][d];
        for (int d = 0; d < 3; d++) cm[d] *= 1.0 / nu;
    }
    return vol;
}

// The forces of one steric pair, f1 = A, f2 = B (the tetrahedra of the faces'
// elements), from its overlap volumes:
// Face::getTetraIntersectionVolumeTotalGradientAndShapeFunctions
// (src/Face.cpp:473-514) and do_steric_interaction's scaling
// (src/VdW_solver.cpp:470-483).  V > 0 and centre cm of A and B; vb[dir] with
// B moved by dr along dir, va[dir] with A moved.  Adds the node forces of the
// side with tetrahedron T, the A side's (phi1 k dV/dr) or the B side's
// (-phi2 k dV/dr), to out.
__device__ void steric_forces(const double (*T)[3], double V, const double *cm, const double *vb, const double *va,
                              double dr, double k, bool a_side, double out[4][3])
{
    // getLocalCoordinatesForLinTet (src/mat_vec_fns_II.cpp:725-734)
    double phi[4];
    phi[0] = st_tet_volume(cm, T[1], T[2], T[3]);
    phi[1] = -st_tet_volume(cm, T[0], T[2], T[3]);
    phi[2] = st_tet_volume(cm, T[0], T[1], T[3]);
    phi[3] = -st_tet_volume(cm, T[0], T[1], T[2]);
    const double tv = st_tet_volume(T[0], T[1], T[2], T[3]);
    for (int i = 0; i < 4; i++) phi[i] /= tv;
    double g[3];
    for (int dir = 0; dir < 3; dir++) {
        g[dir] = (vb[dir] - V) / dr;
        g[dir] -= (va[dir] - V) / dr;
        g[dir] *= k;
    }
    for (int i = 0; i < 4; i++)
        for (int d = 0; d < 3; d++) out[i][d] += a_side ? phi[i] * g[d] : -1.0 * phi[i] * g[d];
}

__constant__ int c_adj[27][3] = {{-1, -1, -1}, {-1, -1, 0}, {-1, -1, 1}, {-1, 0, -1}, {-1, 0, 0}, {-1, 0, 1},
                                 {-1, 1, -1},  {-1, 1, 0},  {-1, 1, 1},  {0, -1, -1}, {0, -1, 0}, {0, -1, 1},
                                 {0, 0, -1},   {0, 0, 0},   {0, 0, 1},   {0, 1, -1},  {0, 1, 0},  {0, 1, 1},
                                 {1, -1, -1},  {1, -1, 0},  {1, -1, 1},  {1, 0, -1},  {1, 0, 0},  {1, 0, 1},
                                 {1, 1, -1},   {1, 1, 0},   {1, 1, 1}};

// warps (faces) per CTA of k_pairs, and CTAs per SM (128 registers a thread):
// sixteen warps keep the FP64 pipes busy while others test candidates
constexpr int kPairWarps = 4, kPairCtas = 4;

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The faces of the 27 cells around face i's cell for one warp: s_beg / s_pre
// hold each cell's first sorted slot and the candidates before it; returns
// the number of candidates.
__device__ __forceinline__ int warp_cells(int ci, int nx, int ny, int nz, const int *__restrict__ start,
                                          const int *__restrict__ block, long long ncell, int nblocks, int lane,
                                          int *s_beg, int *s_pre)
{
    const int cz = ci % nz, cy = (ci / nz) % ny, cx = ci / (nz * ny);
    int len = 0, beg = 0;
    if (lane < 27) {
        const int x = wrap(cx + c_adj[lane][0], nx), y = wrap(cy + c_adj[lane][1], ny),
                  z = wrap(cz + c_adj[lane][2], nz);
        const long long cc = ((long long)x * ny + y) * nz + z;
        beg = cell_begin(start, block, cc);
        len = cell_end(start, block, cc, ncell, nblocks) - beg;
    }
    const int incl = warp_incl_scan(len, lane);
    if (lane < 27) {
        s_beg[lane] = beg;
        s_pre[lane] = incl - len;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 26);
    __syncwarp();
    return total;
}

// candidate k (< total) of the warp's cells
__device__ __forceinline__ int warp_candidate(int k, const int *s_beg, const int *s_pre, const int *__restrict__ sorted)
{
    int c = 0;
    while (c < 26 && s_pre[c + 1] <= k) c++;
    return sorted[s_beg[c] + (k - s_pre[c])];
}

// consider_interaction's checks for the types other than lennard-jones
// (src/VdW_solver.cpp:359-388): faces in front of each other, and within
// one blob (with self-interaction on) no shared node.  Symmetric in (i, j).
// With periodic corrections, cs = blob_corr[blob of A][blob of G] enters the
// separation (c_G - c_A - cs; FFEA's c2 - c1 - blob_corr[b1][b2] with its
// faces in either order, blob_corr being antisymmetric).
// A, G: face records of d_gp.
__device__ __forceinline__ bool steric_type_ok(const double *A, const double *G, bool same_blob, int inc_self,
                                               const int *ni, const int *nj, const double *cs)
{
    double sa = 0.0, sb = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double sep = G[13 + d] - A[13 + d];
        if (cs) sep -= cs[d];
        sa += sep * A[9 + d];
        sb += sep * G[9 + d];
    }
    if (sa < 0 && sb > 0) return false;
    if (inc_self && same_blob) {
        if (ni[3] == nj[3]) return false;
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int w = 0; w < 4; w++)
                if (ni[u] == nj[w]) return false;
    }
    return true;
}

// the element tetrahedron of face f: its corners, then the fourth node
__device__ __forceinline__ void face_tet(const double *__restrict__ geo, int f, double T[4][3])
{
    const double *g = geo + 16 * (long long)f;
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int d = 0; d < 3; d++) T[k][d] = g[3 * k + d];
#pragma unroll
    for (int d = 0; d < 3; d++) T[3][d] = g[13 + d];
}

// Whether face i (normal and blob in ni) admits face j: another face, another
// blob unless self-interaction is on, and normals that do not agree,
// n_i . n_j <= 0 in FP64.  The FP32 product is within 1e-6 of it and decides
// all but the nearly perpendicular pairs, which take the FP64 records.
__device__ __forceinline__ bool admits(int i, int j, float4 ni, const float4 *__restrict__ nb,
                                       const double *__restrict__ gp, int inc_self)
{
    const float4 nj = nb[j];
    if (j == i || (!inc_self && __float_as_int(ni.w) == __float_as_int(nj.w))) return false;
    const float c = ni.x * nj.x + ni.y * nj.y + ni.z * nj.z;
    if (fabsf(c) > 1e-6f) return c < 0.f;  // (a NaN goes on to the FP64 test)
    const double *A = gp + 16 * (long long)i, *G = gp + 16 * (long long)j;
    return !(A[9] * G[9] + A[10] * G[10] + A[11] * G[11] > 0.0);
}

// Whether a face j that `admits` has let pass is a steric partner of face i as
// far as is known without their overlap: consider_interaction takes the pair,
// and the bounding boxes of the two element tetrahedra (lo, hi: face i's) meet.
__device__ __forceinline__ bool steric_candidate(int i, int j, int bi, const int (&ni)[4],
                                                 const double (&lo)[3], const double (&hi)[3],
                                                 const double *__restrict__ geo, const double *__restrict__ gp,
                                                 const int *__restrict__ fblob, const int *__restrict__ corner,
                                                 int num_blobs, int inc_self, const double *__restrict__ corr)
{
    const int bj = fblob[j];
    // periodic: the partner as seen from face i, shifted by -blob_corr[bi][bj]
    const double *cs = corr ? corr + 3 * ((long long)bi * num_blobs + bj) : nullptr;
    int nj[4];
#pragma unroll
    for (int u = 0; u < 4; u++) nj[u] = corner[4 * j + u];
    if (!steric_type_ok(gp + 16 * (long long)i, gp + 16 * (long long)j, bi == bj, inc_self, ni, nj, cs)) return false;
    const double *G = geo + 16 * (long long)j;
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double sh = cs ? cs[d] : 0.0;
        const double a0 = G[d] - sh, a1 = G[3 + d] - sh, a2 = G[6 + d] - sh, a3 = G[13 + d] - sh;
        const double l = fmin(fmin(a0, a1), fmin(a2, a3)), h = fmax(fmax(a0, a1), fmax(a2, a3));
        if (h < lo[d] || l > hi[d]) ok = false;
    }
    return ok;
}

// the bounding box of face i's element tetrahedron
__device__ __forceinline__ void tet_box(const double *__restrict__ geo, int i, double (&lo)[3], double (&hi)[3])
{
    double T[4][3];
    face_tet(geo, i, T);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = fmin(fmin(T[0][d], T[1][d]), fmin(T[2][d], T[3][d]));
        hi[d] = fmax(fmax(T[0][d], T[1][d]), fmax(T[2][d], T[3][d]));
    }
}

// Whether the boxes of faces i (lo, hi) and j may meet: false only where the
// FP64 boxes, which lie within, do not.  cs: the periodic shift of j, or null.
__device__ __forceinline__ bool boxes_meet(float4 lo, float4 hi, const float4 *__restrict__ box, int j, const double *cs)
{
    float4 l = box[2 * (long long)j], h = box[2 * (long long)j + 1];
    if (cs) {
        l.x = __fsub_rd(l.x, __double2float_ru(cs[0]));
        l.y = __fsub_rd(l.y, __double2float_ru(cs[1]));
        l.z = __fsub_rd(l.z, __double2float_ru(cs[2]));
        h.x = __fsub_ru(h.x, __double2float_rd(cs[0]));
        h.y = __fsub_ru(h.y, __double2float_rd(cs[1]));
        h.z = __fsub_ru(h.z, __double2float_rd(cs[2]));
    }
    return !(h.x < lo.x || l.x > hi.x || h.y < lo.y || l.y > hi.y || h.z < lo.z || l.z > hi.z);
}

// The faces that have steric candidates, one warp per face in cell order:
// their number goes to stcnt, the first of them to the face's steric list,
// the face to `work` (stats[5] of them, in no order).  A face without any is
// done here: no partners, no steric force.  Most faces of most surfaces have
// none, and k_steric's registers leave room for eight warps an SM: with the
// candidates tested there, by a CTA a face, a solve of two 30 nm spheres apart
// took 1.95 ms, 0.18 so.  The faces of the 27 cells first pass the tests in
// FP32, which leave few of them, and those are queued for the ones in FP64
// (64 issue slots an instruction however few lanes it has): 21 us for two 4 nm
// spheres in contact and 93 for two 30 nm ones apart, 32 and 124 with every
// test in FP64.
constexpr int kFindWarps = 8;
__global__ void __launch_bounds__(32 * kFindWarps) k_steric_find(
    const double *__restrict__ geo, const double *__restrict__ gp, const float4 *__restrict__ nb,
    const float4 *__restrict__ box, const int *__restrict__ sorted, const int *__restrict__ cell,
    const int *__restrict__ start, const int *__restrict__ block, long long ncell, int nblocks, int nx, int ny, int nz,
    const int *__restrict__ fblob, const int *__restrict__ corner, int num_blobs, int inc_self,
    const double *__restrict__ corr, double *__restrict__ fforce, int *__restrict__ stlist, int *__restrict__ stcnt,
    int *__restrict__ work, unsigned long long *stats)
{
    __shared__ int s_pre[kFindWarps][28];
    __shared__ int s_beg[kFindWarps][27];
    __shared__ int s_q[kFindWarps][64];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kFindWarps + wi;
    if (w >= block[nblocks]) return;  // warp-uniform
    if (stats[3]) return;             // the call fails (a cell too full to sort)
    const int i = sorted[w];
    const int total = warp_cells(cell[i], nx, ny, nz, start, block, ncell, nblocks, lane, s_beg[wi], s_pre[wi]);
    const float4 nbi = nb[i], lo32 = box[2 * (long long)i], hi32 = box[2 * (long long)i + 1];
    const int bi = fblob[i];
    int n = 0, qn = 0;  // candidates found, queue length (< 64): warp-uniform
    // the tests in FP64 of the first (at most 32) of the queue
    auto test = [&] {
        int ni[4];
#pragma unroll
        for (int u = 0; u < 4; u++) ni[u] = corner[4 * i + u];
        double lo[3], hi[3];
        tet_box(geo, i, lo, hi);
        const int j = lane < qn ? s_q[wi][lane] : -1;
        const bool ok =
            j >= 0 && steric_candidate(i, j, bi, ni, lo, hi, geo, gp, fblob, corner, num_blobs, inc_self, corr);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const int slot = n + __popc(m & ((1u << lane) - 1u));
        if (ok && slot < FFEA_GPU_SSINT_MAX_STERIC_PARTNERS)
            stlist[FFEA_GPU_SSINT_MAX_STERIC_PARTNERS * i + slot] = j;
        n += __popc(m);
        const int rest = max(qn - 32, 0);
        const int moved = lane < rest ? s_q[wi][32 + lane] : 0;
        __syncwarp();
        if (lane < rest) s_q[wi][lane] = moved;
        qn = rest;
        __syncwarp();
    };
    for (int base = 0; base < total; base += 32) {
        const int k = base + lane;
        bool ok = false;
        int j = -1;
        if (k < total) {
            j = warp_candidate(k, s_beg[wi], s_pre[wi], sorted);
            ok = admits(i, j, nbi, nb, gp, inc_self) &&
                 boxes_meet(lo32, hi32, box, j, corr ? corr + 3 * ((long long)bi * num_blobs + fblob[j]) : nullptr);
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (ok) s_q[wi][qn + __popc(m & ((1u << lane) - 1u))] = j;
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) test();
    }
    if (qn > 0) test();
    if (lane == 0) {
        stcnt[i] = n;
        if (n) work[atomicAdd(&stats[5], 1ull)] = i;
    }
    if (n == 0 && lane < 12) fforce[12 * (long long)i + lane] = 0.0;
}

// The steric part of the steric types for the faces that k_steric_find
// listed.  A pair needs seven overlap volumes: its own and, where that is not
// zero, six with one tetrahedron moved, for the forward differences.  Each is
// computed as (lower index, higher index) = FFEA's (f1, f2), so both sides of
// a pair compute the same overlap.  Face i's side of the forces goes to fforce
// (12 values; this kernel runs before k_pairs), the partners that overlapped
// to i's steric list (a set: k_pairs skips them), the energy and the pair
// count from the side with the lower index.
//
// The clipping is a long chain of FP64 instructions, 64 issue slots each
// however few lanes it has.  Few faces: the chain itself decides, and with
// eight lanes a candidate, whose seven volumes take nearly the same course,
// and the candidates over many warps it is run about once.  Many faces: the
// FP64 pipes are busy, and the passes count; a lane per candidate for its own
// volume and then a lane per volume for the few that overlap take fewest.
// Lines between the ways, for a solve of two spheres in contact on 152 SMs:
// 130 listed faces, eight warps a face 387 us, four 417; 168 faces, 452 and
// 366; 466 faces, four warps 636 us, one 650; 903 faces, 974 and 800.  Two 8
// nm spheres took 1.94 ms with a lane per pair running the seven volumes in
// turn, 0.43 with eight warps a face for every face, 0.34 so; two 20 nm
// spheres with self-interaction 3.2, 4.2 and 1.1 ms.
constexpr int kStericWarps = 8;  // per CTA, one CTA per SM (registers)
static_assert(FFEA_GPU_SSINT_MAX_STERIC_PARTNERS == 32, "a lane per kept candidate");

struct StericArgs {
    const double *geo, *gp;
    const float4 *nb;
    const int *sorted, *cell, *start, *block;
    long long ncell;
    int nblocks, nx, ny, nz;
    const int *fblob, *corner;
    int num_blobs, inc_self;
    double factor, dr;
    const double *corr;
    double *fforce;
    int *stlist, *stcnt, *work;
    int sms;
    double *energy;
    unsigned long long *stats;
};

// overlap volume of the pair (i, j): v = 0 as they are, 1..3 with f2's
// tetrahedron moved by dr along x, y or z, 4..6 with f1's (clipped out of f2)
__device__ __forceinline__ double pair_overlap(const StericArgs &a, int i, int j, int v, double *cm)
{
    const int f1 = min(i, j), f2 = max(i, j);
    double A[4][3], B[4][3];
    face_tet(a.geo, f1, A);
    face_tet(a.geo, f2, B);
    // periodic: f2's tetrahedron minus blob_corr[b1][b2]
    // (Face::getTetraIntersectionVolumeTotalGradientAndShapeFunctions,
    // src/Face.cpp:517-531)
    if (a.corr) {
        const double *c = a.corr + 3 * ((long long)a.fblob[f1] * a.num_blobs + a.fblob[f2]);
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int d = 0; d < 3; d++) B[u][d] -= c[d];
    }
    const bool swap = v > 3;
    double M[4][3], O[4][3];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            M[u][d] = (swap ? A[u][d] : B[u][d]) + (v > 0 && d == (v - 1) % 3 ? a.dr : 0.0);
            O[u][d] = swap ? B[u][d] : A[u][d];
        }
    return st_overlap(O, M, cm);
}

// Face i's side of an overlapping pair (volume V, centre cm, volumes vb and
// va with f2 and with f1 moved) into out, and the pair's energy; `slot`: its
// place in the face's list
__device__ __forceinline__ void add_steric_pair(const StericArgs &a, int i, int j, double V, const double *cm,
                                                const double *vb, const double *va, int slot, double (&out)[4][3],
                                                unsigned long long &npairs)
{
    const bool lower = i < j;
    const int bi = a.fblob[i], bj = a.fblob[j];
    double T[4][3];
    face_tet(a.geo, i, T);
    if (a.corr && !lower) {
        const double *c = a.corr + 3 * ((long long)bj * a.num_blobs + bi);
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int d = 0; d < 3; d++) T[u][d] -= c[d];
    }
    steric_forces(T, V, cm, vb, va, a.dr, a.factor, lower, out);
    if (slot < FFEA_GPU_SSINT_MAX_STERIC_PARTNERS) a.stlist[FFEA_GPU_SSINT_MAX_STERIC_PARTNERS * i + slot] = j;
    if (lower) {
        atomicAdd(&a.energy[bi * a.num_blobs + bj], V * a.factor);
        npairs++;
    }
}

// The candidates of face i by W warps (this one is number wi) into queue q,
// evaluate(n) called for n > 0 of them at a time: the listed ones, or, where
// there are more than the list keeps, all found again
template <int W, typename Sync, typename Evaluate>
__device__ __forceinline__ void steric_candidates(const StericArgs &a, int i, int wi, int lane, int *q, int *s_beg,
                                                  int *s_pre, int *s_cnt, Sync sync, Evaluate evaluate)
{
    constexpr int NT = 32 * W;
    const int t = 32 * wi + lane, cand = a.stcnt[i];
    if (cand <= FFEA_GPU_SSINT_MAX_STERIC_PARTNERS) {
        if (t < cand) q[t] = a.stlist[FFEA_GPU_SSINT_MAX_STERIC_PARTNERS * i + t];
        sync();
        evaluate(cand);
        return;
    }
    if (wi == 0) {
        const int n = warp_cells(a.cell[i], a.nx, a.ny, a.nz, a.start, a.block, a.ncell, a.nblocks, lane, s_beg, s_pre);
        if (lane == 0) s_cnt[W] = n;
    }
    sync();
    const int total = s_cnt[W], bi = a.fblob[i];
    const float4 nbi = a.nb[i];
    int ni[4];
#pragma unroll
    for (int u = 0; u < 4; u++) ni[u] = a.corner[4 * i + u];
    double lo[3], hi[3];
    tet_box(a.geo, i, lo, hi);
    int qn = 0;  // queue length, the same for all warps
#pragma unroll 1
    for (int base = 0; base < total; base += NT) {
        const int k = base + t;
        const int j = k < total ? warp_candidate(k, s_beg, s_pre, a.sorted) : i;
        const bool ok = admits(i, j, nbi, a.nb, a.gp, a.inc_self) &&
                        steric_candidate(i, j, bi, ni, lo, hi, a.geo, a.gp, a.fblob, a.corner, a.num_blobs, a.inc_self,
                                         a.corr);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) s_cnt[wi] = __popc(m);
        sync();
        int at = qn;
        for (int k2 = 0; k2 < W; k2++) {
            if (k2 == wi && ok) q[at + __popc(m & ((1u << lane) - 1u))] = j;
            at += s_cnt[k2];
        }
        qn = at;
        sync();  // the queue, and s_cnt free
        if (qn >= 32 || base + NT >= total) {
            if (qn > 0) evaluate(qn);
            qn = 0;
            sync();
        }
    }
}

// the sum over a warp's lanes of the twelve values of out: value v in lanes
// 2 v and 2 v + 1 (a transposed butterfly, 16 additions)
__device__ __forceinline__ double warp_sum12(const double (&out)[4][3], int lane)
{
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = k < 12 ? out[k / 3][k % 3] : 0.0;
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const double send = upper ? v[k] : v[k + h], keep = upper ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Shared memory of a group of W warps of k_steric
template <int W>
struct StericGroup {
    int pre[28], beg[27];
    int cnt[W + 1];
    int q[32 * W + 32];
    int hit[32];          // W = 1: the partners that overlap, and their six volumes
    double vol[W == 1 ? 32 : 1][6];
    double out[W][12];
    int listed, next;
};

// The listed faces by groups of W warps.  W > 1: eight lanes per candidate for
// its seven volumes, the candidates dealt over the warps first.  W = 1: a lane
// per candidate for its volume, then a lane per volume for the six of those
// that overlap.
template <int W>
__device__ __forceinline__ void steric_faces(const StericArgs &a, StericGroup<W> *groups, int nwork,
                                             unsigned long long &npairs)
{
    constexpr int G = kStericWarps / W;  // groups of the CTA
    const int lane = threadIdx.x & 31, gi = (threadIdx.x >> 5) / W, wi = (threadIdx.x >> 5) % W;
    StericGroup<W> &s = groups[gi];
    auto sync = [&] {
        if constexpr (W == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + gi), "n"(32 * W) : "memory");
    };
    int w = blockIdx.x + gridDim.x * gi;
#pragma unroll 1
    while (w < nwork) {
        const int i = a.work[w];
        double out[4][3];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int d = 0; d < 3; d++) out[u][d] = 0.0;
        if (wi == 0 && lane == 0) {
            s.listed = 0;
            s.next = gridDim.x * G + (int)atomicAdd(&a.stats[6], 1ull);
        }
        steric_candidates<W>(a, i, wi, lane, s.q, s.beg, s.pre, s.cnt, sync, [&](int n) {
            if constexpr (W > 1) {
                const int g = lane & ~7, v = lane & 7;  // the pair's first lane, and the volume this lane takes
#pragma unroll 1
                for (int q0 = wi; q0 < n; q0 += 4 * W) {
                    const int q = q0 + W * (lane >> 3);
                    const int j = q < n ? s.q[q] : -1;
                    double cm[3] = {0.0, 0.0, 0.0}, V = 0.0;
                    if (j >= 0 && v < 7) V = pair_overlap(a, i, j, v, v == 0 ? cm : nullptr);
                    double va[3], vb[3];
#pragma unroll
                    for (int d = 0; d < 3; d++) {
                        vb[d] = __shfl_sync(0xffffffffu, V, g + 1 + d);
                        va[d] = __shfl_sync(0xffffffffu, V, g + 4 + d);
                    }
                    if (v == 0 && V != 0) add_steric_pair(a, i, j, V, cm, vb, va, atomicAdd(&s.listed, 1), out, npairs);
                }
            } else {
#pragma unroll 1
                for (int q0 = 0; q0 < n; q0 += 32) {
                    const int j = q0 + lane < n ? s.q[q0 + lane] : -1;
                    double cm[3] = {0.0, 0.0, 0.0}, V = 0.0;
                    if (j >= 0) V = pair_overlap(a, i, j, 0, cm);
                    const unsigned hits = __ballot_sync(0xffffffffu, V != 0);
                    const int m = __popc(hits), rank = __popc(hits & ((1u << lane) - 1u)), listed = s.listed;
                    if (V != 0) s.hit[rank] = j;
                    __syncwarp();
#pragma unroll 1
                    for (int t = lane; t < 6 * m; t += 32)
                        s.vol[t / 6][t % 6] = pair_overlap(a, i, s.hit[t / 6], 1 + t % 6, nullptr);
                    __syncwarp();
                    if (V != 0) add_steric_pair(a, i, j, V, cm, s.vol[rank], s.vol[rank] + 3, listed + rank, out, npairs);
                    if (lane == 0) s.listed = listed + m;
                    __syncwarp();  // hit, vol and listed free
                }
            }
        });
        const double sum = warp_sum12(out, lane);
        if ((lane & 1) == 0 && lane < 24) s.out[wi][lane / 2] = sum;
        sync();
        if (wi == 0) {
            if (lane == 0) {
                a.stcnt[i] = min(s.listed, FFEA_GPU_SSINT_MAX_STERIC_PARTNERS);
                if (s.listed > FFEA_GPU_SSINT_MAX_STERIC_PARTNERS) atomicAdd(&a.stats[4], 1ull);
            }
            if (lane < 12) {
                double t = 0.0;
#pragma unroll
                for (int k = 0; k < W; k++) t += s.out[k][lane];
                a.fforce[12 * (long long)i + lane] = t;
            }
        }
        w = s.next;
        sync();  // the group's shared memory free
    }
}

__global__ void __launch_bounds__(32 * kStericWarps, 1) k_steric(const __grid_constant__ StericArgs a)
{
    __shared__ union Shared {
        StericGroup<8> g8[kStericWarps / 8];
        StericGroup<4> g4[kStericWarps / 4];
        StericGroup<1> g1[kStericWarps];
    } s;
    if (a.stats[3]) return;  // the call fails (a cell too full to sort)
    const int n = (int)a.stats[5];
    unsigned long long npairs = 0;
    // (the lines: above)
    if (n <= a.sms) steric_faces<8>(a, s.g8, n, npairs);
    else if (n <= 3 * a.sms) steric_faces<4>(a, s.g4, n, npairs);
    else steric_faces<1>(a, s.g1, n, npairs);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    if ((threadIdx.x & 31) == 0 && npairs) atomicAdd(&a.stats[0], npairs);
}

// One warp per face i (faces taken in cell order): the candidates of the 27
// cells around i's cell are numbered 0..total-1 through a prefix sum over the
// cells, lane l tests candidates l, l + 32, ..., and the partners that pass
// are evaluated from a per-warp queue.  Each lane keeps face i's side of its
// pairs; a fixed shuffle tree sums the lanes.  POT: Lennard-Jones or the soft
// potential; STERIC: the steric types' pair checks apply, the partners of i's
// steric list are skipped (k_steric gave them the steric force) and the
// forces add to what k_steric wrote.
template <int POT, bool STERIC>
__global__ void __launch_bounds__(32 * kPairWarps, kPairCtas) k_pairs(
    const double *__restrict__ gp, const float4 *__restrict__ nb, const int *__restrict__ cell,
    const int *__restrict__ sorted, const int *__restrict__ start, const int *__restrict__ block, long long ncell,
    int nblocks, int nx, int ny, int nz, const int *__restrict__ fblob, const int *__restrict__ ftype,
    const double *__restrict__ emin,
    const double *__restrict__ rmin, const double *__restrict__ k0, const int *__restrict__ corner,
    const int *__restrict__ stlist, const int *__restrict__ stcnt, int num_types, int num_blobs, int inc_self,
    const double *__restrict__ corr, double *__restrict__ fforce, double *__restrict__ energy,
    unsigned long long *stats)
{
    __shared__ int s_pre[kPairWarps][28];
    __shared__ int s_beg[kPairWarps][27];
    __shared__ int s_q[kPairWarps][64];
    __shared__ int s_st[kPairWarps][FFEA_GPU_SSINT_MAX_STERIC_PARTNERS];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * kPairWarps + wi;
    if (w >= block[nblocks]) return;  // warp-uniform; faces outside the box are not binned
    if (stats[3]) return;             // a cell too full to sort: the call fails, nothing to evaluate
    const int i = sorted[w];
    const int total = warp_cells(cell[i], nx, ny, nz, start, block, ncell, nblocks, lane, s_beg[wi], s_pre[wi]);
    int nst = 0;
    int ni[4] = {0, 0, 0, 0};
    if constexpr (STERIC) {
        nst = stcnt[i];
        if (lane < nst) s_st[wi][lane] = stlist[FFEA_GPU_SSINT_MAX_STERIC_PARTNERS * i + lane];
#pragma unroll
        for (int u = 0; u < 4; u++) ni[u] = corner[4 * i + u];
        __syncwarp();
    }
    const double *A = gp + 16 * (long long)i;
    const float4 nbi = nb[i];
    double own[9];
#pragma unroll
    for (int k = 0; k < 9; k++) own[k] = A[k];
    const double area = A[12];
    const int bi = fblob[i], ti = ftype[i];
    double S[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};  // the lane's sum of area products * column sums
    double e_acc = 0.0;
    int e_key = -1;
    unsigned long long npairs = 0;
    // one partner j: face i's side of the pair, FFEA's f1 being the lower index
    auto pair = [&](int j) {
        const double2 *G = reinterpret_cast<const double2 *>(gp + 16 * (long long)j);
        double oth[10];
#pragma unroll
        for (int q = 0; q < 5; q++) {
            const double2 g2 = __ldg(G + q);
            oth[2 * q] = g2.x;
            oth[2 * q + 1] = g2.y;
        }
        const double apaq = area * __ldg(gp + 16 * (long long)j + 12);
        const int bj = fblob[j];
        const bool lower = i < j;
        double q[9];
#pragma unroll
        for (int c = 0; c < 9; c++) q[c] = oth[c];
        if (corr) {
            // periodic: f1's points minus blob_corr[b2][b1]
            // (Face::barycentric_calc_point_f2, src/Face.cpp:271-277), as a
            // shift of the partner's points seen from either side
            const double *c = corr + 3 * (lower ? (long long)bj * num_blobs + bi : (long long)bi * num_blobs + bj);
#pragma unroll
            for (int k = 0; k < 9; k++) q[k] += lower ? c[k % 3] : -c[k % 3];
        }
        const int tt = lower ? ti * num_types + ftype[j] : ftype[j] * num_types + ti;
        const double en = pot_pair<POT>(own, q, apaq, lower, emin[tt], rmin[tt], k0 ? k0[tt] : 0.0, S);
        if (lower) {
            const int key = bi * num_blobs + bj;
            if (key != e_key) {
                if (e_key >= 0) atomicAdd(&energy[e_key], e_acc);
                e_key = key;
                e_acc = 0.0;
            }
            e_acc += en;
            npairs++;
        }
    };
    // The cheap tests (same face, same blob, normals facing the same way) run
    // over all candidates; the partners that pass are queued in shared memory
    // and evaluated 32 at a time, so every lane of the FP64 pair arithmetic
    // does useful work.
    int qn = 0;  // warp-uniform queue length, < 64
    for (int base = 0; base < total; base += 32) {
        const int k = base + lane;
        bool ok = false;
        int j = -1;
        if (k < total) {
            j = warp_candidate(k, s_beg[wi], s_pre[wi], sorted);
            ok = admits(i, j, nbi, nb, gp, inc_self);
            if constexpr (STERIC) {
                if (ok) {
                    int nj[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) nj[u] = corner[4 * j + u];
                    ok = steric_type_ok(A, gp + 16 * (long long)j, bi == fblob[j], inc_self, ni, nj,
                                        corr ? corr + 3 * ((long long)bi * num_blobs + fblob[j]) : nullptr);
                }
                for (int t = 0; ok && t < nst; t++)
                    if (s_st[wi][t] == j) ok = false;  // the steric force applied instead
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (ok) s_q[wi][qn + __popc(m & ((1u << lane) - 1u))] = j;
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
            pair(s_q[wi][lane]);
            const int rest = qn - 32;
            const int moved = lane < rest ? s_q[wi][32 + lane] : 0;
            __syncwarp();
            if (lane < rest) s_q[wi][lane] = moved;
            qn = rest;
            __syncwarp();
        }
    }
    if (lane < qn) pair(s_q[wi][lane]);
    // energy: one atomic per distinct (blob, blob) key left in the warp
    for (;;) {
        const unsigned pending = __ballot_sync(0xffffffffu, e_key >= 0);
        if (!pending) break;
        const int lk = __shfl_sync(0xffffffffu, e_key, __ffs(pending) - 1);
        const double part = warp_sum_d(e_key == lk ? e_acc : 0.0);
        if (lane == 0) atomicAdd(&energy[lk], part);
        if (e_key == lk) e_key = -1;
    }
    // the lanes' sums: nine values by a transposed butterfly (at offsets 16,
    // 8, 4 and 2 a lane keeps half of its values: 16 additions, not 45); the
    // total of value v ends in lanes 2 v and 2 v + 1
    {
        double v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = k < 9 ? S[k / 3][k % 3] : 0.0;
#pragma unroll
        for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < h; k++) {
                const double send = upper ? v[k] : v[k + h], keep = upper ? v[k + h] : v[k];
                v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
#pragma unroll
        for (int k = 0; k < 9; k++) S[k / 3][k % 3] = __shfl_sync(0xffffffffu, v[0], 2 * k);
    }
    unsigned long long np = npairs;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
    if (lane == 0 && np) atomicAdd(&stats[0], np);
    if (lane < 12) {
        const int c = lane / 3, d = lane % 3;
        double f = 0.0;
        if (c < 3)
#pragma unroll
            for (int l = 0; l < 3; l++) {
                const double sl = d == 0 ? S[l][0] : d == 1 ? S[l][1] : S[l][2];
                f = fma(kW * kW * (l == c ? eta(0, 0) : eta(0, 1)), sl, f);
            }
        double *o = &fforce[12 * (long long)i + lane];
        *o = STERIC ? *o + f : f;
    }
}

// The sticky xz walls (VdW_solver::solve_sticky_wall / do_sticky_xz_interaction,
// src/VdW_solver.cpp:216-235, 396-456), after the pair pass: every face whose
// cell lies in the grid's bottom (y = 0) or top (y = ny - 1) row and faces
// that wall feels a y force from it, the Lennard-Jones factor of its own type
// at the height of its Gauss points, added to its corners (the energy is not
// recorded, as in FFEA).  One thread per face.
__global__ void k_sticky(const double *__restrict__ geo, const int *__restrict__ cell, int na,
                         const int *__restrict__ ftype, const double *__restrict__ emin,
                         const double *__restrict__ rmin, int num_types, int ny, int nz, double h,
                         double *__restrict__ fforce)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= na || cell[i] < 0) return;
    const int cy = (cell[i] / nz) % ny;
    if (cy != 0 && cy != ny - 1) return;
    const bool bottom = cy == 0;
    const double *g = geo + 16 * (long long)i;
    if ((bottom && g[10] > 0) || (!bottom && g[10] < 0)) return;
    const double y_wall = bottom ? 0.0 : h * ny;
    const int tt = ftype[i] * num_types + ftype[i];
    const double r6 = pow(rmin[tt], 6.0), em = emin[tt];
    double py[3], fm[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        py[k] = eta(k, 0) * g[1] + eta(k, 1) * g[4] + eta(k, 2) * g[7];
        const double r = py[k] - y_wall;
        fm[k] = -(12 * r6 * em * (pow(r, -7.0) - r6 * pow(r, -13.0)));
    }
    const double asq = g[12] * g[12];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        double fy = 0.0;
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int l = 0; l < 3; l++) fy += kW * kW * eta(l, j) * fm[k < l ? k : l];
        fforce[12 * (long long)i + 3 * j + 1] += fy * asq;
    }
}

__global__ void k_node_gather(const int *__restrict__ ptr, const int *__restrict__ ent, int nn,
                              const double *__restrict__ fforce, const int *__restrict__ cell,
                              double *__restrict__ force)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double f[3] = {0.0, 0.0, 0.0};
    for (int k = ptr[n]; k < ptr[n + 1]; k++) {
        const int fc = ent[k];
        if (cell[fc / 4] < 0) continue;
#pragma unroll
        for (int d = 0; d < 3; d++) f[d] += fforce[3 * (long long)fc + d];
    }
#pragma unroll
    for (int d = 0; d < 3; d++) force[3 * (long long)n + d] = f[d];
}

template <class T>
int dalloc(T **p, size_t n)
{
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (n ? n : 1));
    if (e != cudaSuccess) return fail("cudaMalloc of %zu bytes: %s", sizeof(T) * n, cudaGetErrorString(e));
    return FFEA_GPU_OK;
}

}  // namespace

extern "C" int ffea_gpu_ssint_create(const ffea_gpu_ssint_desc *d, ffea_gpu_ssint_t **out)
{
    if (!d || !out) return fail("ffea_gpu_ssint_create: null argument");
    *out = nullptr;
    if (d->num_nodes < 0 || d->num_faces < 0 || d->num_types <= 0 || d->num_blobs <= 0)
        return fail("ffea_gpu_ssint_create: negative sizes, or no types or blobs");
    if ((d->num_faces && (!d->faces || !d->face_blob || !d->face_type)) || !d->emin || !d->rmin)
        return fail("ffea_gpu_ssint_create: null array");
    if (!(d->cell_size > 0.0)) return fail("ffea_gpu_ssint_create: cell_size must be positive");
    if (d->nx <= 0 || d->ny <= 0 || d->nz <= 0) return fail("ffea_gpu_ssint_create: grid dimensions must be positive");
    const long long ncell = (long long)d->nx * d->ny * d->nz;
    if (ncell > FFEA_GPU_SSINT_MAX_CELLS)
        return fail("ffea_gpu_ssint_create: %lld cells exceed the maximum %d", ncell, FFEA_GPU_SSINT_MAX_CELLS);
    const int stype = d->ssint_type;
    if (stype < FFEA_GPU_SSINT_LJ || stype > FFEA_GPU_SSINT_GENSOFT) return fail("unknown ssint_type %d", stype);
    const bool steric = stype != FFEA_GPU_SSINT_LJ;
    if (steric && d->num_faces && !d->face_apex) return fail("the steric types need face_apex (Face::n[3] per face)");
    if (steric && !(d->steric_dr > 0.0)) return fail("steric_dr must be positive");
    if (stype == FFEA_GPU_SSINT_GENSOFT && !d->k0) return fail("gensoft needs k0");
    std::vector<int> corner, blob, type;
    for (int f = 0; f < d->num_faces; f++) {
        if (d->face_type[f] < 0) continue;  // not ssint-active: not in the pool (src/Blob.cpp:1642-1648)
        if (d->face_type[f] >= d->num_types) return fail("face %d: interaction type %d >= num_types", f, d->face_type[f]);
        if (d->face_blob[f] < 0 || d->face_blob[f] >= d->num_blobs) return fail("face %d: blob %d out of range", f, d->face_blob[f]);
        for (int k = 0; k < 4; k++) {
            const int n = k < 3 ? d->faces[3 * f + k] : (steric ? d->face_apex[f] : -1);
            if (n < -1 || n >= d->num_nodes || (n < 0 && k < 3) || (n < 0 && steric))
                return fail("face %d: node %d out of range", f, n);
            corner.push_back(n);
        }
        blob.push_back(d->face_blob[f]);
        type.push_back(d->face_type[f]);
    }
    const int na = (int)blob.size();
    // node -> (active face, node of the face) entries in face order (the
    // fourth node only for the steric types)
    std::vector<int> ptr(d->num_nodes + 1, 0), ent;
    for (int i = 0; i < 4 * na; i++)
        if (corner[i] >= 0) ptr[corner[i] + 1]++;
    for (int n = 0; n < d->num_nodes; n++) ptr[n + 1] += ptr[n];
    ent.resize((size_t)ptr[d->num_nodes]);
    {
        std::vector<int> fill(ptr.begin(), ptr.end() - 1);
        for (int i = 0; i < 4 * na; i++)
            if (corner[i] >= 0) ent[fill[corner[i]]++] = i;
    }
    auto *s = new ffea_gpu_ssint();
    s->num_nodes = d->num_nodes;
    s->num_faces = d->num_faces;
    s->num_active = na;
    s->num_types = d->num_types;
    s->num_blobs = d->num_blobs;
    s->nx = d->nx;
    s->ny = d->ny;
    s->nz = d->nz;
    s->inc_self = d->inc_self ? 1 : 0;
    s->type = stype;
    s->steric_factor = d->steric_factor;
    s->steric_dr = d->steric_dr;
    s->h = d->cell_size;
    s->ncell = ncell;
    s->nblocks = (int)((ncell + kScanBlock - 1) / kScanBlock);
    const int T2 = d->num_types * d->num_types;
    int rc = FFEA_GPU_OK;
    auto run = [&]() -> int {
        // blocking: its kernels must follow the uploads below, which run on
        // the legacy default stream and may still be in flight when
        // cudaMemcpy returns
        SSINT_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamDefault));
        int dev = 0;
        SSINT_CUDA(cudaGetDevice(&dev));
        SSINT_CUDA(cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, dev));
        if (dalloc(&s->d_corner, 4 * (size_t)na) || dalloc(&s->d_blob, na) || dalloc(&s->d_type, na) ||
            dalloc(&s->d_geo, 16 * (size_t)na) || dalloc(&s->d_gp, 16 * (size_t)na) || dalloc(&s->d_nb, na) || dalloc(&s->d_cell, na) || dalloc(&s->d_fforce, 12 * (size_t)na) ||
            dalloc(&s->d_count, ncell) || dalloc(&s->d_start, ncell) || dalloc(&s->d_block, s->nblocks + 1) ||
            dalloc(&s->d_binned, na) || dalloc(&s->d_sorted, na) || dalloc(&s->d_node_ptr, d->num_nodes + 1) ||
            dalloc(&s->d_node_ent, ent.size()) || dalloc(&s->d_emin, T2) || dalloc(&s->d_rmin, T2) ||
            dalloc(&s->d_pos, 3 * (size_t)d->num_nodes) || dalloc(&s->d_force, 3 * (size_t)d->num_nodes) ||
            dalloc(&s->d_energy, (size_t)d->num_blobs * d->num_blobs) || dalloc(&s->d_stats, kStats) ||
            dalloc(&s->d_large, (size_t)na / (kSortSmall + 1) + 1))
            return FFEA_GPU_ERROR;
        if (steric && (dalloc(&s->d_stlist, (size_t)FFEA_GPU_SSINT_MAX_STERIC_PARTNERS * na) ||
                       dalloc(&s->d_stcnt, na) || dalloc(&s->d_stwork, na) || dalloc(&s->d_box, 2 * (size_t)na)))
            return FFEA_GPU_ERROR;
        if (stype == FFEA_GPU_SSINT_GENSOFT && dalloc(&s->d_k0, T2)) return FFEA_GPU_ERROR;
        if (na) {
            SSINT_CUDA(cudaMemcpy(s->d_corner, corner.data(), sizeof(int) * 4 * na, cudaMemcpyHostToDevice));
            SSINT_CUDA(cudaMemcpy(s->d_blob, blob.data(), sizeof(int) * na, cudaMemcpyHostToDevice));
            SSINT_CUDA(cudaMemcpy(s->d_type, type.data(), sizeof(int) * na, cudaMemcpyHostToDevice));
        }
        if (!ent.empty())
            SSINT_CUDA(cudaMemcpy(s->d_node_ent, ent.data(), sizeof(int) * ent.size(), cudaMemcpyHostToDevice));
        SSINT_CUDA(cudaMemcpy(s->d_node_ptr, ptr.data(), sizeof(int) * (d->num_nodes + 1), cudaMemcpyHostToDevice));
        SSINT_CUDA(cudaMemcpy(s->d_emin, d->emin, sizeof(double) * T2, cudaMemcpyHostToDevice));
        SSINT_CUDA(cudaMemcpy(s->d_rmin, d->rmin, sizeof(double) * T2, cudaMemcpyHostToDevice));
        if (s->d_k0) SSINT_CUDA(cudaMemcpy(s->d_k0, d->k0, sizeof(double) * T2, cudaMemcpyHostToDevice));
        return FFEA_GPU_OK;
    };
    rc = run();
    if (rc != FFEA_GPU_OK) {
        ffea_gpu_ssint_destroy(s);
        return rc;
    }
    *out = s;
    return FFEA_GPU_OK;
}

extern "C" void ffea_gpu_ssint_destroy(ffea_gpu_ssint_t *s)
{
    if (!s) return;
    if (s->stream) cudaStreamSynchronize(s->stream);
    void *bufs[] = {s->d_corner, s->d_blob, s->d_type, s->d_geo, s->d_gp, s->d_nb, s->d_box, s->d_cell, s->d_fforce,
                    s->d_count, s->d_start, s->d_block, s->d_binned, s->d_sorted, s->d_node_ptr, s->d_node_ent, s->d_emin, s->d_rmin,
                    s->d_pos, s->d_force, s->d_energy, s->d_stats, s->d_large, s->d_stlist, s->d_stcnt, s->d_stwork, s->d_k0,
                    s->d_corr};
    for (void *p : bufs)
        if (p) cudaFree(p);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

extern "C" void *ffea_gpu_ssint_stream(ffea_gpu_ssint_t *s) { return s ? (void *)s->stream : nullptr; }

extern "C" int ffea_gpu_ssint_forces_device(ffea_gpu_ssint_t *s, const double *pos, double *force, double *energy)
{
    if (!s || !pos || !force || !energy) return fail("ffea_gpu_ssint_forces_device: null argument");
    cudaStream_t st = s->stream;
    const int na = s->num_active;
    SSINT_CUDA(cudaMemsetAsync(energy, 0, sizeof(double) * s->num_blobs * s->num_blobs, st));
    SSINT_CUDA(cudaMemsetAsync(s->d_stats, 0, sizeof(unsigned long long) * kStats, st));
    if (na == 0) {
        SSINT_CUDA(cudaMemsetAsync(force, 0, sizeof(double) * 3 * (size_t)s->num_nodes, st));
        return FFEA_GPU_OK;
    }
    SSINT_CUDA(cudaMemsetAsync(s->d_count, 0, sizeof(int) * s->ncell, st));
    const int fb = (na + 127) / 128;
    k_face_geom<<<fb, 128, 0, st>>>(pos, s->d_corner, na, s->h, s->nx, s->ny, s->nz, s->d_blob, s->d_geo,
                                    s->d_gp, s->d_nb, s->d_box, s->d_cell, s->d_count, s->d_stats);
    k_scan_local<<<s->nblocks, kScanBlock, 0, st>>>(s->d_count, s->ncell, s->d_start, s->d_block);
    k_scan_blocks<<<1, kScanBlock, 0, st>>>(s->d_block, s->nblocks);
    k_scatter<<<fb, 128, 0, st>>>(s->d_cell, na, s->d_start, s->d_block, s->d_count, s->d_binned);
    // faces outside the box are left out of the grid (and make the call an
    // error); the kernels below bound every segment by the scan's total
    k_sort_cells<<<fb, 128, 0, st>>>(s->ncell, s->nblocks, s->d_start, s->d_block, s->d_cell, s->d_binned,
                                     s->d_sorted, s->d_large, s->d_stats);
    k_sort_large<<<kSortLargeCtas, 256, 0, st>>>(s->ncell, s->nblocks, s->d_start, s->d_block, s->d_sorted,
                                                 s->d_large, s->d_stats);
    const int pw = (na + kPairWarps - 1) / kPairWarps;
    if (s->type != FFEA_GPU_SSINT_LJ) {
        const double *corr = s->has_corr ? s->d_corr : nullptr;
        k_steric_find<<<(na + kFindWarps - 1) / kFindWarps, 32 * kFindWarps, 0, st>>>(
            s->d_geo, s->d_gp, s->d_nb, s->d_box, s->d_sorted, s->d_cell, s->d_start, s->d_block, s->ncell,
            s->nblocks, s->nx, s->ny, s->nz, s->d_blob, s->d_corner, s->num_blobs, s->inc_self, corr, s->d_fforce,
            s->d_stlist, s->d_stcnt, s->d_stwork, s->d_stats);
        const StericArgs args{s->d_geo,    s->d_gp,  s->d_nb,      s->d_sorted, s->d_cell,        s->d_start,
                              s->d_block,  s->ncell, s->nblocks,   s->nx,       s->ny,            s->nz,
                              s->d_blob,   s->d_corner, s->num_blobs, s->inc_self, s->steric_factor, s->steric_dr,
                              corr,        s->d_fforce, s->d_stlist,  s->d_stcnt,  s->d_stwork,      s->sms,
                              energy,      s->d_stats};
        // as many CTAs as run at a time: each takes listed faces until none is left
        k_steric<<<std::min(na, s->sms), 32 * kStericWarps, 0, st>>>(args);
    }
#define SSINT_PAIRS(POT, STERIC)                                                                                   \
    k_pairs<POT, STERIC><<<pw, 32 * kPairWarps, 0, st>>>(                                                           \
        s->d_gp, s->d_nb, s->d_cell, s->d_sorted, s->d_start, s->d_block, s->ncell, s->nblocks, s->nx, s->ny, s->nz, \
        s->d_blob, s->d_type, s->d_emin, s->d_rmin, s->d_k0, s->d_corner, s->d_stlist, s->d_stcnt, s->num_types,     \
        s->num_blobs, s->inc_self, s->has_corr ? s->d_corr : nullptr, s->d_fforce, energy, s->d_stats)
    if (s->type == FFEA_GPU_SSINT_LJ) SSINT_PAIRS(POT_LJ, false);
    else if (s->type == FFEA_GPU_SSINT_LJSTERIC) SSINT_PAIRS(POT_LJ, true);
    else if (s->type == FFEA_GPU_SSINT_GENSOFT) SSINT_PAIRS(POT_SOFT, true);
#undef SSINT_PAIRS
    if (s->sticky)
        k_sticky<<<fb, 128, 0, st>>>(s->d_geo, s->d_cell, na, s->d_type, s->d_emin, s->d_rmin, s->num_types, s->ny,
                                     s->nz, s->h, s->d_fforce);
    k_node_gather<<<(s->num_nodes + 255) / 256, 256, 0, st>>>(s->d_node_ptr, s->d_node_ent, s->num_nodes,
                                                              s->d_fforce, s->d_cell, force);
    SSINT_CUDA(cudaGetLastError());
    return FFEA_GPU_OK;
}

extern "C" int ffea_gpu_ssint_set_pbc(ffea_gpu_ssint_t *s, const double *blob_corr)
{
    if (!s) return fail("ffea_gpu_ssint_set_pbc: null handle");
    if (!blob_corr) {
        s->has_corr = 0;
        return FFEA_GPU_OK;
    }
    const size_t n = 3 * (size_t)s->num_blobs * s->num_blobs;
    if (!s->d_corr) SSINT_CUDA(cudaMalloc(&s->d_corr, sizeof(double) * n));
    // ordered on the handle's stream before the next pass
    SSINT_CUDA(cudaMemcpyAsync(s->d_corr, blob_corr, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream));
    SSINT_CUDA(cudaStreamSynchronize(s->stream));
    s->has_corr = 1;
    return FFEA_GPU_OK;
}

extern "C" int ffea_gpu_ssint_set_sticky_wall(ffea_gpu_ssint_t *s, int32_t enable)
{
    if (!s) return fail("ffea_gpu_ssint_set_sticky_wall: null handle");
    if (enable && s->ny < 2)
        return fail("the sticky wall needs at least two rows of cells in y (FFEA's row loop would not end)");
    s->sticky = enable ? 1 : 0;
    return FFEA_GPU_OK;
}

extern "C" int ffea_gpu_ssint_blob_corr(int32_t num_blobs, const double *centroids, const double box[3],
                                        double *blob_corr)
{
    if (num_blobs < 0 || (num_blobs > 0 && (!centroids || !box || !blob_corr)))
        return fail("ffea_gpu_ssint_blob_corr: null argument");
    for (int i = 0; i < num_blobs; ++i) {
        for (int d = 0; d < 3; d++) blob_corr[3 * ((size_t)i * num_blobs + i) + d] = 0.0;
        for (int j = i + 1; j < num_blobs; ++j)
            for (int d = 0; d < 3; d++) {
                const double v = box[d] * floor((centroids[3 * j + d] - centroids[3 * i + d] + 0.5 * box[d]) / box[d]);
                blob_corr[3 * ((size_t)i * num_blobs + j) + d] = v;
                blob_corr[3 * ((size_t)j * num_blobs + i) + d] = -1 * v;
            }
    }
    return FFEA_GPU_OK;
}

extern "C" int ffea_gpu_ssint_synchronize(ffea_gpu_ssint_t *s, int64_t *pairs)
{
    if (!s) return fail("ffea_gpu_ssint_synchronize: null handle");
    unsigned long long st[kStats] = {};
    SSINT_CUDA(cudaMemcpyAsync(st, s->d_stats, sizeof(st), cudaMemcpyDeviceToHost, s->stream));
    SSINT_CUDA(cudaStreamSynchronize(s->stream));
    if (pairs) *pairs = (int64_t)st[0];
    if (st[1]) return fail("%llu face centroids lie outside the interaction grid (FFEA reports this as an error)", st[1]);
    if (st[3])
        return fail("%llu grid cells hold more than %d faces each: the interaction grid is too coarse for this mesh "
                    "(use more, smaller cells)", st[3], kSortMax);
    if (st[4])
        return fail("%llu faces' tetrahedra overlap more than %d others (their steric partners beyond that are "
                    "not excluded from the Lennard-Jones or soft pairs)", st[4], FFEA_GPU_SSINT_MAX_STERIC_PARTNERS);
    return FFEA_GPU_OK;
}

extern "C" int ffea_gpu_ssint_forces(ffea_gpu_ssint_t *s, const double *pos, double *force, double *energy,
                                     int64_t *pairs)
{
    if (!s || !pos || !force || !energy) return fail("ffea_gpu_ssint_forces: null argument");
    const size_t nb = sizeof(double) * 3 * (size_t)s->num_nodes;
    SSINT_CUDA(cudaMemcpyAsync(s->d_pos, pos, nb, cudaMemcpyHostToDevice, s->stream));
    if (ffea_gpu_ssint_forces_device(s, s->d_pos, s->d_force, s->d_energy)) return FFEA_GPU_ERROR;
    SSINT_CUDA(cudaMemcpyAsync(force, s->d_force, nb, cudaMemcpyDeviceToHost, s->stream));
    SSINT_CUDA(cudaMemcpyAsync(energy, s->d_energy, sizeof(double) * s->num_blobs * s->num_blobs,
                               cudaMemcpyDeviceToHost, s->stream));
    return ffea_gpu_ssint_synchronize(s, pairs);
}
