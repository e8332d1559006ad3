// cg_group.cu -- the CG solve of blobs that fit on chip.
//
// One persistent cooperative launch solves every blob of a batch to
// convergence.  A blob's CG segments (at most CG_SEG_MAX_ROWS rows each) are
// its group of CTAs, a segment to each, or two in a batch with a blob of more
// segments than CTAs.  Groups are independent: each exchanges only among its
// own CTAs and stops when its own blob has converged, and a CTA then goes on
// to the next task (its one or two segments of a blob) of its list.  Every
// CTA's list follows one order of the blobs, so a group's CTAs wait for each
// other without a cycle.
//
// The recurrences, the stopping rule and the order of every FP32 sum are
// those of the memory-resident solve (k_cg in kernels.cu): Jacobi- or
// two-level-PCG in the Chronopoulos-Gear form, one product and one group of
// sums per iteration.
//
// What bounds an iteration is the latency of its two exchanges and of the
// instructions between them and, for full segments, the L2 reads of the
// matrix.  So nothing waits on a barrier word:
//   - u is published row by row as one 128-bit store (x, y, z, tag); a CTA
//     reads the rows its segment couples to (its halo, each row once) until
//     their tags are the iteration's, into shared memory beside its own rows,
//     and the product's inner loop reads shared memory alone;
//   - a segment's partial sums are published the same way, and every CTA of
//     the group reads all of them: a few warps wait for the dot terms, and the
//     coarse restrictions are read once those are in, while the CG transition
//     runs.
// Two things decide the time of an exchange (152 CTAs, alone, in thousand
// cycles): words of one CTA leave in whole 32-byte sectors (2.0; stored 16
// bytes at a time into sectors that others are reading, 7 to 9), and few
// threads wait (with one in every thread 4.5: their reads hold up the stores
// they wait for).  A counter that all CTAs add to took 3.6.
// The tag travels in the same single-copy-atomic word as the value, so no
// fence, no counter and no second round trip is needed.  A row of u is
// rewritten only after its CTA has read the group's sums of the iteration,
// which every CTA publishes after its last read of u; the sums alternate
// between two buffers for the same reason.  Tags never repeat from one launch
// to the next (the base in bar[6] grows by the tags a launch used).
// A wait ends with its tag or, when no solve of the grid gets on any more,
// with a time-out (check_wait): the CTA then fails the blobs of all tasks it
// has left, and returns.
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_common.cuh"
#include "kernels.h"
#include "mrg32k3a.cuh"

namespace ffea {

namespace {

extern __shared__ __align__(16) unsigned char grp_dyn[];

template <typename X>
__device__ __forceinline__ X *dyn(int32_t off)
{
    return reinterpret_cast<X *>(grp_dyn + off);
}

// ---------------------------------------------------------------- tagged words
__device__ __forceinline__ void st_b128(void *p, uint64_t lo, uint64_t hi)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi)
                 : "memory");
}
__device__ __forceinline__ void ld_b128(const void *p, uint64_t &lo, uint64_t &hi)
{
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p));
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) { return (uint64_t)hi << 32 | lo; }

// A published row: x, y, z and the tag, in one 128-bit word (FP32), or each
// component with the tag in its own plane of n words (FP64: neighbouring rows
// then store whole sectors).
template <typename T> struct PubRow;
template <> struct PubRow<float> {
    float x, y, z;
    uint32_t tag;
    static __device__ __forceinline__ void put(uint4 *base, int, int row, const float v[3], uint32_t tag)
    {
        st_b128(base + row, pack2(__float_as_uint(v[0]), __float_as_uint(v[1])), pack2(__float_as_uint(v[2]), tag));
    }
    __device__ __forceinline__ void get(const uint4 *base, int, int row)
    {
        uint64_t lo, hi;
        ld_b128(base + row, lo, hi);
        x = __uint_as_float((uint32_t)lo);
        y = __uint_as_float((uint32_t)(lo >> 32));
        z = __uint_as_float((uint32_t)hi);
        tag = (uint32_t)(hi >> 32);
    }
    __device__ __forceinline__ bool is(uint32_t t) const { return tag == t; }
};
template <> struct PubRow<double> {
    double x, y, z;
    uint32_t tag, tag1, tag2;
    static __device__ __forceinline__ void put(uint4 *base, int n, int row, const double v[3], uint32_t tag)
    {
#pragma unroll
        for (int k = 0; k < 3; k++) st_b128(base + (size_t)k * n + row, (uint64_t)__double_as_longlong(v[k]), tag);
    }
    __device__ __forceinline__ void get(const uint4 *base, int n, int row)
    {
        uint64_t a, b, c, ta, tb, tc;
        ld_b128(base + row, a, ta);
        ld_b128(base + (size_t)n + row, b, tb);
        ld_b128(base + 2 * (size_t)n + row, c, tc);
        x = __longlong_as_double((long long)a);
        y = __longlong_as_double((long long)b);
        z = __longlong_as_double((long long)c);
        tag = (uint32_t)ta;
        tag1 = (uint32_t)tb;
        tag2 = (uint32_t)tc;
    }
    __device__ __forceinline__ bool is(uint32_t t) const { return tag == t && tag1 == t && tag2 == t; }
};

// A read of a matrix that is larger than L2, which an iteration reads once:
// evicted first, but for a tenth of it, so that it does not displace what
// else the iteration reads (50 nm sphere, 138 MB of matrix: 47.1 us an
// iteration with plain reads, 36.1 with all of it evicted first, 35.7 with a
// tenth kept, 37.4 with three tenths).
__device__ __forceinline__ uint64_t stream_policy()
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.L2::evict_first.b64 %0, %1;" : "=l"(pol) : "f"(0.1f));
    return pol;
}
__device__ __forceinline__ float ld_stream(const float *p, uint64_t pol)
{
    float v;
    asm volatile("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ double ld_stream(const double *p, uint64_t) { return __ldg(p); }

// The bounds of a wait: the published sums of all n segments, the reads after
// which they are looked at, and the flags of a wait that ran out.
struct WaitBound {
    const uint4 *words;
    int n;
    unsigned int limit;
    volatile int *s_err;
    unsigned int *bar;
};

// Whether a wait goes on.  It is given up when another wait of the CTA or of
// the grid has run out (bar[4]), or when no solve of the grid has got on in
// GroupBatch::spin_limit reads; a wait that runs out raises both flags.  The
// CTAs waited for may still be solving the blobs before this one, for as long
// as those take: the tags of the dot terms, which every exchange of every
// segment moves up, tell whether anything does.
constexpr unsigned int kGaveUp = ~0u;
__device__ __noinline__ uint64_t check_wait(unsigned int spins, unsigned int seen, const WaitBound &w)
{
    bool out = *w.s_err || ((volatile unsigned int *)w.bar)[4];
    if (!out && spins > w.limit) {
        unsigned int sum = 0;
#pragma unroll 4
        for (int k = 0; k < 2 * w.n; k++) {  // (two words of dot terms a segment, two buffers)
            uint64_t lo, hi;
            ld_b128(w.words + 2 * (size_t)k, lo, hi);
            sum += (unsigned int)(hi >> 32);
        }
        out = sum == seen;
        seen = sum;
        spins = 0;
    }
    if (out) {
        *w.s_err = 1;
        atomicExch(&w.bar[4], 1u);
        spins = kGaveUp;
    }
    return pack2(spins, seen);
}
__device__ __forceinline__ bool keep_waiting(unsigned int &spins, unsigned int &seen, const WaitBound &w)
{
    if ((++spins & 63u) != 0) return true;
    const uint64_t s = check_wait(spins, seen, w);
    spins = (unsigned int)s;
    seen = (unsigned int)(s >> 32);
    return spins != kGaveUp;
}

// Words a thread waits for at once when it reads the restrictions.
constexpr int kBulk = 3;

// The first n of N words, `stride` words apart, once each carries the tag: a
// round reads every word still missing, so that it takes one trip to L2
// however many are late.
template <int N>
__device__ __forceinline__ void wait_words(const uint4 *p, int stride, int n, uint32_t tag, uint64_t (&lo)[N],
                                           uint64_t (&hi)[N], const WaitBound &w)
{
    unsigned int spins = 0, seen = ~0u;
    bool missing[N], any;
#pragma unroll
    for (int g = 0; g < N; g++) missing[g] = g < n;
    do {
#pragma unroll
        for (int g = 0; g < N; g++)
            if (missing[g]) ld_b128(p + (size_t)g * stride, lo[g], hi[g]);
        any = false;
#pragma unroll
        for (int g = 0; g < N; g++) {
            if (missing[g]) missing[g] = (uint32_t)(hi[g] >> 32) != tag;
            any |= missing[g];
        }
    } while (any && keep_waiting(spins, seen, w));
}

// The row again until it carries the tag (the slow path of a neighbour read).
template <typename T>
__device__ __noinline__ PubRow<T> wait_row(const uint4 *base, int n, int row, uint32_t tag, const WaitBound &w)
{
    PubRow<T> y;
    unsigned int spins = 0, seen = ~0u;
    do y.get(base, n, row);
    while (!y.is(tag) && keep_waiting(spins, seen, w));
    return y;
}

// transition_core out of line: its FP64 arithmetic (64 issue slots an
// instruction on GB300) stays out of the iteration's code.
__device__ __noinline__ bool transition_any(CgScalars *cg, const BlobParams *bp, const DF *sums, int *bits, bool fast)
{
    return transition_core(*cg, *bp, sums, bits, fast);
}

// An RNG stream's state one step's draws on.
__device__ __noinline__ void advance_stream(uint32_t *state, const mrg::JumpMat *step)
{
    uint32_t st[6];
#pragma unroll 1
    for (int i = 0; i < 6; i++) st[i] = state[i];
    mrg::apply(*step, st);
#pragma unroll 1
    for (int i = 0; i < 6; i++) state[i] = st[i];
}

// A sum in three FP32 parts (about 70 bits): FP32 runs at 64 times the FP64
// rate on GB300.
struct Sum3 {
    float s0, s1, s2;
};
__device__ __forceinline__ float two_sum(float a, float b, float &err)
{
    const float s = a + b, bb = s - a;
    err = (a - (s - bb)) + (b - bb);
    return s;
}
// S += K (dh + dl), the products exact (two FMAs each)
__device__ __forceinline__ void add_product(Sum3 &S, float K, float dh, float dl)
{
    const float p = __fmul_rn(K, dh), e = fmaf(K, dh, -p);
    const float q = __fmul_rn(K, dl), f = fmaf(K, dl, -q);
    float t0, t1, t2, t3;
    S.s0 = two_sum(S.s0, p, t0);
    t0 = two_sum(t0, e, t1);
    t0 = two_sum(t0, q, t2);
    S.s1 = two_sum(S.s1, t0, t3);
    S.s2 += (t1 + t2) + (t3 + f);
}

// Slots j0 .. j1 - 1 of a row's product A x added to a, with at least FP64
// precision: entry e + 32 j, column places lcol into su, the row's own x in
// xr (NoMass: difference form).  FP32 data: exact products and differences in
// three-part sums on the FP32 pipes.  One FP64 instruction takes 64 issue
// slots on GB300; in FP64 the 24 of a slot made the check of a 1,000-row CTA
// take 80 us, the 330 FP32 ones take a fifth of that.
__device__ __noinline__ void add_residual_slots(double (&a)[3], const float *val, const uint16_t *lcol, const float *su,
                                                const float *xr, int e, int j0, int j1, bool nomass)
{
    const float x[3] = {nomass ? xr[0] : 0.f, nomass ? xr[1] : 0.f, nomass ? xr[2] : 0.f};
    Sum3 S[3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
        const float *y = su + 4 * (size_t)__ldg(&lcol[e + 32 * j]);
        float dh[3], dl[3];
#pragma unroll
        for (int k = 0; k < 3; k++) dh[k] = two_sum(y[k], -x[k], dl[k]);
        if (nomass) {
            const float *v = val + sell_vidx(e + 32 * j, 0);
            float K[9];
#pragma unroll
            for (int k = 0; k < 9; k++) K[k] = __ldg(&v[32 * k]);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int k = 0; k < 3; k++) add_product(S[i], K[3 * i + k], dh[k], dl[k]);
        } else {
            const float m = __ldg(&val[e + 32 * j]);
#pragma unroll
            for (int k = 0; k < 3; k++) add_product(S[k], m, dh[k], dl[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) a[k] += (double)S[k].s0 + ((double)S[k].s1 + (double)S[k].s2);
}

// The same for FP64 data.
__device__ __noinline__ void add_residual_slots(double (&a)[3], const double *val, const uint16_t *lcol,
                                                const double *su, const double *xr, int e, int j0, int j1, bool nomass)
{
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
        const double *y = su + 4 * (size_t)__ldg(&lcol[e + 32 * j]);
        if (nomass) {
            const double *K = val + sell_vidx(e + 32 * j, 0);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int k = 0; k < 3; k++) a[i] += __ldg(&K[32 * (3 * i + k)]) * (y[k] - xr[k]);
        } else {
            const double m = __ldg(&val[e + 32 * j]);
#pragma unroll
            for (int k = 0; k < 3; k++) a[k] += m * y[k];
        }
    }
}

// The transition of an iteration that goes on, in FP32: transition_core's
// arithmetic.  False, with nothing changed, where the solve may stop or fail.
__device__ __forceinline__ bool transition_on(CgScalars &cg, int limit, const DF sums[3])
{
    const float g = sums[0].hi + sums[0].lo, dl = sums[1].hi + sums[1].lo, rr = sums[2].hi + sums[2].lo;
    const int iters = cg.iters;
    if (cg.state != CG_ACTIVE || (iters > 0 && rr < cg.stop_f) || !(rr == rr) || !(dl == dl) || iters >= limit)
        return false;
    const float beta = iters == 0 ? 0.f : g / cg.gamma_f;
    const float pap = iters == 0 ? dl : fmaf(-beta * beta, cg.pap_f, dl);
    if (!(pap > 0.f) || !(g > 0.f)) return false;
    cg.beta_f = beta;
    cg.pap_f = pap;
    cg.alpha_f = g / pap;
    cg.gamma_f = g;
    cg.iters = iters + 1;
    return true;
}

// The same in FP64, run by a warp (lane q < 3 with sum q): the conversions of
// the sums on a lane each and two of the four divisions on two lanes at once
// (a division takes nine times an instruction's 64 issue slots).
__device__ __forceinline__ bool transition_on64(CgScalars &cg, const BlobParams &bp, int limit, DF mine)
{
    const int lane = threadIdx.x & 31;
    const double v = (double)mine.hi + (double)mine.lo;
    const double g = __shfl_sync(0xffffffffu, v, 0), dl = __shfl_sync(0xffffffffu, v, 1),
                 rr = __shfl_sync(0xffffffffu, v, 2);
    const int iters = cg.iters;
    const double ff = cg.ff, gamma = cg.gamma, alpha = cg.alpha;
    if (cg.state != CG_ACTIVE || iters == 0 || iters >= limit || ff == 0.0) return false;
    const double t = (lane == 0 ? rr : g) / (lane == 0 ? ff : gamma);
    const double res = __shfl_sync(0xffffffffu, t, 0), beta = __shfl_sync(0xffffffffu, t, 1);
    if (!(res >= bp.epsilon2) || !(g == g) || !(dl == dl)) return false;  // (a NaN res too)
    const double an = g / (dl - beta * g / alpha);
    __syncwarp();
    if (lane == 0) {
        cg.rr = rr;
        cg.alpha = an;
        cg.beta = beta;
        cg.gamma = g;
        cg.iters = iters + 1;
    }
    return true;
}

// Matrix slots per step of the product: values on chip, and values from L2 (9
// registers in flight each).
template <typename T, int MAXT> struct SlotDepth { static constexpr int kOn = 4, kOff = 4; };
template <> struct SlotDepth<float, 1024> { static constexpr int kOn = 2, kOff = 2; };
template <> struct SlotDepth<double, 512> { static constexpr int kOn = 2, kOff = 2; };
template <> struct SlotDepth<double, 1024> { static constexpr int kOn = 1, kOff = 1; };

// ---------------------------------------------------------------- tensor memory
// Matrix values in the SM's tensor memory, 256 KB beside shared memory: a
// thread's lane of it is private to it, so its row's blocks are stored and
// read back with no address arithmetic and no bank conflicts.  W: 32-bit
// words of a block, at `addr` (lane in bits 16 up, column below).  A warp
// reaches the 32 lanes of its number modulo 4.
constexpr int kTmemCols = 512;

__device__ __forceinline__ void tmem_alloc(uint32_t *slot)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(slot);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "n"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(kTmemCols) : "memory");
}
__device__ __forceinline__ void tmem_put(uint32_t addr, const uint32_t (&v)[9])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%2, %3, %4, %5, %6, %7, %8, %9};\n\t"
                 "tcgen05.st.sync.aligned.32x32b.x1.b32 [%1], {%10};" ::"r"(addr), "r"(addr + 8), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8])
                 : "memory");
}
__device__ __forceinline__ void tmem_put(uint32_t addr, const uint32_t (&v)[18])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15, %16, %17};\n\t"
                 "tcgen05.st.sync.aligned.32x32b.x2.b32 [%1], {%18, %19};" ::"r"(addr), "r"(addr + 16), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17])
                 : "memory");
}
__device__ __forceinline__ void tmem_put_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// (the wait is part of the read: nothing can use the registers before it)
__device__ __forceinline__ void tmem_get(uint32_t addr, uint32_t (&v)[9])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%9];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%8}, [%10];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8])
                 : "r"(addr), "r"(addr + 8)
                 : "memory");
}
__device__ __forceinline__ void tmem_get(uint32_t addr, uint32_t (&v)[18])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15}, [%18];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%16, %17}, [%19];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                   "=r"(v[16]), "=r"(v[17])
                 : "r"(addr), "r"(addr + 16)
                 : "memory");
}
// row q of the CTA's copy of u
template <bool VEC, typename T>
__device__ __forceinline__ void put_u(T *su, int q, T x, T y, T z)
{
    T *o = su + 4 * (size_t)q;
    if constexpr (!VEC) {
        o[0] = x;
        o[1] = y;
        o[2] = z;
    } else if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4 *>(o) = make_float4(x, y, z, 0.f);
    } else {
        *reinterpret_cast<double2 *>(o) = make_double2(x, y);
        o[2] = z;
    }
}
template <typename T>
__device__ __forceinline__ T word_at(const uint32_t *v, int k)
{
    if constexpr (sizeof(T) == 4) return __uint_as_float(v[k]);
    else return __hiloint2double((int)v[2 * k + 1], (int)v[2 * k]);
}

// ---------------------------------------------------------------- the kernel
// T: arithmetic type of the vectors and the matrix.  COARSE: the two-level
// preconditioner (FP32).  MAXT: threads per CTA at most, which sets the
// registers a thread may use and the strides of the shared-memory arrays.
//
// R: segments of a CTA, two where a blob has more of them than there are CTAs
// (a 50 nm sphere: 304 of 931 rows; 59.1 us an iteration in the
// memory-resident solve, 35.1 here, 16 of them the matrix from HBM).  A
// thread has one row of each.  The values of a row's first cache_slots matrix
// slots are in shared memory, those of the next tmem_slots in tensor memory
// (not MAXT = 256, where shared memory has room for nearly all), the others
// come from L2.  With 965 rows to a CTA (a 40 nm sphere, 14 slots a row) the
// product was bound by L2, 469 KB a CTA at 34 bytes a clock: seven slots in
// tensor memory take 229 KB off that, 12.6 to 10.1 thousand clocks a product,
// 1,174 to 1,080 us a solve.
template <typename T, bool COARSE, int MAXT, int R>
__global__ void __launch_bounds__(MAXT, 1) k_cg_group(DeviceBatch d, GroupBatch gb)
{
    constexpr bool fast = sizeof(T) == 4;
    constexpr bool kRegs = MAXT <= 512;      // x, D^-1, p and s in registers, else in shared memory
    constexpr bool kWide = R > 1;            // u of the own rows from su, phi and X from L2: no room elsewhere
    constexpr bool kVec = MAXT > 512;        // (16-byte stores of u: 1 % slower in the small variants)
    using Row = PubRow<T>;
    using T2 = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
    __shared__ double s_dots[R][3 * 32];     // per slice: r.u, w.u, r.r (T, or FP64 for the true residual)
    __shared__ float s_ress[R][12 * 32];     // per slice: P^T r, P^T w
    __shared__ float s_red6[R][6 * 32];
    __shared__ float s_cvec[R][8];
    __shared__ CgScalars s_cg;
    __shared__ float s_outs[R][18];          // a segment's sums: r.u, w.u, r.r (hi, lo), P^T r, P^T w
    __shared__ DF s_part[3 * 32];            // the dot terms summed over 32 segments of the group each
    __shared__ DF s_last[3];                 // the sums of the last transition
    __shared__ BlobParams s_bp;
    __shared__ int s_err, s_stop;
    __shared__ WaitBound s_bound;
    __shared__ uint32_t s_tmem;
    constexpr bool kTmem = MAXT > 256;
    constexpr int kBlockWords = 9 * (int)sizeof(T) / 4;
    // FP64 products run in quarters of a slice, dealt over the CTA's warps,
    // where whole slices would leave some of the four schedulers idle: an FP64
    // instruction takes 64 issue slots, so the 160 of a row's product took a
    // warp 17 thousand clocks (two slices a CTA), its quarters 9 on eight warps
    constexpr bool kSplit = sizeof(T) == 8 && MAXT == 256;
    constexpr int kSplitRows = kSplit ? 192 : 1;
    __shared__ T s_acc[kSplit ? 3 : 1][3][kSplitRows];
    __shared__ int s_rowL[kSplitRows], s_rowE[kSplitRows];  // slots and first entry of a row
    const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = NT >> 5;
    const uint32_t base = __ldcg(&d.bar[6]);  // the tags of this launch start above it
    T *const sx = dyn<T>(gb.o_state);         // per segment x | D^-1 | p | s, 3 MAXT each (unless kRegs)
    T *const su = dyn<T>(gb.o_u);             // u of the CTA's rows, then of its halo, (x, y, z, 0) each
    uint4 *const pub = gb.pub;
    uint32_t maxseq = 0;
    const uint64_t pol = kWide ? stream_policy() : 0;
    int maxloops = 0;
    if (tid == 0) {
        s_err = s_stop = 0;
        s_bound = {gb.words, d.n_segs, gb.spin_limit, &s_err, d.bar};
    }
    uint32_t tmem = 0;  // the warp's part: its lanes, and its share of their columns
    if constexpr (kTmem) {
        if (gb.tmem_slots > 0) {
            __syncwarp();
            if (warp == 0) tmem_alloc(&s_tmem);
            __syncthreads();
            tmem = s_tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * R * gb.tmem_slots * kBlockWords);
        }
    }

#pragma unroll 1
    for (int ti = gb.ptr[blockIdx.x]; ti < gb.ptr[blockIdx.x + 1]; ti++) {
        const int seg = gb.task[ti], b = d.seg_blob[seg];
        __syncthreads();  // the previous task is done with shared memory
#pragma unroll 1
        for (int k = tid; k < (int)(sizeof(BlobParams) / 4); k += NT)
            reinterpret_cast<int *>(&s_bp)[k] = reinterpret_cast<const int *>(d.bp + b)[k];
#pragma unroll 1
        for (int k = tid; k < (int)(sizeof(CgScalars) / 4); k += NT)
            reinterpret_cast<int *>(&s_cg)[k] = __ldcg(reinterpret_cast<const int *>(d.cg + b) + k);
        __syncthreads();
        const int cnt = s_bp.seg_cnt;          // segments of the group
        const bool solo = cnt == 1;
        int row0[R], nsl[R];
        bool in[R], valid[R];  // a row of the segment, a free one
#pragma unroll
        for (int q = 0; q < R; q++) {
            const bool has = q == 0 || seg + q < s_bp.seg_off + cnt;
            row0[q] = has ? d.seg_row0[seg + q] : 0;
            const int nrows = has ? d.seg_rows[seg + q] : 0;
            nsl[q] = (nrows + 31) >> 5;
            in[q] = tid < nrows;
            valid[q] = in[q] && !(d.flags[row0[q] + tid] & NODE_PINNED);
        }
        const bool leader = seg == s_bp.seg_off;
        const bool nomass = s_bp.solver == SOLVER_NOMASS;
        const int cn = COARSE ? s_bp.coarse_n : 0;
        const int limit = s_bp.solver == SOLVER_MASS ? s_bp.max_iter - 1 : s_bp.max_iter;
        const bool run = s_cg.state == CG_ACTIVE;
        const int h0 = gb.hptr[seg], nh = gb.hptr[seg + 1] - h0;  // halo rows
        T diag[R];
        int L[R], ebase[R];  // slots of the row, its first entry
        T r[R][3], u[kWide ? 1 : R][3], w[R][3];
        T st[4][kRegs ? 3 : 1];  // x, D^-1, p, s
        auto state_of = [&](int q, int f, int k) -> T & {
            if constexpr (kRegs) return st[f][k];
            else return sx[((4 * q + f) * 3 + k) * MAXT + tid];
        };
        auto phi_of = [&](int q) -> float4 {
            if constexpr (kWide) return __ldg(&d.phi[row0[q] + tid]);
            else return dyn<float4>(gb.o_phi)[tid];
        };
#pragma unroll
        for (int q = 0; q < R; q++) {
            const int row = row0[q] + tid;
            diag[q] = (T)0;
            L[q] = ebase[q] = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                r[q][k] = w[q][k] = (T)0;
                if (!kWide) u[q][k] = (T)0;
#pragma unroll
                for (int f = 0; f < 4; f++) state_of(q, f, k) = (T)0;
            }
            if (kWide) put_u<kVec>(su, q * MAXT + tid, (T)0, (T)0, (T)0);
            if (run && in[q]) {
                const size_t o = 3 * (size_t)row;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    r[q][k] = static_cast<const T *>(d.r)[o + k];
                    state_of(q, 1, k) = static_cast<const T *>(d.dinv)[o + k];
                }
            }
            if (run && valid[q]) {
                diag[q] = nomass ? (T)(s_bp.calc_stokes == 1 ? d.drag[row] : 0.0)
                                 : static_cast<const T *>(d.mass_diag)[row];
                L[q] = d.slice_len[row >> 5];
                ebase[q] = d.slice_ptr[row >> 5] + (row & 31);
            }
        }
        // the row's neighbours (places in su) and matrix values on chip:
        // constant during the solve
        if (kSplit && tid < kSplitRows) {
            s_rowL[kSplit ? tid : 0] = L[0];
            s_rowE[kSplit ? tid : 0] = ebase[0];
        }
        int T0[R], T1[R];  // the slots in tensor memory, the same for the warp
#pragma unroll
        for (int q = 0; q < R; q++) {
            if (run && valid[q]) {
                // kFill slots' loads in flight (one where the registers do not
                // suffice): the setup of a 64-row CTA 19 -> 12 thousand clocks
                constexpr int kFill = MAXT <= 256 ? 4 : 1;
                uint16_t *col = dyn<uint16_t>(gb.o_col) + q * gb.cache_cols * MAXT + tid;
#pragma unroll kFill
                for (int j = 0; j < min(gb.cache_cols, L[q]); j++) col[j * MAXT] = __ldg(&gb.lcol[ebase[q] + 32 * j]);
                T *kv1 = dyn<T>(gb.o_kv1) + q * gb.cache_slots * MAXT + tid;
                T2 *kv2 = dyn<T2>(gb.o_kv2) + q * 4 * gb.cache_slots * MAXT + tid;
                const int n = min(gb.cache_slots, L[q]);
#pragma unroll 1
                for (int i0 = 0; i0 < n; i0 += kFill) {
                    T v[kFill][9];
#pragma unroll
                    for (int g = 0; g < kFill; g++) {
                        if (i0 + g >= n) continue;
                        const int e = ebase[q] + 32 * (i0 + g);
                        if (nomass) {
                            const T *val = static_cast<const T *>(d.sell_val) + sell_vidx(e, 0);
#pragma unroll
                            for (int m = 0; m < 9; m++) v[g][m] = __ldg(&val[32 * m]);
                        } else {
                            v[g][8] = __ldg(static_cast<const T *>(d.sell_mval) + e);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < kFill; g++) {
                        if (i0 + g >= n) continue;
                        const int i = i0 + g;
                        if (nomass)
#pragma unroll
                            for (int m = 0; m < 4; m++) {
                                T2 kp;
                                kp.x = v[g][2 * m];
                                kp.y = v[g][2 * m + 1];
                                kv2[(4 * i + m) * MAXT] = kp;
                            }
                        kv1[i * MAXT] = v[g][8];
                    }
                }
            }
            T0[q] = T1[q] = 0;
            if constexpr (kTmem) {
                if (run && nomass && warp < nsl[q]) {
                    const int Lw = d.slice_len[(row0[q] >> 5) + warp];
                    // every other warp of a scheduler keeps its last slots there,
                    // so that half of the warps read L2 while the others do not
                    T0[q] = min(gb.cache_slots, Lw);
                    if (warp & 4) T0[q] = max(T0[q], min(gb.cache_cols, Lw) - gb.tmem_slots);
                    T1[q] = min(T0[q] + gb.tmem_slots, min(gb.cache_cols, Lw));
                    __syncwarp();
#pragma unroll 1
                    for (int j = T0[q]; j < T1[q]; j++) {
                        const T *val = static_cast<const T *>(d.sell_val) + sell_vidx(ebase[q] + 32 * j, 0);
                        uint32_t v[kBlockWords];
#pragma unroll
                        for (int k = 0; k < 9; k++) {
                            const T x = valid[q] ? val[32 * k] : (T)0;
                            if constexpr (fast) {
                                v[k] = __float_as_uint(x);
                            } else {
                                v[2 * k] = (uint32_t)__double2loint(x);
                                v[2 * k + 1] = (uint32_t)__double2hiint(x);
                            }
                        }
                        tmem_put(tmem + (q * gb.tmem_slots + j - T0[q]) * kBlockWords, v);
                    }
                    tmem_put_done();
                }
            }
            if (COARSE && !kWide && run && in[q])
                dyn<float4>(gb.o_phi)[tid] = valid[q] ? d.phi[row0[q] + tid] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (run) {
            int *halo = dyn<int>(gb.o_halo);
#pragma unroll 1
            for (int k = tid; k < nh; k += NT) halo[k] = gb.halo[h0 + k];
            if (COARSE) {
                float *h = dyn<float>(gb.o_h);
                if (!kWide) {
                    const float *Xg = d.coarse_X + s_bp.coarse_xoff + (size_t)(6 * (seg - s_bp.seg_off)) * cn;
                    float *xr = dyn<float>(gb.o_xrow);
#pragma unroll 1
                    for (int k = tid; k < 6 * cn; k += NT) xr[k] = Xg[k];
                }
#pragma unroll 1
                for (int k = tid; k < cn; k += NT) h[k] = 0.f;
            }
#pragma unroll 1
            for (int k = tid; k < R * 3 * 32; k += NT) s_dots[0][k] = 0.0;
#pragma unroll 1
            for (int k = tid; k < R * 12 * 32; k += NT) s_ress[0][k] = 0.f;
        }
        __syncthreads();

        uint32_t seq = 0;  // exchanges of this solve
        int parity = 0, loops = -1;
        // fresh: the vectors restart (the first trip, and after a failed true
        // residual): no update.  first_coarse: the restriction of r_0, which
        // the first u needs
        bool fresh = true, first_coarse = COARSE;
        bool going = run;
        while (going) {
            const int state = s_cg.state;
            const uint32_t tag = base + ++seq;
            const bool verify = state == CG_VERIFY;
            const bool product = !verify && !first_coarse;
            // the row's terms of r.u and r.r and its restriction of r, and
            // their slice sums (a slice is a warp)
            T pg[R], pr[R];
            float ex[R][6];
#pragma unroll
            for (int q = 0; q < R; q++) {
                double *s_dot = s_dots[q];
                float *s_res = s_ress[q];
                const int me = q * MAXT + tid;  // the row's place in su
                T uq[3];
#pragma unroll
                for (int k = 0; k < 3; k++) uq[k] = kWide ? su[4 * me + k] : u[kWide ? 0 : q][k];
                if (product) {
                    // phase A: p = u + beta p; s = w + beta s; x += alpha p;
                    // r -= alpha s; u = M r; publish u
                    T a, be;
                    cg_coefs<T>(s_cg, a, be);
                    if (valid[q]) {
                        if (!fresh) {
                            const bool first = be == (T)0;
#pragma unroll
                            for (int k = 0; k < 3; k++) {
                                T &p = state_of(q, 2, k), &s = state_of(q, 3, k);
                                const T pn = first ? uq[k] : uq[k] + be * p;
                                const T sn = first ? w[q][k] : w[q][k] + be * s;
                                p = pn;
                                s = sn;
                                state_of(q, 0, k) += a * pn;
                                r[q][k] -= a * sn;
                            }
                        }
                        T dinv[3];
#pragma unroll
                        for (int k = 0; k < 3; k++) dinv[k] = state_of(q, 1, k);
                        if (COARSE) {
                            coarse_u_of<T>(phi_of(q), s_cvec[q], dinv, r[q], uq);
                        } else {
#pragma unroll
                            for (int k = 0; k < 3; k++) uq[k] = dinv[k] * r[q][k];
                        }
                    }
                    if (in[q]) {
                        if (!solo) Row::put(pub, d.nl_pad, row0[q] + tid, uq, tag);
                        put_u<kVec>(su, me, uq[0], uq[1], uq[2]);
                    }
                    if (!kWide)
#pragma unroll
                        for (int k = 0; k < 3; k++) u[kWide ? 0 : q][k] = uq[k];
                } else if (verify) {
                    // publish x for the true residual
                    if (in[q]) {
                        const T xv[3] = {state_of(q, 0, 0), state_of(q, 0, 1), state_of(q, 0, 2)};
                        if (!solo) Row::put(pub, d.nl_pad, row0[q] + tid, xv, tag);
                        put_u<kVec>(su, me, xv[0], xv[1], xv[2]);
                    }
                }
                pg[q] = pr[q] = (T)0;
#pragma unroll
                for (int k = 0; k < 6; k++) ex[q][k] = 0.f;
                if (valid[q] && product)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        pg[q] += r[q][k] * uq[k];
                        pr[q] += r[q][k] * r[q][k];
                    }
                if (COARSE && valid[q] && !verify) restrict6_of<T>(phi_of(q), r[q], ex[q]);
                if constexpr (fast) {
                    if (product) {
                        constexpr int NV = COARSE ? 8 : 2;
                        float v[NV];
                        v[0] = (float)pg[q];
                        v[1] = (float)pr[q];
                        if (COARSE)
#pragma unroll
                            for (int k = 0; k < 6; k++) v[2 + k] = ex[q][k];
                        int idx;
                        const float t = warp_sum_multi<NV>(v, idx);
                        if ((lane & (32 / NV - 1)) == 0) {
                            if (idx < 2) reinterpret_cast<float *>(s_dot)[(idx == 0 ? 0 : 2) * 32 + warp] = t;
                            else s_res[(idx - 2) * 32 + warp] = t;
                        }
                    }
                }
            }
            // the halo's rows of u (or x), when their CTAs have published them
            if (!solo && !first_coarse)
#pragma unroll 1
                for (int k = tid; k < nh; k += NT) {
                    const int q = dyn<int>(gb.o_halo)[k];
                    Row y;
                    y.get(pub, d.nl_pad, q);
                    if (!y.is(tag)) y = wait_row<T>(pub, d.nl_pad, q, tag, s_bound);
                    put_u<kVec>(su, R * MAXT + k, y.x, y.y, y.z);
                }
            __syncthreads();  // su
            auto load3 = [&](int q, T y[3]) {
                const T *s = su + 4 * (size_t)q;
                if constexpr (fast) {
                    const float4 f = *reinterpret_cast<const float4 *>(s);
                    y[0] = f.x;
                    y[1] = f.y;
                    y[2] = f.z;
                } else {
                    const double2 f = *reinterpret_cast<const double2 *>(s);
                    y[0] = f.x;
                    y[1] = f.y;
                    y[2] = s[2];
                }
            };
#pragma unroll
            for (int q = 0; q < R; q++) {
                double *s_dot = s_dots[q];
                float *s_res = s_ress[q];
                const int me = q * MAXT + tid;
                if (product) {
                    // phase B: w = A u
                    T uq[3];
                    if (kWide) {
                        load3(me, uq);  // (zeros past the segment's rows)
                    } else {
#pragma unroll
                        for (int k = 0; k < 3; k++) uq[k] = u[kWide ? 0 : q][k];
                    }
                    T acc[3] = {diag[q] * uq[0], diag[q] * uq[1], diag[q] * uq[2]};
                    bool split = false;
                    if constexpr (kSplit) split = (nsl[0] & 3) != 0 && 32 * nsl[0] <= kSplitRows;
                    if (kSplit && split) {
#pragma unroll 1
                        for (int item = warp; item < 4 * nsl[0]; item += nw) {
                            const int part = item / nsl[0], hr = 32 * (item % nsl[0]) + lane;
                            const int Lr = s_rowL[kSplit ? hr : 0], er = s_rowE[kSplit ? hr : 0];
                            const uint16_t *col = dyn<uint16_t>(gb.o_col) + hr;
                            const T *kv1 = dyn<T>(gb.o_kv1) + hr;
                            const T2 *kv2 = dyn<T2>(gb.o_kv2) + hr;
                            T uh[3], sum[3] = {0, 0, 0};
                            load3(hr, uh);
#pragma unroll 2
                            for (int j = part; j < Lr; j += 4) {
                                const int e = er + 32 * j;
                                const bool on = j < gb.cache_slots;
                                T y[3];
                                load3(j < gb.cache_cols ? col[j * MAXT] : __ldg(&gb.lcol[e]), y);
                                if (nomass) {
                                    T Kj[9];
                                    if (on) {
#pragma unroll
                                        for (int m = 0; m < 4; m++) {
                                            const T2 kp = kv2[(4 * j + m) * MAXT];
                                            Kj[2 * m] = kp.x;
                                            Kj[2 * m + 1] = kp.y;
                                        }
                                        Kj[8] = kv1[j * MAXT];
                                    } else {
                                        const T *vp = static_cast<const T *>(d.sell_val) + sell_vidx(e, 0);
#pragma unroll
                                        for (int k = 0; k < 9; k++) Kj[k] = __ldg(vp + 32 * k);
                                    }
                                    block_fma(Kj, y[0] - uh[0], y[1] - uh[1], y[2] - uh[2], sum[0], sum[1], sum[2]);
                                } else {
                                    const T m = on ? kv1[j * MAXT] : __ldg(static_cast<const T *>(d.sell_mval) + e);
#pragma unroll
                                    for (int k = 0; k < 3; k++) sum[k] = fma(m, y[k], sum[k]);
                                }
                            }
                            // (the first quarter of a slice is its own warp's)
#pragma unroll
                            for (int k = 0; k < 3; k++) {
                                if (part > 0) s_acc[kSplit ? part - 1 : 0][k][kSplit ? hr : 0] = sum[k];
                                else acc[k] += sum[k];
                            }
                        }
                        __syncthreads();  // s_acc
                        if (valid[q])
#pragma unroll
                            for (int k = 0; k < 3; k++)
                                acc[k] = (acc[k] + s_acc[0][k][kSplit ? tid : 0]) +
                                         (s_acc[kSplit ? 1 : 0][k][kSplit ? tid : 0] +
                                          s_acc[kSplit ? 2 : 0][k][kSplit ? tid : 0]);
                    } else {
                        // slots on chip, then the others.  Past the last of them a
                        // step takes the row itself with zero values
                        const int JC = gb.cache_cols, J1 = min(gb.cache_slots, L[q]);
                        const uint16_t *col = dyn<uint16_t>(gb.o_col) + q * gb.cache_cols * MAXT + tid;
                        const T *kv1 = dyn<T>(gb.o_kv1) + q * gb.cache_slots * MAXT + tid;
                        if (nomass) {
                            const T2 *kv2 = dyn<T2>(gb.o_kv2) + q * 4 * gb.cache_slots * MAXT + tid;
                            constexpr int G1 = SlotDepth<T, MAXT>::kOn, G2 = SlotDepth<T, MAXT>::kOff;
#pragma unroll 1
                            for (int j0 = 0; j0 < J1; j0 += G1) {
                                T y[G1][3];
#pragma unroll
                                for (int g = 0; g < G1; g++) load3(j0 + g < J1 ? col[(j0 + g) * MAXT] : me, y[g]);
#pragma unroll
                                for (int g = 0; g < G1; g++) {
                                    const int j = j0 + g < J1 ? j0 + g : j0;
                                    T Kj[9];
#pragma unroll
                                    for (int m = 0; m < 4; m++) {
                                        const T2 kp = kv2[(4 * j + m) * MAXT];
                                        Kj[2 * m] = kp.x;
                                        Kj[2 * m + 1] = kp.y;
                                    }
                                    Kj[8] = kv1[j * MAXT];
                                    // (past the last slot y is u: the products are zeros)
                                    block_fma(Kj, y[g][0] - uq[0], y[g][1] - uq[1], y[g][2] - uq[2], acc[0], acc[1],
                                              acc[2]);
                                }
                            }
                            // values from L2, slots ja .. jb - 1
                            auto from_l2 = [&](int ja, int jb) {
                                const T *vp = static_cast<const T *>(d.sell_val) + sell_vidx(ebase[q] + 32 * ja, 0);
#pragma unroll 1
                                for (int j0 = ja; j0 < jb; j0 += G2, vp += 288 * G2) {
                                    T Kj[G2][9];
#pragma unroll
                                    for (int g = 0; g < G2; g++)
#pragma unroll
                                        for (int k = 0; k < 9; k++)
                                            Kj[g][k] = j0 + g >= jb ? (T)0
                                                       : kWide      ? ld_stream(vp + 288 * g + 32 * k, pol)
                                                                    : __ldg(vp + 288 * g + 32 * k);
#pragma unroll
                                    for (int g = 0; g < G2; g++) {
                                        const int j = j0 + g;
                                        T y[3];
                                        load3(j >= jb  ? me
                                              : j < JC ? col[j * MAXT]
                                                       : __ldg(&gb.lcol[ebase[q] + 32 * j]),
                                              y);
                                        block_fma(Kj[g], y[0] - uq[0], y[1] - uq[1], y[2] - uq[2], acc[0], acc[1],
                                                  acc[2]);
                                    }
                                }
                            };
                            if constexpr (kTmem) {
                                constexpr int GT = sizeof(T) == 4 ? 2 : 1;
                                constexpr int W = GT * kBlockWords;
#pragma unroll 1
                                for (int pass = 0; pass < 2; pass++) {
                                    const int ja = pass == 0 ? J1 : max(J1, min(T1[q], L[q]));
                                    from_l2(ja, pass == 0 ? min(T0[q], L[q]) : L[q]);
                                    if (pass > 0) break;
                                    __syncwarp();
                                    int j = T0[q];
#pragma unroll 1
                                    for (; j + GT <= T1[q]; j += GT) {
                                        uint32_t v[W];
                                        T y[GT][3];
#pragma unroll
                                        for (int g = 0; g < GT; g++)
                                            load3(j + g < L[q] ? col[(j + g) * MAXT] : me, y[g]);
                                        tmem_get(tmem + (q * gb.tmem_slots + j - T0[q]) * kBlockWords, v);
#pragma unroll
                                        for (int g = 0; g < GT; g++) {
                                            T Kj[9];
#pragma unroll
                                            for (int k = 0; k < 9; k++) Kj[k] = word_at<T>(v + g * kBlockWords, k);
                                            block_fma(Kj, y[g][0] - uq[0], y[g][1] - uq[1], y[g][2] - uq[2], acc[0],
                                                      acc[1], acc[2]);
                                        }
                                    }
                                    if (GT > 1 && j < T1[q]) {
                                        uint32_t v[kBlockWords];
                                        T y[3], Kj[9];
                                        load3(j < L[q] ? col[j * MAXT] : me, y);
                                        tmem_get(tmem + (q * gb.tmem_slots + j - T0[q]) * kBlockWords, v);
#pragma unroll
                                        for (int k = 0; k < 9; k++) Kj[k] = word_at<T>(v, k);
                                        block_fma(Kj, y[0] - uq[0], y[1] - uq[1], y[2] - uq[2], acc[0], acc[1], acc[2]);
                                    }
                                }
                            } else {
                                from_l2(J1, L[q]);
                            }
                        } else {
                            const T *mv = static_cast<const T *>(d.sell_mval);
#pragma unroll 2
                            for (int j = 0; j < L[q]; j++) {
                                T y[3];
                                load3(j < JC ? col[j * MAXT] : __ldg(&gb.lcol[ebase[q] + 32 * j]), y);
                                const T m = j < J1 ? kv1[j * MAXT] : __ldg(&mv[ebase[q] + 32 * j]);
#pragma unroll
                                for (int k = 0; k < 3; k++) acc[k] = fma(m, y[k], acc[k]);
                            }
                        }
                    }
                    T pd = (T)0;
                    if (valid[q])
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            w[q][k] = acc[k];
                            pd += w[q][k] * uq[k];
                        }
                    if constexpr (fast) {
                        float ew[6] = {0, 0, 0, 0, 0, 0};
                        if (COARSE && valid[q]) restrict6_of<T>(phi_of(q), w[q], ew);
                        constexpr int NV = COARSE ? 8 : 2;
                        float v[NV];
                        v[0] = (float)pd;
                        v[1] = 0.f;
                        if (COARSE)
#pragma unroll
                            for (int k = 0; k < 6; k++) v[2 + k] = ew[k];
                        int idx;
                        const float t = warp_sum_multi<NV>(v, idx);
                        if ((lane & (32 / NV - 1)) == 0) {
                            if (idx == 0) reinterpret_cast<float *>(s_dot)[1 * 32 + warp] = t;
                            else if (idx >= 2) s_res[(6 + idx - 2) * 32 + warp] = t;
                        }
                    } else {
                        T v[4] = {pg[q], pd, pr[q], (T)0}, t = (T)0;
                        int idx = lane >> 3;
                        if (warp < nsl[q]) t = warp_sum_multi<4>(v, idx);
                        if ((lane & 7) == 0 && idx < 3) reinterpret_cast<T *>(s_dot)[idx * 32 + warp] = t;
                    }
                } else {
                    // the FP64 true residual b - A x of the published x becomes r
                    // (VERIFY), or the restriction of r_0 alone.
                    double vr = 0.0, vg = 0.0;
                    if (verify) {
                        double a[3] = {0.0, 0.0, 0.0};
                        if (valid[q]) {
                            const T *xr = su + 4 * (size_t)me;
#pragma unroll
                            for (int k = 0; k < 3; k++) a[k] = (double)diag[q] * (double)xr[k];
                            add_residual_slots(a, static_cast<const T *>(nomass ? d.sell_val : d.sell_mval), gb.lcol,
                                                  su, xr, ebase[q], 0, L[q], nomass);
                        }
                        if (valid[q]) {
                            const size_t o = 3 * (size_t)(row0[q] + tid);
#pragma unroll
                            for (int k = 0; k < 3; k++) {
                                const double rt = d.rhs[o + k] - a[k];
                                r[q][k] = (T)rt;
                                const T uk = state_of(q, 1, k) * r[q][k];
                                vr += rt * rt;
                                vg += (double)r[q][k] * (double)uk;
                            }
                            if (COARSE) restrict6_of<T>(phi_of(q), r[q], ex[q]);
                        }
                        vg = warp_sum<double>(vg);
                        vr = warp_sum<double>(vr);
                    }
                    if (lane == 0) {
                        s_dot[0 * 32 + warp] = vg;
                        s_dot[1 * 32 + warp] = 0.0;
                        s_dot[2 * 32 + warp] = vr;
                    }
                    if (COARSE) {
#pragma unroll
                        for (int k = 0; k < 6; k++) {
                            const float t = warp_sum<float>(ex[q][k]);
                            if (lane == 0) {
                                s_res[k * 32 + warp] = t;
                                s_res[(6 + k) * 32 + warp] = 0.f;
                            }
                        }
                    }
                }
            }
            __syncthreads();  // the slices' sums
            // butterflies as wide as the slices need
            const int most = max(nsl[0], nsl[R - 1]);
            const int half = most > 1 ? 1 << (31 - __clz(most - 1)) : 0;
            // A segment's sums over its slices into s_outs: warps 0..2 a dot
            // term each (hi, lo), warps 3..6 three values each of P^T r, P^T w
            auto combine = [&](int q, int l) {
                const int n = R == 1 || q == 0 ? nsl[0] : nsl[R - 1];
                float *s_out = s_outs[q];
                if (l < 3) {
                    float hi, lo;
                    if (sizeof(T) == 8 || !product) {
                        double a = lane < n ? s_dots[q][l * 32 + lane] : 0.0;
#pragma unroll
                        for (int k = 16; k > 0; k >>= 1)
                            if (k <= half) a += __shfl_xor_sync(0xffffffffu, a, k);
                        hi = (float)a;
                        lo = (float)(a - (double)hi);
                    } else {
                        DF v{lane < n ? reinterpret_cast<const float *>(s_dots[q])[l * 32 + lane] : 0.f, 0.f};
#pragma unroll
                        for (int k = 16; k > 0; k >>= 1)
                            if (k <= half)
                                v = df_add(v, DF{__shfl_xor_sync(0xffffffffu, v.hi, k),
                                                 __shfl_xor_sync(0xffffffffu, v.lo, k)});
                        hi = v.hi;
                        lo = v.lo;
                    }
                    if (lane == 0) {
                        s_out[2 * l] = hi;
                        s_out[2 * l + 1] = lo;
                    }
                } else if (COARSE) {
                    const int k0 = 3 * (l - 3);
                    float v[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) v[c] = lane < n ? s_ress[q][(k0 + c) * 32 + lane] : 0.f;
#pragma unroll
                    for (int k = 16; k > 0; k >>= 1)
                        if (k <= half)
#pragma unroll
                            for (int c = 0; c < 3; c++) v[c] += __shfl_xor_sync(0xffffffffu, v[c], k);
                    if (lane == 0)
#pragma unroll
                        for (int c = 0; c < 3; c++) s_out[6 + k0 + c] = v[c];
                }
            };
            if constexpr (R == 1) {
                if (warp < 7) combine(0, warp);
            } else {
#pragma unroll 1
                for (int k = warp; k < 7 * R; k += nw) combine(k / 7, k % 7);
            }
            __syncthreads();  // s_outs
            // published in whole 32-byte sectors by one store: words 0, 1 the
            // dot terms, 2..5 P^T r and P^T w, three values each
            uint4 *const dots = gb.words + (size_t)parity * 2 * d.n_segs;
            uint4 *const rest = gb.words + (size_t)4 * d.n_segs + (size_t)parity * 4 * d.n_segs;
            float *const swr = dyn<float>(gb.o_words), *const sww = swr + 6 * cnt;  // the group's P^T r and P^T w
            const int pq = R == 1 ? 0 : lane >> 3, l = R == 1 ? lane : lane & 7;
            if (warp == 0 && l < (COARSE ? 6 : 2) && (pq == 0 || (pq < R && nsl[R - 1] > 0))) {
                const int q = R == 1 ? 0 : pq;
                const float a = s_outs[q][3 * l], b2 = s_outs[q][3 * l + 1], c = s_outs[q][3 * l + 2];
                // (a blob of one segment publishes its dot terms for the waits' sake alone)
                if (!solo || l < 2) {
                    uint4 *o = l < 2 ? dots + 2 * (size_t)(seg + q) + l : rest + 4 * (size_t)(seg + q) + l - 2;
                    st_b128(o, pack2(__float_as_uint(a), __float_as_uint(b2)), pack2(__float_as_uint(c), tag));
                } else {
                    float *o = swr + 3 * (l - 2);  // (sww follows: one segment)
                    o[0] = a;
                    o[1] = b2;
                    o[2] = c;
                }
            }
            // the dot terms of every segment of the group, a segment per lane
            // of the first warps, summed per warp
            if (32 * warp < cnt) {
                DF sum[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
                const int sg = 32 * warp + lane;
                if (solo) {
                    if (lane == 0)
#pragma unroll
                        for (int q = 0; q < 3; q++) sum[q] = DF{s_outs[0][2 * q], s_outs[0][2 * q + 1]};
                } else if (sg < cnt) {
                    uint64_t lo[2], hi[2];
                    wait_words<2>(dots + 2 * (size_t)(s_bp.seg_off + sg), 1, 2, tag, lo, hi, s_bound);
                    sum[0] = DF{__uint_as_float((uint32_t)lo[0]), __uint_as_float((uint32_t)(lo[0] >> 32))};
                    sum[1] = DF{__uint_as_float((uint32_t)hi[0]), __uint_as_float((uint32_t)lo[1])};
                    sum[2] = DF{__uint_as_float((uint32_t)(lo[1] >> 32)), __uint_as_float((uint32_t)hi[1])};
                }
                __syncwarp();
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    if (o < cnt)  // (lanes past cnt hold zeros)
#pragma unroll
                        for (int q = 0; q < 3; q++)
                            sum[q] = df_add(sum[q], DF{__shfl_xor_sync(0xffffffffu, sum[q].hi, o),
                                                       __shfl_xor_sync(0xffffffffu, sum[q].lo, o)});
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 3; q++) s_part[3 * warp + q] = sum[q];
            }
            __syncthreads();  // sw
            if (warp == 0) {
                // a lane for each sum over the parts
                DF sum{0.f, 0.f};
                if (lane < 3) {
                    sum = s_part[lane];
                    for (int k = 1; 32 * k < cnt; k++) sum = df_add(sum, s_part[3 * k + lane]);
                }
                DF sums[3];
#pragma unroll
                for (int q = 0; q < 3; q++)
                    sums[q] = DF{__shfl_sync(0xffffffffu, sum.hi, q), __shfl_sync(0xffffffffu, sum.lo, q)};
                bool on = false;
                if constexpr (!fast) on = transition_on64(s_cg, s_bp, limit, sum);
                if (lane == 0) {
                    if (!first_coarse) {
#pragma unroll
                        for (int q = 0; q < 3; q++) s_last[q] = sums[q];
                        int bits;
                        if (!(fast ? transition_on(s_cg, limit, sums) : on) &&
                            transition_any(&s_cg, &s_bp, s_last, &bits, fast) && bits && leader)
                            atomicOr(&d.status[b], bits);
                    }
                    s_stop = s_err;
                }
            } else if (COARSE && !solo) {
                // meanwhile every segment's restrictions, kBulk words in flight
                const uint4 *gr = rest + 4 * (size_t)s_bp.seg_off;
                const int n = 4 * cnt, step = NT - 32;
#pragma unroll 1
                for (int i0 = tid - 32; i0 < n; i0 += kBulk * step) {
                    uint64_t lo[kBulk], hi[kBulk];
                    wait_words<kBulk>(gr + i0, step, (n - i0 + step - 1) / step, tag, lo, hi, s_bound);
#pragma unroll
                    for (int g = 0; g < kBulk; g++) {
                        const int i = i0 + g * step;
                        if (i >= n) break;
                        float *o = ((i & 2) ? sww : swr) + 6 * (i >> 2) + 3 * (i & 1);
                        o[0] = __uint_as_float((uint32_t)lo[g]);
                        o[1] = __uint_as_float((uint32_t)(lo[g] >> 32));
                        o[2] = __uint_as_float((uint32_t)hi[g]);
                    }
                }
            }
            __syncthreads();  // the new state
            const int nst = s_cg.state;
            going = nst != CG_CONVERGED && nst != CG_FAILED && !s_stop;
            if (COARSE && going && nst != CG_VERIFY) {
                // the coarse correction of the next u: h = P^T w + beta h,
                // g = P^T r - alpha h (P^T r of the next residual; after a
                // restart P^T r itself), c = X g for the CTA's segment
                const bool restart = first_coarse || nst == CG_RESTART;
                float *h = dyn<float>(gb.o_h);
                const float al = s_cg.alpha_f, be = s_cg.beta_f;
#pragma unroll
                for (int q = 0; q < R; q++) {
                    const float *xr = dyn<float>(gb.o_xrow);
                    if (kWide)
                        xr = d.coarse_X + s_bp.coarse_xoff +
                             (size_t)(6 * (seg - s_bp.seg_off + (nsl[q] > 0 ? q : 0))) * cn;
                    float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 2
                    for (int j = tid; j < cn; j += NT) {
                        const float pr_j = swr[j];
                        float hn = h[j];
                        if (q == 0) {
                            hn = restart ? 0.f : sww[j] + be * hn;
                            h[j] = hn;
                        }
                        const float g = restart ? pr_j : pr_j - al * hn;
#pragma unroll
                        for (int l = 0; l < 6; l++) v[l] = fmaf(xr[l * cn + j], g, v[l]);
                    }
                    int idx;
                    const float t = warp_sum_multi<8>(v, idx);
                    if ((lane & 3) == 0 && idx < 6) s_red6[q][idx * 32 + warp] = t;
                }
                __syncthreads();
#pragma unroll 1
                for (int l = warp; l < 6 * R; l += nw) {
                    const int q = R == 1 ? 0 : l / 6, k = l - 6 * q;
                    const float c = warp_sum<float>(lane < nw ? s_red6[q][k * 32 + lane] : 0.f);
                    if (lane == 0) s_cvec[q][k] = c;
                }
                __syncthreads();  // s_cvec
            }
            if (!first_coarse) loops++;
            fresh = first_coarse || nst == CG_RESTART;
            first_coarse = false;
            parity ^= 1;
        }
        maxseq = max(maxseq, seq);
        maxloops = max(maxloops, loops);
        // x of the own rows, and the step's Euler update (Blob::euler_integrate,
        // src/Blob.cpp:3937-3969) for a blob that had not failed before the
        // solve and whose solve converged
        const bool err = run && s_stop;
        const bool move = d.cg_euler && !err && s_cg.state == CG_CONVERGED && __ldcg(&d.status[b]) == 0;
        const double dt = s_bp.dt;
#pragma unroll
        for (int q = 0; q < R; q++) {
            if (!in[q]) continue;
            const int row = row0[q] + tid;
            if (run) {
#pragma unroll
                for (int k = 0; k < 3; k++) static_cast<T *>(d.x)[3 * (size_t)row + k] = state_of(q, 0, k);
            }
            if (!move || row - s_bp.node_off >= s_bp.node_cnt) continue;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const size_t kk = 3 * (size_t)row + k;
                const double xi = run ? (double)state_of(q, 0, k) : (double)static_cast<const T *>(d.x)[kk];
                double pn;
                if (nomass) {
                    d.vel[kk] = xi;
                    pn = d.pos[kk] + xi * dt;
                } else {
                    const double v = d.vel[kk] + xi * dt;
                    d.vel[kk] = v;
                    pn = d.pos[kk] + v * dt;
                }
                d.pos[kk] = pn;
                if (d.pos_df) d.pos_df[kk] = split_pos(pn);
            }
        }
        if (leader && tid == 0) {
            if (run) {
                d.cg[b] = s_cg;
                record_sums(d, b, s_last);  // (FP64 conversions: once per solve, off the iteration)
            }
            // the blob's own stream moves on by one step's draws unless the
            // blob failed (a shared stream: below)
            if (d.cg_euler && !err && d.num_streams == d.num_blobs && __ldcg(&d.status[b]) == 0) {
                advance_stream(d.stream_state + 6 * s_bp.stream, d.stream_step + s_bp.stream);
            }
        }
        if (err) {
            // the blobs of the tasks that are given up with this one have not
            // been solved either: all of them fail here
#pragma unroll 1
            for (int k = ti + tid; k < gb.ptr[blockIdx.x + 1]; k += NT)
                atomicOr(&d.status[d.seg_blob[gb.task[k]]], BLOB_FAIL_CG | BLOB_FAIL_TIMEOUT);
            break;  // CTA-uniform: s_stop was read after a barrier by every thread
        }
    }
    if constexpr (kTmem) {
        if (gb.tmem_slots > 0) {
            __syncthreads();
            if (warp == 0) tmem_free(s_tmem);
        }
    }
    if (tid == 0) {
        // a shared stream moves on whichever blobs failed (after a time-out
        // too: the draws of the blobs that were solved are used up)
        if (blockIdx.x == 0 && d.cg_euler && d.num_streams != d.num_blobs)
#pragma unroll 1
            for (int sm = 0; sm < d.num_streams; sm++)
                advance_stream(d.stream_state + 6 * sm, d.stream_step + sm);
        // the last CTA out moves the tag base past every tag of this launch
        // (all CTAs read it when they started) and adds the longest solve's
        // iterations to the loop count
        atomicMax(&d.bar[7], maxseq);
        atomicMax(&d.bar[8], (unsigned int)max(maxloops, 0));
        __threadfence();
        if (atomicAdd(&d.bar[9], 1u) == gridDim.x - 1) {
            __threadfence();
            d.bar[6] = base + atomicExch(&d.bar[7], 0u) + 1u;
            *d.loop_count += (unsigned long long)atomicExch(&d.bar[8], 0u);
            d.bar[9] = 0;
        }
    }
}

// The variant by the rows of a segment (the longest) and the segments of a CTA.
template <typename T, bool COARSE>
const void *kernel_for(const GroupBatch &g)
{
    if constexpr (sizeof(T) == 4)
        if (g.per > 1) return reinterpret_cast<const void *>(&k_cg_group<T, COARSE, 1024, 2>);
    if (g.rows <= 256) return reinterpret_cast<const void *>(&k_cg_group<T, COARSE, 256, 1>);
    if (g.rows <= 512) return reinterpret_cast<const void *>(&k_cg_group<T, COARSE, 512, 1>);
    return reinterpret_cast<const void *>(&k_cg_group<T, COARSE, 1024, 1>);
}

const void *group_kernel(const DeviceBatch &d, const GroupBatch &g)
{
    if (d.precision == PREC_FP64) return kernel_for<double, false>(g);
    return d.coarse ? kernel_for<float, true>(g) : kernel_for<float, false>(g);
}

}  // namespace

int cg_group_plan(const DeviceBatch &d, GroupBatch &g, int max_slots, int max_cols, int max_rows, int max_halo,
                  int max_segs)
{
    const bool f64 = d.precision == PREC_FP64;
    if (g.per > 1 && f64) return -1;
    g.rows = g.per > 1 || max_rows > 512 ? 1024 : max_rows > 256 ? 512 : 256;  // the variant's MAXT
    // (a lane for each segment whose sums are waited for)
    g.threads = std::max({256, (max_rows + 31) / 32 * 32, (max_segs + 31) / 32 * 32});
    if (g.threads > g.rows) return -1;
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return -1;
    const void *fn = group_kernel(d, g);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return -1;
    const size_t R = (size_t)g.per * g.rows, ts = f64 ? 8 : 4;
    const bool wide = g.per > 1;
    const size_t reserve = 1024;  // per-CTA system use
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 15) & ~(size_t)15;
        return (int32_t)o;
    };
    g.o_state = take(g.rows <= 512 ? 0 : 12 * R * ts);
    g.o_u = take(4 * (R + max_halo) * ts);
    g.o_halo = take(4 * (size_t)max_halo);
    g.o_words = take(d.coarse ? 48 * (size_t)max_segs : 0);
    if (d.coarse) {
        g.o_phi = take(wide ? 0 : 16 * R);
        g.o_xrow = take(wide ? 0 : 24 * (size_t)d.coarse_nmax);
        g.o_h = take(4 * (size_t)d.coarse_nmax);
    }
    const size_t fixed = fa.sharedSizeBytes + reserve + off + 64;
    if ((size_t)optin < fixed) return -1;
    size_t room = optin - fixed;
    const size_t per_col = R * sizeof(uint16_t), per_slot = R * (d.any_nomass ? 9 : 1) * ts;
    g.cache_cols = (int32_t)std::min<size_t>(room / per_col, (size_t)std::max(0, max_cols));
    room -= (size_t)g.cache_cols * per_col;
    g.cache_slots = (int32_t)std::min<size_t>(
        room / per_slot, (size_t)std::max(0, std::min(max_slots, (int)g.cache_cols)));
    g.o_col = take((size_t)g.cache_cols * per_col);
    g.o_kv2 = take(d.any_nomass ? 8 * ts * R * g.cache_slots : 0);
    g.o_kv1 = take(ts * R * g.cache_slots);
    g.tmem_slots = 0;
    if (g.rows > 256 && d.any_nomass) {
        // the warps of a quarter of the lanes share its columns.  The places
        // of a block in tensor memory are read from shared memory
        const int warps = (g.threads / 32 + 3) / 4;
        g.tmem_slots = std::min(kTmemCols / warps / g.per / (int)(9 * ts / 4),
                                std::min(max_slots, (int)g.cache_cols) - (int)g.cache_slots);
        // a CTA takes all of its SM's tensor memory: no second one beside it
        if (g.tmem_slots > 0) off = std::max<size_t>(off, (size_t)optin / 2 + 1024);
    }
    g.dyn_smem = (int32_t)off;
    // the limit is a property of the kernel, shared by every handle: the
    // device maximum, so that no handle's plan lowers another's
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes) !=
        cudaSuccess)
        return -1;
    return 0;
}

int cg_group_max_grid(const DeviceBatch &d, const GroupBatch &g)
{
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, group_kernel(d, g),
                                                      g.threads, g.dyn_smem) != cudaSuccess)
        return 0;
    return sms * per_sm;
}

cudaError_t launch_cg_group(const DeviceBatch &d, cudaStream_t s)
{
    GroupBatch g = *d.group;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g.grid);
    cfg.blockDim = dim3((unsigned)g.threads);
    cfg.dynamicSmemBytes = (size_t)g.dyn_smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DeviceBatch arg = d;
    void *args[] = {&arg, &g};
    count_launches(1);
    return cudaLaunchKernelExC(&cfg, group_kernel(d, g), args);
}

}  // namespace ffea
