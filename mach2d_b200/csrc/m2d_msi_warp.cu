// m2d_msi_warp.cu -- cluster wavefront MSI kernel (ny <= 1024).
//
// Same arithmetic as k_msi (m2d_msi.cu), spread over a thread-block cluster:
//   * rows are dealt in groups of 32 ("wavefront-major" planes: the 32 cells
//     (s - 2 l, 32 g + l), l = 0..31, of group g at step s are one contiguous
//     256-byte line), WPC groups per CTA and up to 16 CTAs per cluster;
//   * each group has three warps.  A front warp factorises line by line and
//     later runs the backward sweep; a forward warp on another SM
//     sub-partition follows it one batch behind with the first forward
//     sweep, reading the factors where the front warp left them; a mover
//     warp brings batches of LAG lines into a ring of shared-memory frames
//     and stores the finished ones, with bulk copies.  So the front warp,
//     whose recurrence sets the time, touches shared memory and registers
//     only: no global access, no copy and no proxy fence sits on it.  A
//     factorisation step takes 295 to 320 cycles (a one-warp probe of its
//     chain alone: 280) against 690 when one warp did everything, a backward
//     step 80 against 235; solves of 514x258 cells queued one after the other,
//     one iteration each, 327 us against 799 (nine diagonals 434 against 928);
//   * within a warp lane = row, and a row's value reaches the next row with
//     one shuffle per step.  The values of the last row travel to the next
//     group's ring (distributed shared memory) once a batch, as asynchronous
//     stores that complete on the consumer's mbarrier of that batch (one store
//     per step, on the recurrence, cost 90 cycles a step);
//   * divisions on the recurrence use reciprocal approximations refined
//     without a branch (m2d_div.cuh).  Idle warps check every factor afterwards
//     from its stored inputs: each quotient by its exact remainder, every
//     other value bit for bit; a factorisation that fails is repeated, with
//     its first sweep pair, with IEEE division before x changes.  The forward
//     sweep checks its own quotients and repeats a batch with IEEE division
//     where one fails;
//   * r = A x - b and its norm come with the transpose of A (k_skew, whole
//     GPU); after each sweep pair x += z and the new residual run on the
//     whole GPU on large grids and as cluster-wide passes on small ones.
// Cells outside the grid are unit rows with zero residual, so they produce
// the zeros of the reference's out-of-grid neighbours, and results stay
// bitwise equal to the lexicographic reference loop, but for the sign of a
// zero (x of a cell whose start value and residual are zeros can come back +0
// for -0).  Every wait is bounded in %globaltimer time (on timeout the kernel
// records ERR_SPIN_TIMEOUT and runs to its end).
#include <cstdint>
#include <type_traits>
#include <cooperative_groups.h>
#include "m2d_div.cuh"
#include "m2d_solvers.cuh"

namespace cg = cooperative_groups;

namespace m2d {

namespace {
constexpr int kThreads = 256;
constexpr int kMaxCluster = 16;
constexpr int kSkewPad = 62;      // slots per group = nx + 62 (slot s = i + 2 lane)
constexpr int kLine = 32;         // values per slot line, one per lane
constexpr int kRingSlots = 4;     // hand-off batches a channel holds
constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxIterUnbounded = 10000;
constexpr unsigned long long kWaitLimitNs = 4000000000ull;   // bound of every wait (4 s of %globaltimer)

// One frame = one batch (LAG lines) of every plane a phase touches.  The
// factorisation overwrites A in place: l1..l4, u and 1/l1 take the places
// behind A's first plane, which for nine diagonals is l5 itself.  The forward
// sweep keeps the residual (a batch may be repeated) and puts w beside it;
// z takes the place of w.
template <int ND, int LAG> struct Frame {
    static constexpr int NU = (ND == 9) ? 4 : 3;
    static constexpr int kR = 0, kA = 1;
    static constexpr int kL = (ND == 9) ? 2 : 1;
    static constexpr int kU = kL + 4, kY = kU + NU, kW = kY + 1, kPlanes = kW + 1;
    static constexpr int kBlock = LAG * kLine;    // elements of one plane
    // the group below is this many batches ahead: slot s needs its slot s + 63
    static constexpr int kAhead = 64 / LAG;
    static_assert(64 % LAG == 0 && LAG >= 4, "a batch divides the 64-slot lead of the group below");
};
}

#define PL(p, k, np) (p)[(long long)((k) - 1) * N + (np)]

__device__ __forceinline__ void stamp(const MsiLaunch &L, int rank, int k)
{
    if (L.prof && rank == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        L.prof[k] = t;
    }
}

// ---- bulk asynchronous copies into shared memory, completion on an mbarrier
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
template <typename T> __device__ __forceinline__ T lds_v(unsigned addr);
template <> __device__ __forceinline__ double lds_v<double>(unsigned addr)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
template <> __device__ __forceinline__ float lds_v<float>(unsigned addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ double shfl_up_v(double x)
{
    double v;
    asm volatile("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\t"
                 "shfl.sync.up.b32 lo, lo, 1, 0, -1;\n\tshfl.sync.up.b32 hi, hi, 1, 0, -1;\n\t"
                 "mov.b64 %0, {lo, hi};\n\t}" : "=d"(v) : "d"(x));
    return v;
}
// 1 for a zero or non-finite pivot, from the bits (no branch)
__device__ __forceinline__ unsigned pivot_bad(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return ((b << 1) == 0ull || ((unsigned)(b >> 52) & 0x7ffu) == 0x7ffu) ? 1u : 0u;
}
__device__ __forceinline__ unsigned pivot_bad(float x)
{
    const unsigned b = (unsigned)__float_as_int(x);
    return ((b << 1) == 0u || ((b >> 23) & 0xffu) == 0xffu) ? 1u : 0u;
}
__device__ __forceinline__ float shfl_up_v(float x)
{
    float v;
    asm volatile("shfl.sync.up.b32 %0, %1, 1, 0, -1;" : "=f"(v) : "f"(x));
    return v;
}
__device__ __forceinline__ float shfl_down_v(float x)
{
    float v;
    asm volatile("shfl.sync.down.b32 %0, %1, 1, 31, -1;" : "=f"(v) : "f"(x));
    return v;
}
__device__ __forceinline__ double shfl_down_v(double x)
{
    double v;
    asm volatile("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\t"
                 "shfl.sync.down.b32 lo, lo, 1, 31, -1;\n\tshfl.sync.down.b32 hi, hi, 1, 31, -1;\n\t"
                 "mov.b64 %0, {lo, hi};\n\t}" : "=d"(v) : "d"(x));
    return v;
}

// 32-bit shared::cluster address of the same variable in CTA `rank`
__device__ __forceinline__ unsigned cluster_addr(const void *p, int rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// whether phase `parity` has completed, without waiting
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// true once phase `parity` of the mbarrier has completed; false when
// limit_ns of %globaltimer time passed first
__device__ __forceinline__ bool mbar_wait_for(unsigned long long *bar, unsigned parity, unsigned long long limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
#pragma unroll 1
    for (;;) {
#pragma unroll 1
        for (int k = 0; k < 32; k++)
            if (mbar_try_wait(bar, parity)) return true;
        if (gtimer() - t0 > limit_ns) return false;
    }
}
// all lanes: bounded wait for the completion of phase `parity` (after an
// earlier timeout the warp no longer waits at all)
__device__ __forceinline__ void mbar_wait(unsigned long long *bar, unsigned parity, bool &timed_out)
{
    if (!timed_out && !mbar_wait_for(bar, parity, kWaitLimitNs)) timed_out = true;
    __syncwarp();
}
__device__ __forceinline__ void mbar_remote_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// generic-proxy global writes become visible to later bulk copies
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// wavefront-major slot of cell (i, j): warp j/32, step offset i + 2 (j%32), lane j%32
__device__ __forceinline__ long long skew_slot(int i, int j, int sw)
{
    return ((long long)(j >> 5) * sw + i + 2 * (j & 31)) * kLine + (j & 31);
}

// r = A x - b for one cell, in-range neighbours in ascending diagonal order
template <int ND>
__device__ __forceinline__ double residual_cell(const double *__restrict__ a, const double *__restrict__ b,
                                                const double *__restrict__ x, long long np, int i, int j, int nx,
                                                int ny, long long N)
{
    const bool w = i > 0, e = i < nx - 1, s = j > 0, n = j < ny - 1;
    double v = -b[np];
    if (ND == 9) {
        if (s && w) v = v + PL(a, 1, np) * x[np - nx - 1];
        if (s) v = v + PL(a, 2, np) * x[np - nx];
        if (s && e) v = v + PL(a, 3, np) * x[np - nx + 1];
        if (w) v = v + PL(a, 4, np) * x[np - 1];
        v = v + PL(a, 5, np) * x[np];
        if (e) v = v + PL(a, 6, np) * x[np + 1];
        if (n && w) v = v + PL(a, 7, np) * x[np + nx - 1];
        if (n) v = v + PL(a, 8, np) * x[np + nx];
        if (n && e) v = v + PL(a, 9, np) * x[np + nx + 1];
    } else {
        if (s) v = v + PL(a, 1, np) * x[np - nx];
        if (w) v = v + PL(a, 2, np) * x[np - 1];
        v = v + PL(a, 3, np) * x[np];
        if (e) v = v + PL(a, 4, np) * x[np + 1];
        if (n) v = v + PL(a, 5, np) * x[np + nx];
    }
    return v;
}

// r = A x - b over cells lo + threadIdx.x + kThreads k of [lo, hi), stored
// wavefront-major; returns this thread's sum of r^2 in cell order.  Four
// cells per round with their loads issued together.
template <int ND, typename TS>
__device__ __forceinline__ double residual_pass(const double *__restrict__ a, const double *__restrict__ b,
                                                const double *__restrict__ x, TS *__restrict__ r, long long lo,
                                                long long hi, int nx, int ny, int sw)
{
    const long long N = (long long)nx * ny;
    double acc = 0.0;
    long long np = lo + threadIdx.x;
    for (; np + 3 * kThreads < hi; np += 4 * kThreads) {
        double v[4];
        int ii[4], jj[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const long long c = np + q * kThreads;
            jj[q] = (int)((unsigned)c / (unsigned)nx);   // N < 2^31
            ii[q] = (int)c - jj[q] * nx;
            v[q] = residual_cell<ND>(a, b, x, c, ii[q], jj[q], nx, ny, N);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            r[skew_slot(ii[q], jj[q], sw)] = (TS)v[q];
            acc = acc + v[q] * v[q];
        }
    }
    for (; np < hi; np += kThreads) {
        const int j = (int)((unsigned)np / (unsigned)nx), i = (int)np - j * nx;
        const double v = residual_cell<ND>(a, b, x, np, i, j, nx, ny, N);
        r[skew_slot(i, j, sw)] = (TS)v;
        acc = acc + v * v;
    }
    return acc;
}

// Cluster-wide pass (this CTA takes a contiguous slice of cells): first
// x += z when z (wavefront-major) is given, then r = A x - b stored
// wavefront-major.  Returns the cluster-wide sum of r^2, identical in every
// thread.  Starts with a cluster barrier: every row's sweep must be final.
template <int ND, typename TS>
__device__ double cluster_residual(cg::cluster_group &cl, const double *__restrict__ a,
                                   const double *__restrict__ b, double *x, const TS *z, TS *r,
                                   int nx, int ny, int sw, double *red, double *part)
{
    cl.sync();
    const long long N = (long long)nx * ny;
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const long long per = (N + C - 1) / C;
    const long long lo = per * rank, hi = (lo + per < N) ? lo + per : N;
    if (z) {
        double *__restrict__ xw = x;
        const TS *__restrict__ zr = z;
#pragma unroll 8
        for (long long np = lo + threadIdx.x; np < hi; np += kThreads) {
            const int j = (int)((unsigned)np / (unsigned)nx), i = (int)np - j * nx;   // N < 2^31
            xw[np] = (double)zr[skew_slot(i, j, sw)] + xw[np];
        }
        cl.sync();
    }
    // x is final (read-only) from here on, and r is separate workspace
    const double acc = residual_pass<ND, TS>(a, b, x, r, lo, hi, nx, ny, sw);
    fence_async_global();   // the forward sweep reads r with bulk copies
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double *p0 = cl.map_shared_rank(part, 0);
        p0[rank] = red[0];
    }
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double s = 0.0;
        for (int c = 0; c < C; c++) s = s + part[c];
        for (int c = 0; c < C; c++) cl.map_shared_rank(part, c)[kMaxCluster] = s;
    }
    cl.sync();
    return part[kMaxCluster];
}

// One factorisation step of one cell (lu2d9 / lu2d5).  cb is the row of A
// (a unit row for an invalid cell), mw the own row's previous u, a1/a2/a3
// the row below's u at SE/S/SW.  FAST divides with quotients from refined
// reciprocal approximations (checked afterwards, line_ok), otherwise with '/'.
// Fill-in along a wall decays into the subnormals, so u takes the scaled
// remainders: without them one factorisation in six was repeated over 1500
// iterations of a 512x256 Euler nozzle, 2.69 s, none with them, 1.98 s; a solve
// that has no such fill-in takes 555 us instead of 551 (514x258, five
// diagonals, two iterations) and 715 instead of 711 (nine).
template <int ND, bool FAST>
__device__ __forceinline__ void lu_cell(const double (&cb)[ND], double alpha, const double *mw,
                                        const double *a1, const double *a2, const double *a3, double *l,
                                        double *u, double &y1)
{
    auto dv = [&](double n, double d) -> double { return FAST ? div_fast(n, d, rcp_start(d)) : n / d; };
    auto dr = [&](double n, double d) -> double { return FAST ? div_ready(n, d, rcp_start(d)) : n / d; };   // d comes early
    if (ND == 9) {
        const double b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        const double b6 = cb[5], b7 = cb[6], b8 = cb[7], b9 = cb[8];
        double l5 = b1;
        double l4 = dv(b2 - l5 * a3[0] - alpha * b3 * a1[0], 1.0 - alpha * a2[0] * a1[0]);
        double l3 = b3 - l4 * a2[0];
        double l2 = dr(b4 - l4 * a2[1] - l5 * a3[2] - 2.0 * alpha * l5 * a3[1], 1 + 2.0 * alpha * mw[1]);
        double phi1 = l3 * a1[0], phi2 = l5 * a3[1], phi3 = l3 * a1[3], phi4 = l2 * mw[1];
        double l1 = b5 - l2 * mw[0] - l3 * a1[1] - l4 * a2[2] - l5 * a3[3]
                  + alpha * (2.0 * phi1 + phi2 + phi3 + 2.0 * phi4);
        const double n0 = b6 - l3 * a1[2] - l4 * a2[3] - 2.0 * alpha * (phi1 + phi3);
        const double n1 = b7 - l2 * mw[2];
        const double n2 = b8 - l2 * mw[3] - alpha * phi4;
        if (FAST) {
            const Rcp r = rcp_start_scaled(l1);
            const double ls = l1 * 0x1p128;
            u[0] = div_scaled(n0, ls, r); u[1] = div_scaled(n1, ls, r);
            u[2] = div_scaled(n2, ls, r); u[3] = div_scaled(b9, ls, r);
        } else {
            u[0] = n0 / l1; u[1] = n1 / l1; u[2] = n2 / l1; u[3] = b9 / l1;
            y1 = __drcp_rn(l1);
        }
        l[0] = l1; l[1] = l2; l[2] = l3; l[3] = l4; l[4] = l5;
    } else {
        const double b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        double l4 = dv(b1, 1.0 - alpha * a2[0] * a1[0]);
        double l3 = -l4 * a2[0];
        double l2 = dr(b2 - l4 * a2[1], 1.0 + 2.0 * alpha * mw[1]);
        double phi1 = l3 * a1[0], phi4 = l2 * mw[1];
        double l1 = b3 - l2 * mw[0] - l3 * a1[1] - l4 * a2[2] + 2.0 * alpha * (phi1 + phi4);
        const double n0 = b4 - l3 * a1[2] - 2.0 * alpha * phi1;
        const double n1 = -l2 * mw[2];
        const double n2 = b5 - alpha * phi4;
        if (FAST) {
            const Rcp r = rcp_start_scaled(l1);
            const double ls = l1 * 0x1p128;
            u[0] = div_scaled(n0, ls, r); u[1] = div_scaled(n1, ls, r); u[2] = div_scaled(n2, ls, r);
        } else {
            u[0] = n0 / l1; u[1] = n1 / l1; u[2] = n2 / l1;
            y1 = __drcp_rn(l1);
        }
        l[0] = l1; l[1] = l2; l[2] = l3; l[3] = l4;
    }
}

// The same factorisation step in FP32 for the mixed-precision solve.  Its
// factors only precondition an FP64 iteration, so the operation order is
// free: fused multiply-adds and approximate reciprocals; y1 = 1/l1.
template <int ND>
__device__ __forceinline__ void lu_cell_f(const float (&cb)[ND], float alpha, const float *mw,
                                          const float *a1, const float *a2, const float *a3, float *l,
                                          float *u, float &y1)
{
    if (ND == 9) {
        const float b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        const float b6 = cb[5], b7 = cb[6], b8 = cb[7], b9 = cb[8];
        const float l5 = b1;
        const float l4 = __fdividef(fmaf(-alpha * b3, a1[0], fmaf(-l5, a3[0], b2)), fmaf(-alpha * a2[0], a1[0], 1.0f));
        const float l3 = fmaf(-l4, a2[0], b3);
        const float l2 = __fdividef(fmaf(-2.0f * alpha * l5, a3[1], fmaf(-l5, a3[2], fmaf(-l4, a2[1], b4))),
                                    fmaf(2.0f * alpha, mw[1], 1.0f));
        const float phi1 = l3 * a1[0], phi2 = l5 * a3[1], phi3 = l3 * a1[3], phi4 = l2 * mw[1];
        const float t = fmaf(-l5, a3[3], fmaf(-l4, a2[2], fmaf(-l3, a1[1], fmaf(-l2, mw[0], b5))));
        const float l1 = fmaf(alpha, 2.0f * phi1 + phi2 + phi3 + 2.0f * phi4, t);
        const float y = __fdividef(1.0f, l1);
        u[0] = fmaf(-2.0f * alpha, phi1 + phi3, fmaf(-l4, a2[3], fmaf(-l3, a1[2], b6))) * y;
        u[1] = fmaf(-l2, mw[2], b7) * y;
        u[2] = fmaf(-alpha, phi4, fmaf(-l2, mw[3], b8)) * y;
        u[3] = b9 * y;
        y1 = y;
        l[0] = l1; l[1] = l2; l[2] = l3; l[3] = l4; l[4] = l5;
    } else {
        const float b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        const float l4 = __fdividef(b1, fmaf(-alpha * a2[0], a1[0], 1.0f));
        const float l3 = -l4 * a2[0];
        const float l2 = __fdividef(fmaf(-l4, a2[1], b2), fmaf(2.0f * alpha, mw[1], 1.0f));
        const float phi1 = l3 * a1[0], phi4 = l2 * mw[1];
        const float t = fmaf(-l4, a2[2], fmaf(-l3, a1[1], fmaf(-l2, mw[0], b3)));
        const float l1 = fmaf(2.0f * alpha, phi1 + phi4, t);
        const float y = __fdividef(1.0f, l1);
        u[0] = fmaf(-2.0f * alpha, phi1, fmaf(-l3, a1[2], b4)) * y;
        u[1] = -l2 * mw[2] * y;
        u[2] = fmaf(-alpha, phi4, b5) * y;
        y1 = y;
        l[0] = l1; l[1] = l2; l[2] = l3; l[3] = l4;
    }
}

// ---- asynchronous stores to a neighbour's shared memory and bulk stores
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(addr), "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(addr), "r"(__float_as_int(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void sts_v(unsigned addr, double v)
{
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void sts_v(unsigned addr, float v)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void bulk_g2s(unsigned dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_s2g(void *dst, unsigned src, unsigned bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait()
{
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// progress words read across the cluster
__device__ __forceinline__ unsigned ld_cluster_acquire(unsigned addr)
{
    unsigned v;
    asm volatile("ld.acquire.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster_release(unsigned addr, unsigned v)
{
    asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// factorisations repeated with IEEE division on this device since load
__device__ unsigned long long g_lu_redo = 0;

// The check of one line of a factorisation: cell (s - 2 lane, 32 wg + lane)
// from its row of A and the stored u of its W, S, SE [and SW] neighbours
// (zero outside the grid).  If every cell passes, the stored factors are
// those of the IEEE recurrence (induction over the wavefront order).  The
// loads are whole lines: the cell's own values and the W neighbour's on the
// lines s and s-1, the S, SE and SW neighbours' one lane down on s-2, s-1,
// s-3 (lane 0: lane 31 of the group below on s+62, s+63, s+61).  They bypass
// L1: the lines were written by bulk stores of this launch.
template <int ND>
__device__ __forceinline__ bool line_ok(const double *asp, const double *dl, const double *du, const double *rl,
                                        int nx, int ny, int sw, long long PS, int wg, int s)
{
    constexpr int NU = (ND == 9) ? 4 : 3;
    const int lane = threadIdx.x & 31;
    const int j = 32 * wg + lane, i = s - 2 * lane;
    if (j >= ny || i < 0 || i >= nx) return true;
    const long long P = ((long long)wg * sw + s) * kLine + lane;
    const long long B = (lane > 0) ? P - 1 : ((long long)(wg - 1) * sw + s + 64) * kLine + 31;
    double cb[ND], l[4], u[NU], mw[NU], a1[NU], a2[NU], a3[NU];
#pragma unroll
    for (int k = 0; k < ND; k++) cb[k] = __ldcg(asp + k * PS + P);
#pragma unroll
    for (int k = 0; k < 4; k++) l[k] = __ldcg(dl + k * PS + P);
#pragma unroll
    for (int q = 0; q < NU; q++) {
        u[q] = __ldcg(du + q * PS + P);
        mw[q] = (i >= 1) ? __ldcg(du + q * PS + P - kLine) : 0.0;
        a2[q] = (j >= 1) ? __ldcg(du + q * PS + B - 2 * kLine) : 0.0;
        a1[q] = (j >= 1 && i + 1 <= nx - 1) ? __ldcg(du + q * PS + B - kLine) : 0.0;
        a3[q] = (ND == 9 && j >= 1 && i >= 1) ? __ldcg(du + q * PS + B - 3 * kLine) : 0.0;
    }
    const double y = __ldcg(rl + P);
    const double alpha = (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2) ? 0.5 : 0.0;
    auto same = [](double p, double q) { return __double_as_longlong(p) == __double_as_longlong(q); };
    const double l1 = l[0], l2 = l[1], l3 = l[2], l4 = l[3];
    bool ok;
    // the expressions of lu_cell, with the stored quotients in place
    if (ND == 9) {
        const double b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        const double b6 = cb[5], b7 = cb[6], b8 = cb[7], b9 = cb[8];
        const double l5 = b1;
        ok = quot_ok(b2 - l5 * a3[0] - alpha * b3 * a1[0], 1.0 - alpha * a2[0] * a1[0], l4);
        ok = ok & same(l3, b3 - l4 * a2[0]);
        ok = ok & quot_ok(b4 - l4 * a2[1] - l5 * a3[2] - 2.0 * alpha * l5 * a3[1], 1 + 2.0 * alpha * mw[1], l2);
        const double phi1 = l3 * a1[0], phi2 = l5 * a3[1], phi3 = l3 * a1[3], phi4 = l2 * mw[1];
        ok = ok & same(l1, b5 - l2 * mw[0] - l3 * a1[1] - l4 * a2[2] - l5 * a3[3]
                                + alpha * (2.0 * phi1 + phi2 + phi3 + 2.0 * phi4));
        ok = ok & quot_ok(b6 - l3 * a1[2] - l4 * a2[3] - 2.0 * alpha * (phi1 + phi3), l1, u[0]);
        ok = ok & quot_ok(b7 - l2 * mw[2], l1, u[1]);
        ok = ok & quot_ok(b8 - l2 * mw[3] - alpha * phi4, l1, u[2]);
        ok = ok & quot_ok(b9, l1, u[3]);
    } else {
        const double b1 = cb[0], b2 = cb[1], b3 = cb[2], b4 = cb[3], b5 = cb[4];
        ok = quot_ok(b1, 1.0 - alpha * a2[0] * a1[0], l4);
        ok = ok & same(l3, -l4 * a2[0]);
        ok = ok & quot_ok(b2 - l4 * a2[1], 1.0 + 2.0 * alpha * mw[1], l2);
        const double phi1 = l3 * a1[0], phi4 = l2 * mw[1];
        ok = ok & same(l1, b3 - l2 * mw[0] - l3 * a1[1] - l4 * a2[2] + 2.0 * alpha * (phi1 + phi4));
        ok = ok & quot_ok(b4 - l3 * a1[2] - 2.0 * alpha * phi1, l1, u[0]);
        ok = ok & quot_ok(-l2 * mw[2], l1, u[1]);
        ok = ok & quot_ok(b5 - alpha * phi4, l1, u[2]);
    }
    return ok & quot_ok(1.0, l1, y);
}

// lagged factorisation (MsiLaunch::lag_max): does this solve reuse the
// factors in its workspace?  Read by the transpose and by every thread of
// the solve before anything writes the record, so all agree.
template <typename TS>
__device__ __forceinline__ bool lag_reuse(const MsiLaunch &L, const MsiSys &S)
{
    if (std::is_same<TS, double>::value || L.lag_max <= 0 || !S.lag || L.reuse_lu || L.apply_only) return false;
    return S.lag[0] == S.tag && S.lag[1] >= 1 && S.lag[1] < L.lag_max;
}

constexpr int kExtBlocks = 296;
constexpr int kSkewParts = 512;                  // block sums of the initial residual
constexpr long long kExtMinCells = 1LL << 16;
constexpr int kExtTimedOut = 1, kExtLagged = 2, kExtBadPivot = 4;   // status bits of the first launch

// the scratch behind the wavefront-major planes
struct ExtWords {
    double *part0;                // k_skew's block sums of the initial residual
    double *partB;                // block sums of the new residual
    unsigned *cntB;               // finished blocks of that reduction
    int *status;                  // kExt* bits from the first launch
    int *done;                    // the stopping test passed (or the solve must stop)
};
__device__ __forceinline__ ExtWords ext_words(const MsiSys &S, int nd, int nx, int ny)
{
    const long long PS = (long long)((ny + 31) / 32) * (nx + kSkewPad) * kLine;
    double *e = S.ws + (long long)(nd == 9 ? 21 : 15) * PS;
    ExtWords w;
    w.part0 = e;
    w.partB = e + kSkewParts;
    w.cntB = reinterpret_cast<unsigned *>(e + kSkewParts + kExtBlocks);
    w.status = reinterpret_cast<int *>(e + kSkewParts + kExtBlocks + 1);
    w.done = reinterpret_cast<int *>(e + kSkewParts + kExtBlocks + 2);
    return w;
}
static_assert(kSkewParts + kExtBlocks + 3 <= kMsiExtScratch, "scratch words fit");

// The start of a solve, on the whole GPU: A (plane-major, cell order) to
// wavefront-major planes of element type TS, and r = A x - b of the same
// cells with its sum of squares.  Line (w, s) lane l holds cell
// (s - 2 l, 32 w + l); cells outside the grid become unit rows with r = 0.
// A CTA takes tiles of 32 rows x kSkewTile lines: row r of a tile is
// kSkewTile consecutive cells (its start shifted by 2 r), so the reads are
// coalesced and none is wasted.  A thread's cells load every plane before
// the first transpose, so that a tile costs one memory latency and not one
// per plane (a solve of 82x42 cells spent 15 us here with a load and a
// barrier per plane); the planes then go through a shared-memory transpose
// (two buffers, one barrier per plane) to whole lines.  Modes: with factors
// reused (MsiLaunch::reuse_lu, or a lagged solve) only r; with apply_only
// r = -b.  Grid: (blocks over line tiles, row groups, systems),
// gridDim.x * gridDim.y <= kSkewParts.
constexpr int kSkewTile = 32;
template <int ND, typename TS>
__global__ void __launch_bounds__(256, 2) k_skew(MsiLaunch L)
{
    constexpr int NL = (ND == 9) ? 5 : 4, NU = (ND == 9) ? 4 : 3;
    constexpr int DIAG = (ND == 9) ? 4 : 2;
    constexpr int M = 32 * kSkewTile / 256;      // cells per thread: rows r0 + 8 m
    __shared__ double tile[2][kSkewTile][33];
    __shared__ double red[8];
    const MsiSys S = L.s[blockIdx.z];
    const ExtWords ew = ext_words(S, ND, L.nx, L.ny);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        // the whole-GPU passes after the sweeps start from a clean state
        *ew.status = 0;
        *ew.done = 0;
    }
    const bool planes = !(L.reuse_lu || lag_reuse<TS>(L, S));
    const bool rhs_only = L.apply_only != 0;
    const int nx = L.nx, ny = L.ny;
    const long long N = (long long)nx * ny;
    const int SW = nx + kSkewPad;
    const long long PS = (long long)((ny + 31) / 32) * SW * kLine;
    TS *rp = reinterpret_cast<TS *>(S.ws) + (long long)(NL + NU + 1) * PS;
    TS *as = reinterpret_cast<TS *>(S.ws) + (long long)(NL + NU + 3) * PS;
    const int w = blockIdx.y, t = threadIdx.x & 31, r0 = threadIdx.x >> 5;
    const double *__restrict__ a = S.a;
    const double *__restrict__ b = S.b;
    const double *__restrict__ x = S.x;
    double sum = 0.0;
    int buf = 0;
    for (int c0 = blockIdx.x * kSkewTile; c0 < SW; c0 += gridDim.x * kSkewTile) {
        double acc[M], v[ND][M];
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int j = 32 * w + r0 + 8 * m, i = c0 + t - 2 * (r0 + 8 * m);
            const bool ok = j < ny && i >= 0 && i < nx;
            const bool hw = i > 0, he = i < nx - 1, hs = j > 0, hn = j < ny - 1;
            const long long np = (long long)j * nx + i;
            acc[m] = ok ? -b[np] : 0.0;
            if (rhs_only) continue;
            double xv[ND];
#pragma unroll
            for (int k = 0; k < ND; k++) {
                const int di = (ND == 9) ? k % 3 - 1 : (k == 1 ? -1 : (k == 3 ? 1 : 0));
                const int dj = (ND == 9) ? k / 3 - 1 : (k == 0 ? -1 : (k == 4 ? 1 : 0));
                const bool in = ok && (di >= 0 || hw) && (di <= 0 || he) && (dj >= 0 || hs) && (dj <= 0 || hn);
                v[k][m] = ok ? a[k * N + np] : (k == DIAG ? 1.0 : 0.0);
                xv[k] = in ? x[np + (long long)dj * nx + di] : 0.0;
            }
            // in-range neighbours in ascending diagonal order; the others add
            // nothing, not even a zero's sign
#pragma unroll
            for (int k = 0; k < ND; k++) {
                const int di = (ND == 9) ? k % 3 - 1 : (k == 1 ? -1 : (k == 3 ? 1 : 0));
                const int dj = (ND == 9) ? k / 3 - 1 : (k == 0 ? -1 : (k == 4 ? 1 : 0));
                const bool in = ok && (di >= 0 || hw) && (di <= 0 || he) && (dj >= 0 || hs) && (dj <= 0 || hn);
                const double s1 = acc[m] + v[k][m] * xv[k];
                acc[m] = in ? s1 : acc[m];
            }
        }
        auto put = [&](const double (&d)[M], TS *dst) {
#pragma unroll
            for (int m = 0; m < M; m++) tile[buf][t][r0 + 8 * m] = d[m];
            __syncthreads();
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int q = r0 + 8 * m, s = c0 + q;
                if (s < SW) dst[((long long)w * SW + s) * kLine + t] = (TS)tile[buf][q][t];
            }
            buf ^= 1;   // the other buffer's readers passed this barrier
        };
        if (planes && !rhs_only) {
#pragma unroll
            for (int k = 0; k < ND; k++) put(v[k], as + k * PS);
        }
        put(acc, rp);
#pragma unroll
        for (int m = 0; m < M; m++) sum = sum + acc[m] * acc[m];
    }
    if (rhs_only) return;
    // this block's share of |r|^2, by a fixed tree
    for (int o = 16; o > 0; o >>= 1) sum = sum + __shfl_down_sync(kFull, sum, o);
    if (t == 0) red[r0] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double q = red[0];
        for (int k = 1; k < 8; k++) q = q + red[k];
        ew.part0[blockIdx.y * gridDim.x + blockIdx.x] = q;
    }
}
// blocks of k_skew over the line tiles of one row group
static int skew_blocks(int nx, int ny)
{
    const int tiles = (nx + kSkewPad + kSkewTile - 1) / kSkewTile, groups = (ny + 31) / 32;
    return tiles < kSkewParts / groups ? tiles : kSkewParts / groups;
}

// An application of stored factors (MsiLaunch::apply_only) ends with
// x += z from the sweep-result plane as one whole-GPU pass.  Grid: (cell
// blocks, systems).
template <int ND, typename TS>
__global__ void k_unskew_add(MsiLaunch L)
{
    const MsiSys S = L.s[blockIdx.y];
    const int nx = L.nx, ny = L.ny;
    const int NL = (ND == 9) ? 5 : 4, NU = (ND == 9) ? 4 : 3;
    const int SW = nx + kSkewPad;
    const long long PS = (long long)((ny + 31) / 32) * SW * kLine;
    const TS *z = reinterpret_cast<const TS *>(S.ws) + (long long)(NL + NU + 2) * PS;
    const long long N = (long long)nx * ny;
    for (long long np = blockIdx.x * (long long)blockDim.x + threadIdx.x; np < N;
         np += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(np / nx), i = (int)(np - (long long)j * nx);
        S.x[np] = (double)z[skew_slot(i, j, SW)] + S.x[np];
    }
}

// ---- whole-GPU residual passes (MsiLaunch::ext).  On a large grid the
// passes over all cells after a sweep pair (x += z, the new residual, its
// norm) run on the cluster's 9-16 SMs far below what the whole GPU moves
// (47 us at 514x258 with five diagonals against 12 here).  So the first two
// iterations are launches of one sweep pair each, with these kernels behind
// them on every SM, and a last launch of the cluster kernel iterates further;
// all of them return at once when an earlier iteration met the stopping test.
// Reductions are deterministic: kExtBlocks blocks take fixed contiguous
// shares, a thread sums its cells in order, a block adds its threads' sums by
// a fixed tree, and the last block to finish adds the block sums in index
// order (from shared memory: one thread reading them one after the other from
// global memory took most of the pass).

// The deterministic sum of r^2, r = A x - b (kept, wavefront-major, for the
// next iteration): the total in thread 0 of the last block to finish (last =
// true there), after resetting the counter.
template <int ND, typename TS>
__device__ double ext_residual(const MsiSys &S, int nx, int ny, TS *__restrict__ r, double *part, unsigned *cnt,
                               bool &last)
{
    __shared__ double red[kExtBlocks];
    __shared__ bool is_last;
    const long long N = (long long)nx * ny;
    const int SW = nx + kSkewPad;
    const long long per = (N + kExtBlocks - 1) / kExtBlocks;
    const long long lo = per * blockIdx.x, hi = (lo + per < N) ? lo + per : N;
    double acc = 0.0;
    for (long long np = lo + threadIdx.x; np < hi; np += blockDim.x) {
        const int j = (int)((unsigned)np / (unsigned)nx), i = (int)np - j * nx;   // N < 2^31
        const double v = residual_cell<ND>(S.a, S.b, S.x, np, i, j, nx, ny, N);
        r[skew_slot(i, j, SW)] = (TS)v;
        acc = acc + v * v;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[blockIdx.x] = red[0];
        __threadfence();
        is_last = atomicAdd(cnt, 1u) == (unsigned)gridDim.x - 1u;
    }
    __syncthreads();
    last = is_last && threadIdx.x == 0;
    double total = 0.0;
    if (is_last) {
        __threadfence();
        for (int k = threadIdx.x; k < kExtBlocks; k += blockDim.x) red[k] = __ldcg(part + k);
        __syncthreads();
        if (last) {
#pragma unroll 8
            for (int k = 0; k < kExtBlocks; k++) total = total + red[k];
            *cnt = 0u;
        }
    }
    return total;
}

// x += z after a sweep pair; zeroes the counter of the next pass.  Grid
// (blocks, systems).
template <int ND, typename TS>
__global__ void k_ext_update(MsiLaunch L)
{
    const MsiSys S = L.s[blockIdx.y];
    const int nx = L.nx, ny = L.ny;
    constexpr int NL = (ND == 9) ? 5 : 4, NU = (ND == 9) ? 4 : 3;
    const int SW = nx + kSkewPad;
    const long long PS = (long long)((ny + 31) / 32) * SW * kLine;
    const TS *z = reinterpret_cast<const TS *>(S.ws) + (long long)(NL + NU + 2) * PS;
    const ExtWords w = ext_words(S, ND, nx, ny);
    if (*w.done) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *w.cntB = 0u;
    const long long N = (long long)nx * ny;
    for (long long np = blockIdx.x * (long long)blockDim.x + threadIdx.x; np < N;
         np += (long long)gridDim.x * blockDim.x) {
        const int j = (int)((unsigned)np / (unsigned)nx), i = (int)np - j * nx;   // N < 2^31
        S.x[np] = (double)z[skew_slot(i, j, SW)] + S.x[np];
    }
}

// the new residual, its norm and the stopping test of iteration nit0 + 1;
// when the solve ends here the last block also writes the factor record.
// Grid (kExtBlocks, systems).
template <int ND, typename TS>
__global__ void __launch_bounds__(256) k_ext_resid(MsiLaunch L)
{
    const MsiSys S = L.s[blockIdx.y];
    const int nx = L.nx, ny = L.ny;
    constexpr int NL = (ND == 9) ? 5 : 4, NU = (ND == 9) ? 4 : 3;
    const long long PS = (long long)((ny + 31) / 32) * (nx + kSkewPad) * kLine;
    TS *rp = reinterpret_cast<TS *>(S.ws) + (long long)(NL + NU + 1) * PS;
    const ExtWords w = ext_words(S, ND, nx, ny);
    if (*w.done) return;   // (written below only after every block came by here)
    bool last;
    const double rr = ext_residual<ND, TS>(S, nx, ny, rp, w.partB, w.cntB, last);
    if (!last) return;
    const double rr0 = S.rr[0];
    S.rr[1] = rr;
    const int st = *w.status, nit = L.nit0 + 1;
    const int cap = (L.nitm > 0) ? L.nitm : kMaxIterUnbounded;
    const bool done = (st & kExtTimedOut) || sqrt(rr) < L.tol * sqrt(rr0) || cap == nit;
    *w.done = done ? 1 : 0;
    if (done && !std::is_same<TS, double>::value && L.lag_max > 0 && S.lag) {
        const bool lagged = (st & kExtLagged) != 0;
        const bool renew = (st & (kExtTimedOut | kExtBadPivot)) != 0 || (lagged && nit > 1);
        const int age = S.lag[1];
        S.lag[0] = S.tag;
        S.lag[1] = renew ? L.lag_max : (lagged ? age + 1 : 1);
    }
}

// One direction of hand-offs between neighbouring row groups: batches of LAG
// values (V of them per line) in a ring of kRingSlots slots in the consumer's
// shared memory, with a slot of zeros behind it.  The producer's lanes ship a
// batch with asynchronous stores that complete on the slot's full barrier,
// which the consumer armed with the batch's bytes; the consumer frees the
// slot by arriving on the producer's empty barrier.  A ready barrier still
// costs about 125 cycles to wait for, so the warps test the barriers of their
// next batch two or three steps before the current one ends (no earlier: a
// group would have to trail its neighbour by as much to pass) and wait only
// where that failed.
template <typename TS, int LAG, int V> struct Channel {
    static constexpr unsigned kBytes = LAG * V * sizeof(TS);
    TS *ring;
    unsigned long long *full, *empty;
    unsigned dst = 0, dst_full = 0, rel = 0;   // consumer's ring and full barriers, producer's empty barriers
    int in = 0, out = 0;                       // batches received and sent
    __device__ __forceinline__ unsigned slot(int seq) const
    {
        return smem_u32(ring) + (unsigned)(seq & (kRingSlots - 1)) * kBytes;
    }
    __device__ __forceinline__ unsigned zeros() const { return smem_u32(ring) + kRingSlots * kBytes; }
    // nothing is armed after a timeout: a barrier whose batch never came stays as it is
    __device__ __forceinline__ void arm(int seq, bool timed_out) const
    {
        if ((threadIdx.x & 31) == 0 && !timed_out) mbar_arrive_tx(&full[seq & (kRingSlots - 1)], kBytes);
    }
    __device__ __forceinline__ bool arrived(int seq) const
    {
        return mbar_test(smem_u32(&full[seq & (kRingSlots - 1)]), (unsigned)(seq / kRingSlots) & 1u);
    }
    __device__ __forceinline__ void receive(int seq, bool &timed_out) const
    {
        mbar_wait(&full[seq & (kRingSlots - 1)], (unsigned)(seq / kRingSlots) & 1u, timed_out);
    }
    __device__ __forceinline__ void release(int seq) const
    {
        if ((threadIdx.x & 31) == 0) mbar_remote_arrive(rel + (unsigned)(seq & (kRingSlots - 1)) * 8u);
    }
    __device__ __forceinline__ void wait_free(int seq, bool &timed_out) const
    {
        if (seq >= kRingSlots)
            mbar_wait(&empty[seq & (kRingSlots - 1)], (unsigned)(seq / kRingSlots - 1) & 1u, timed_out);
    }
    // lane k < LAG ships line k's values (value v of the line from plane v of
    // the frame, `planes` bytes apart)
    __device__ __forceinline__ void send(int seq, unsigned line, unsigned planes) const
    {
        const unsigned k = threadIdx.x & 31, so = (unsigned)(seq & (kRingSlots - 1));
        if (k < LAG) {
#pragma unroll
            for (int v = 0; v < V; v++)
                st_async(dst + so * kBytes + (k * V + (unsigned)v) * (unsigned)sizeof(TS),
                         lds_v<TS>(line + k * kLine * (unsigned)sizeof(TS) + (unsigned)v * planes), dst_full + so * 8u);
        }
    }
};

// TS = double: the reference's FP64 algorithm, bitwise.  TS = float: the
// factors and both sweeps in FP32 inside the FP64 iteration (residual, x,
// norm and stopping test stay FP64): iterative refinement preconditioned by
// the FP32 factorisation.
template <int ND, int WPC, int NF, typename TS, int LAG>
__global__ void __launch_bounds__(kThreads, 1) k_msi_c(MsiLaunch L)
{
    using F = Frame<ND, LAG>;
    constexpr bool EXACT = std::is_same<TS, double>::value;
    constexpr int NU = F::NU, NL = (ND == 9) ? 5 : 4;
    constexpr unsigned ES = sizeof(TS);
    constexpr int kBlock = F::kBlock, P = F::kAhead;
    constexpr unsigned kFrameBytes = F::kPlanes * kBlock * ES;
    static_assert(WPC == 1 || WPC == 2, "one or two row groups per CTA");
    // hand-off rings from the neighbour groups (one slot more, of zeros) and
    // their barriers: "full" here, "empty" at the producer
    __shared__ __align__(16) TS ring_lu[WPC][(kRingSlots + 1) * LAG * NU];   // from below: u
    __shared__ __align__(16) TS ring_fw[WPC][(kRingSlots + 1) * LAG];        // from below: w
    __shared__ __align__(16) TS ring_bw[WPC][(kRingSlots + 1) * LAG];        // from above: z
    __shared__ unsigned long long full_lu[WPC][kRingSlots], empty_lu[WPC][kRingSlots];
    __shared__ unsigned long long full_fw[WPC][kRingSlots], empty_fw[WPC][kRingSlots];
    __shared__ unsigned long long full_bw[WPC][kRingSlots], empty_bw[WPC][kRingSlots];
    // frames: loaded (mover), factorised (front), finished with (forward or front)
    __shared__ unsigned long long f_full[WPC][NF], f_lu[WPC][NF], f_done[WPC][NF];
    __shared__ unsigned long long f_turn[WPC];    // the forward sweep is over
    __shared__ unsigned long long idle_bar;       // nothing ever arrives on it (test hook)
    __shared__ unsigned vbad;                     // a factor is not its IEEE value
    __shared__ unsigned prog[WPC];                // batches whose factors are in global memory
    __shared__ int chk_next;                      // next batch to check
    __shared__ double red[kThreads];
    __shared__ double part[kMaxCluster + 1];
    __shared__ double rr0_s;
    extern __shared__ __align__(128) double stage_raw[];   // WPC x NF frames
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int sys = blockIdx.x / C;
    const MsiSys S = L.dev ? L.dev[sys] : L.s[sys];
    const int nx = L.nx, ny = L.ny;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    // roles: warp w runs on SM sub-partition w % 4, so front and forward
    // warps have theirs to themselves but for idle and checking warps
    const bool front = wl < WPC, fwd = !front && wl < 2 * WPC;
    const bool mover = (WPC == 1) ? wl == 2 : wl >= 6;
    const int fw = front ? wl : fwd ? wl - WPC : (mover && WPC == 2) ? wl - 6 : 0;
    const int NG = (ny + 31) / 32;                // row groups
    const int wg = rank * WPC + fw;               // this warp's
    const int j = wg * 32 + lane;
    const int SW = nx + kSkewPad;                 // lines per group
    const long long PS = (long long)NG * SW * kLine;   // one wavefront-major plane
    // batches of a group: to its last row's last cell
    auto batches = [&](int g) { return (nx + 2 * (min(32, ny - 32 * g) - 1) + LAG - 1) / LAG; };
    const int nb = wg < NG ? batches(wg) : 0;
    const bool has_below = wg < NG && wg > 0, has_above = wg + 1 < NG;
    const int nb_below = has_below ? batches(wg - 1) : 0, nb_above = has_above ? batches(wg + 1) : 0;
    // hand-offs going up: batches P-1 .. up_last of the producer; going down:
    // batches dn_top .. 0
    const int up_last_in = has_below ? min(nb_below - 1, nb - 1 + P) : -1;
    const int up_last_out = has_above ? min(nb - 1, nb_above - 1 + P) : -1;
    const int dn_top_in = has_above ? min(nb - P, nb_above - 1) : -1;
    const int dn_top_out = has_below ? min(nb_below - P, nb - 1) : -1;
    const double *__restrict__ a = S.a;
    double *x = S.x;
    // wavefront-major planes of TS: dl1..dl4 (the fifth stays free: dl5 is A's
    // first plane), du1..duNU, 1/dl1, residual, sweep result, then A
    TS *dlp = reinterpret_cast<TS *>(S.ws);
    TS *dup = dlp + NL * PS;
    TS *rl1 = dup + NU * PS;
    TS *rp = rl1 + PS;
    TS *wp = rp + PS;
    TS *asp = wp + PS;
    const long long line0 = (long long)wg * SW;

    // a further launch of a solve with whole-GPU passes: nothing to do when an
    // earlier iteration already met the stopping test (every CTA of a cluster
    // reads the same word, so all return before any cluster barrier)
    const bool cont = L.nit0 > 0;
    const ExtWords ew = ext_words(S, ND, nx, ny);
    if (cont) {
        if (L.nit0 == 1) stamp(L, rank, 5);
        if (*ew.done) {
            stamp(L, rank, 6);
            return;
        }
    }
    if (threadIdx.x == 0) {
        vbad = 0u;
        chk_next = 0;
        mbar_init(&idle_bar, 1);
    }
    if (threadIdx.x < WPC) {
        const int f = threadIdx.x;
        prog[f] = 0u;
        mbar_init(&f_turn[f], 1);
        for (int q = 0; q < kRingSlots; q++) {
            mbar_init(&full_lu[f][q], 1); mbar_init(&empty_lu[f][q], 1);
            mbar_init(&full_fw[f][q], 1); mbar_init(&empty_fw[f][q], 1);
            mbar_init(&full_bw[f][q], 1); mbar_init(&empty_bw[f][q], 1);
        }
        for (int q = 0; q < NF; q++) {
            mbar_init(&f_full[f][q], 1); mbar_init(&f_lu[f][q], 1); mbar_init(&f_done[f][q], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int k = threadIdx.x; k < WPC * LAG * NU; k += kThreads) {
        const int f = k / (LAG * NU), e = k - f * (LAG * NU);
        ring_lu[f][kRingSlots * LAG * NU + e] = (TS)0;
        if (e < LAG) ring_fw[f][kRingSlots * LAG + e] = ring_bw[f][kRingSlots * LAG + e] = (TS)0;
    }
    if (wl == 7) {
        // |r0|^2 from k_skew's block sums, in the same fixed order in every CTA
        double v = 0.0;
        if (cont) v = lane == 0 ? S.rr[0] : 0.0;
        else if (!L.apply_only)
            for (int k = lane; k < L.nparts; k += 32) v = v + ew.part0[k];
        for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(kFull, v, o);
        if (lane == 0) rr0_s = v;
    }
    const unsigned frames = smem_u32(stage_raw) + (unsigned)fw * NF * kFrameBytes;
    // lagged factorisation: reuse the workspace's factors (decided from the
    // record as the launch found it; rank 0 rewrites it at the end)
    const bool lagged = lag_reuse<TS>(L, S);
    const int lag_age = lagged ? S.lag[1] : 0;
    const bool reuse = L.reuse_lu || lagged || cont;
    cl.sync();   // barriers initialised before any use
    bool bad_pivot = false, timed_out = false, hook_ran_out = false;
    int use = 0;                 // frame uses so far (all roles of a group count alike)
    int lu_uses = 0;             // factorised batches so far
    int turns = 0;               // sweep pairs so far
    bool nit_first = true;
    stamp(L, rank, 0);

    auto wait_frame = [&](unsigned long long *bar, int u) {
        mbar_wait(&bar[u % NF], (unsigned)(u / NF) & 1u, timed_out);
    };
    auto frame_ready = [&](unsigned long long *bar, int u) {
        return mbar_test(smem_u32(&bar[u % NF]), (unsigned)(u / NF) & 1u);
    };
    // hand-off channels: up for the factorisation (front warp) and the forward
    // sweep (forward warp), down for the backward sweep
    Channel<TS, LAG, NU> ch_lu{&ring_lu[fw][0], full_lu[fw], empty_lu[fw]};
    Channel<TS, LAG, 1> ch_fw{&ring_fw[fw][0], full_fw[fw], empty_fw[fw]};
    Channel<TS, LAG, 1> ch_bw{&ring_bw[fw][0], full_bw[fw], empty_bw[fw]};
    {
        const int up_cta = (fw + 1 < WPC) ? rank : rank + 1, up_f = (fw + 1 < WPC) ? fw + 1 : 0;
        const int dn_cta = (fw > 0) ? rank : rank - 1, dn_f = (fw > 0) ? fw - 1 : WPC - 1;
        if (has_above) {
            ch_lu.dst = cluster_addr(&ring_lu[up_f][0], up_cta);
            ch_lu.dst_full = cluster_addr(&full_lu[up_f][0], up_cta);
            ch_fw.dst = cluster_addr(&ring_fw[up_f][0], up_cta);
            ch_fw.dst_full = cluster_addr(&full_fw[up_f][0], up_cta);
            ch_bw.rel = cluster_addr(&empty_bw[up_f][0], up_cta);
        }
        if (has_below) {
            ch_lu.rel = cluster_addr(&empty_lu[dn_f][0], dn_cta);
            ch_fw.rel = cluster_addr(&empty_fw[dn_f][0], dn_cta);
            ch_bw.dst = cluster_addr(&ring_bw[dn_f][0], dn_cta);
            ch_bw.dst_full = cluster_addr(&full_bw[dn_f][0], dn_cta);
        }
    }
    // up-going sends start with batch P-1: the consumer's first lines need it
    auto sends_up = [&](int b) { return has_above && b >= P - 1 && b <= up_last_out; };

    // ---- incomplete LU (lu2d9 msi2d9-v03.f90:277-432, lu2d5 msi2d5-v03.f90:247-330),
    // front warp.  A step's shuffles of the previous step's u come first, then
    // the previous step's stores and the next step's loads, then its
    // arithmetic; nothing in it branches.  IEEE = true: '/' throughout, and
    // cells outside the grid forced to zero.
    auto run_lu = [&](auto ieee_tag) {
        constexpr bool IEEE = decltype(ieee_tag)::value;
        unsigned piv = 0;                              // a zero or non-finite pivot was seen
        TS mw[NU], a1[NU], a2[NU], a3[NU], carry[NU];
        unsigned rb = ch_lu.zeros();
        const bool any_in = P - 1 <= up_last_in;
        if (any_in) {
            ch_lu.arm(ch_lu.in, timed_out);
            ch_lu.receive(ch_lu.in, timed_out);
            rb = ch_lu.slot(ch_lu.in);
        }
#pragma unroll
        for (int q = 0; q < NU; q++) {
            const TS v = lds_v<TS>(rb + (unsigned)((LAG - 2) * NU + q) * ES);
            carry[q] = lds_v<TS>(rb + (unsigned)((LAG - 1) * NU + q) * ES);
            a1[q] = lane == 0 ? v : (TS)0;
            mw[q] = 0; a2[q] = 0; a3[q] = 0;
        }
        __syncwarp();
        if (any_in) {
            ch_lu.release(ch_lu.in++);
            if (P <= up_last_in) ch_lu.arm(ch_lu.in, timed_out);
        }
        bool ready = false;            // the early tests of the next batch (alike in all lanes)
        for (int b = 0; b < nb; b++) {
            const bool in = b + P <= up_last_in;
            if (!ready) {
                if (in) ch_lu.receive(ch_lu.in, timed_out);
                wait_frame(f_full[fw], use + b);
            }
            __syncwarp();
            rb = in ? ch_lu.slot(ch_lu.in) : ch_lu.zeros();
            const unsigned fb = frames + (unsigned)((use + b) % NF) * kFrameBytes, fa = fb + (unsigned)lane * ES;
            [[maybe_unused]] const int lines = SW - b * LAG;   // lines of this batch inside the planes
            TS cn[ND], rn[NU], pl[4], pu[NU], py = 0;
#pragma unroll
            for (int q = 0; q < NU; q++) { rn[q] = carry[q]; pu[q] = 0; }
#pragma unroll
            for (int k = 0; k < 4; k++) pl[k] = 0;
            auto load_step = [&](int k2) {
#pragma unroll
                for (int k = 0; k < ND; k++)
                    cn[k] = lds_v<TS>(fa + (unsigned)((F::kA + k) * kBlock + k2 * kLine) * ES);
                if (k2 > 0) {
#pragma unroll
                    for (int q = 0; q < NU; q++) rn[q] = lds_v<TS>(rb + (unsigned)((k2 - 1) * NU + q) * ES);
                }
            };
            // y = 1/dl1, the forward sweep's reciprocal pivot (the forward warp
            // makes it for the fast FP64 factorisation)
            auto store_step = [&](int k2) {
#pragma unroll
                for (int k = 0; k < 4; k++) sts_v(fa + (unsigned)((F::kL + k) * kBlock + k2 * kLine) * ES, pl[k]);
#pragma unroll
                for (int q = 0; q < NU; q++) sts_v(fa + (unsigned)((F::kU + q) * kBlock + k2 * kLine) * ES, pu[q]);
                if (!EXACT || IEEE) sts_v(fa + (unsigned)(F::kY * kBlock + k2 * kLine) * ES, py);
            };
            load_step(0);
#pragma unroll(IEEE ? 1 : LAG)
            for (int kk = 0; kk < LAG; kk++) {
                const int i = b * LAG + kk - 2 * lane;
                TS v[NU], cb[ND];
#pragma unroll
                for (int q = 0; q < NU; q++) v[q] = shfl_up_v(mw[q]);
#pragma unroll
                for (int k = 0; k < ND; k++) cb[k] = cn[k];
#pragma unroll
                for (int q = 0; q < NU; q++) {
                    if (lane == 0) v[q] = rn[q];
                    a3[q] = a2[q]; a2[q] = a1[q]; a1[q] = v[q];
                }
                if (kk > 0) store_step(kk - 1);
                if (kk + 1 < LAG) load_step(kk + 1);
                if (kk == LAG / 2 && b + 1 + P <= up_last_in) ch_lu.arm(ch_lu.in + 1, timed_out);
                if (kk == LAG - 2) {
                    const bool more = b + 1 + P <= up_last_in;
                    ready = __all_sync(kFull, b + 1 < nb && frame_ready(f_full[fw], use + b + 1) &&
                                                  (!more || ch_lu.arrived(ch_lu.in + 1)));
                }
                const bool inner = (unsigned)(i - 1) < (unsigned)(nx - 2) && (unsigned)(j - 1) < (unsigned)(ny - 2);
                const TS alpha = inner ? (TS)0.5 : (TS)0;
                TS l[NL], u[NU], y = 0;
                if constexpr (EXACT) lu_cell<ND, !IEEE>(cb, alpha, mw, a1, a2, a3, l, u, y);
                else lu_cell_f<ND>(cb, alpha, mw, a1, a2, a3, l, u, y);
                // (a bad pivot of the checked factorisation fails the check)
                if (!EXACT || IEEE) piv |= kk < lines ? pivot_bad(l[0]) : 0u;
                if (IEEE) {
                    const bool valid = i >= 0 && i < nx && j < ny;
#pragma unroll
                    for (int q = 0; q < NU; q++) u[q] = valid ? u[q] : (TS)0;
#pragma unroll
                    for (int k = 0; k < 4; k++) l[k] = valid ? l[k] : (TS)(k == 0 ? 1 : 0);
                    y = valid ? y : (TS)1;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) pl[k] = l[k];
#pragma unroll
                for (int q = 0; q < NU; q++) pu[q] = mw[q] = u[q];
                py = y;
            }
            store_step(LAG - 1);
#pragma unroll
            for (int q = 0; q < NU; q++) carry[q] = lds_v<TS>(rb + (unsigned)((LAG - 1) * NU + q) * ES);
            fence_async_shared();   // (each writer's own fence: see move)
            __syncwarp();
            if (in) ch_lu.release(ch_lu.in++);
            if (lane == 0) mbar_arrive(&f_lu[fw][(lu_uses + b) % NF]);
        }
        if (piv) bad_pivot = true;
    };

    // ---- forward sweep L w = -r (fb2d9 msi2d9-v03.f90:42-262, fb2d5
    // msi2d5-v03.f90:42-233), forward warp; fused: one batch behind the
    // factorisation of the same frames; make_y: 1/l1 is made here
    auto run_fw = [&](bool fused, [[maybe_unused]] bool make_y) {
        // the planes of a step: r, l1 (FP64 only), l2..l4 [, l5], 1/l1
        constexpr int NC = (EXACT ? 2 : 1) + 3 + (ND == 9 ? 1 : 0) + 1;
        constexpr int cL = EXACT ? 2 : 1;              // index of l2
        unsigned rb = ch_fw.zeros();
        const bool any_in = P - 1 <= up_last_in;
        if (any_in) {
            ch_fw.arm(ch_fw.in, timed_out);
            ch_fw.receive(ch_fw.in, timed_out);
            rb = ch_fw.slot(ch_fw.in);
        }
        TS mine = 0, a2 = 0, a3 = 0;
        TS a1 = lds_v<TS>(rb + (unsigned)(LAG - 2) * ES), carry = lds_v<TS>(rb + (unsigned)(LAG - 1) * ES);
        if (lane != 0) a1 = 0;
        __syncwarp();
        if (any_in) {
            ch_fw.release(ch_fw.in++);
            if (P <= up_last_in) ch_fw.arm(ch_fw.in, timed_out);
        }
        bool ready = false;
        for (int b = 0; b < nb; b++) {
            const bool in = b + P <= up_last_in;
            if (fused) {
                // the front warp's u of this batch go to the group above from
                // here, off its recurrence
                wait_frame(f_lu[fw], lu_uses + b);
                if (sends_up(b)) {
                    ch_lu.wait_free(ch_lu.out, timed_out);
                    ch_lu.send(ch_lu.out++, frames + (unsigned)((use + b) % NF) * kFrameBytes +
                                                (unsigned)(F::kU * kBlock + 31) * ES, kBlock * ES);
                }
            }
            if (!ready) {
                if (in) ch_fw.receive(ch_fw.in, timed_out);
                wait_frame(f_full[fw], use + b);
            }
            __syncwarp();
            rb = in ? ch_fw.slot(ch_fw.in) : ch_fw.zeros();
            const unsigned fa = frames + (unsigned)((use + b) % NF) * kFrameBytes + (unsigned)lane * ES;
            [[maybe_unused]] const int lines = SW - b * LAG;
            if constexpr (EXACT) {
                if (make_y) {
#pragma unroll
                    for (int k = 0; k < LAG; k++) {
                        const double l1 = lds_v<double>(fa + (unsigned)(F::kL * kBlock + k * kLine) * ES);
                        sts_v(fa + (unsigned)(F::kY * kBlock + k * kLine) * ES, rcp_fast(l1, rcp_start(l1)));
                    }
                }
            }
            const TS m0 = mine, s1 = a1, s2 = a2, s3 = a3;   // the state at the batch's start
            TS c[NC] = {}, cn[NC], rn = carry, pw = 0;
            [[maybe_unused]] unsigned bad = 0;
            auto load_step = [&](int k2) {
                auto at = [&](int pl) { return lds_v<TS>(fa + (unsigned)(pl * kBlock + k2 * kLine) * ES); };
                cn[0] = at(F::kR);
                if (EXACT) cn[1] = at(F::kL);
#pragma unroll
                for (int k = 0; k < 3; k++) cn[cL + k] = at(F::kL + 1 + k);
                if (ND == 9) cn[cL + 3] = at(F::kA);
                cn[NC - 1] = at(F::kY);
                if (k2 > 0) rn = lds_v<TS>(rb + (unsigned)(k2 - 1) * ES);
            };
            // w = -(r + l2 w_W + l3 w_SE + l4 w_S [+ l5 w_SW]) / l1
            auto numerator = [&]() -> TS {
                if constexpr (EXACT) {
                    if (ND == 9) return c[0] + c[cL] * mine + c[cL + 1] * a1 + c[cL + 2] * a2 + c[cL + 3] * a3;
                    return c[0] + c[cL] * mine + c[cL + 1] * a1 + c[cL + 2] * a2;
                } else {
                    const float num = fmaf(c[cL + 2], a2, fmaf(c[cL + 1], a1, fmaf(c[cL], mine, c[0])));
                    return ND == 9 ? fmaf(c[cL + 3], a3, num) : num;
                }
            };
            load_step(0);
#pragma unroll
            for (int kk = 0; kk < LAG; kk++) {
                TS v = shfl_up_v(mine);
#pragma unroll
                for (int k = 0; k < NC; k++) c[k] = cn[k];
                if (lane == 0) v = rn;
                a3 = a2; a2 = a1; a1 = v;
                if (kk > 0) sts_v(fa + (unsigned)(F::kW * kBlock + (kk - 1) * kLine) * ES, pw);
                if (kk + 1 < LAG) load_step(kk + 1);
                if (kk == LAG / 2 && b + 1 + P <= up_last_in) ch_fw.arm(ch_fw.in + 1, timed_out);
                if (kk == LAG - 3) {
                    const bool more = b + 1 + P <= up_last_in;
                    ready = __all_sync(kFull, b + 1 < nb && frame_ready(f_full[fw], use + b + 1) &&
                                                  (!more || ch_fw.arrived(ch_fw.in + 1)));
                }
                const TS num = numerator();
                if constexpr (EXACT) {
                    // one correction with the exact remainder (Markstein, IBM J.
                    // Res. Dev. 34, 1990) and its check, off the recurrence: 119
                    // cycles a step in a one-warp probe, 165 with a second
                    // correction and tests of the operands' range
                    const double q0 = num * c[NC - 1];
                    const double q1 = fma(fma(-q0, c[1], num), c[NC - 1], q0);
                    mine = -q1;
                    bad |= (unsigned)(kk < lines) & (unsigned)!quot_common(num, c[1], q1);
                } else {
                    mine = -num * c[NC - 1];
                }
                pw = mine;
            }
            sts_v(fa + (unsigned)(F::kW * kBlock + (LAG - 1) * kLine) * ES, pw);
            if constexpr (EXACT) {
                if (__any_sync(kFull, bad != 0u)) {
                    // some quotient may not be IEEE division's: the batch again
                    // from its start with '/'.  (Where the residual is zero w
                    // decays over hundreds of cells, so this is not rare.)
                    mine = m0; a1 = s1; a2 = s2; a3 = s3;
                    rn = carry;
                    load_step(0);
#pragma unroll 1
                    for (int kk = 0; kk < LAG; kk++) {
                        TS v = shfl_up_v(mine);
#pragma unroll
                        for (int k = 0; k < NC; k++) c[k] = cn[k];
                        if (lane == 0) v = rn;
                        a3 = a2; a2 = a1; a1 = v;
                        if (kk + 1 < LAG) load_step(kk + 1);
                        mine = -(numerator() / c[1]);
                        sts_v(fa + (unsigned)(F::kW * kBlock + kk * kLine) * ES, mine);
                    }
                }
            }
            carry = lds_v<TS>(rb + (unsigned)(LAG - 1) * ES);
            fence_async_shared();
            __syncwarp();
            if (in) ch_fw.release(ch_fw.in++);
            if (lane == 0) mbar_arrive(&f_done[fw][(use + b) % NF]);
        }
    };

    // ---- backward sweep U z = w, front warp: batches and lines descend, the
    // row above is the neighbour; E is the row's own previous value
    auto run_bw = [&]() {
        auto comes = [&](int n) { return n >= 0 && n <= dn_top_in; };
        unsigned rb = ch_bw.zeros();
        const bool any_in = comes(nb - P);
        if (has_above) ch_bw.arm(ch_bw.in, timed_out);   // (dn_top_in >= 0 there)
        if (any_in) {
            ch_bw.receive(ch_bw.in, timed_out);
            rb = ch_bw.slot(ch_bw.in);
        }
        TS mine = 0, a3 = 0, carry = lds_v<TS>(rb);
        TS a1 = lds_v<TS>(rb + ES), a2 = lds_v<TS>(rb + 2 * ES);
        if (lane != 31) a1 = a2 = 0;
        __syncwarp();
        if (any_in) {
            ch_bw.release(ch_bw.in++);
            if (comes(nb - P - 1)) ch_bw.arm(ch_bw.in, timed_out);
        }
        bool ready = false;
        for (int q = 0; q < nb; q++) {
            const int b = nb - 1 - q;
            const bool in = comes(b - P);
            if (!ready) {
                if (in) ch_bw.receive(ch_bw.in, timed_out);
                wait_frame(f_full[fw], use + q);
            }
            __syncwarp();
            if (q == 0 && nit_first) stamp(L, rank, 3);
            rb = in ? ch_bw.slot(ch_bw.in) : ch_bw.zeros();
            const unsigned fa = frames + (unsigned)((use + q) % NF) * kFrameBytes + (unsigned)lane * ES;
            if (SW - b * LAG < LAG) {
                // lines past the group's last hold other planes' values: the
                // sweep starts from zeros there
                for (int k = SW - b * LAG; k < LAG; k++) {
                    sts_v(fa + (unsigned)(F::kW * kBlock + k * kLine) * ES, (TS)0);
#pragma unroll
                    for (int v = 0; v < NU; v++) sts_v(fa + (unsigned)((F::kU + v) * kBlock + k * kLine) * ES, (TS)0);
                }
            }
            TS c[NU + 1], cn[NU + 1], rn = carry, pz = 0;
            auto load_step = [&](int kk) {             // line LAG - 1 - kk
                cn[0] = lds_v<TS>(fa + (unsigned)(F::kW * kBlock + (LAG - 1 - kk) * kLine) * ES);
#pragma unroll
                for (int k = 0; k < NU; k++)
                    cn[k + 1] = lds_v<TS>(fa + (unsigned)((F::kU + k) * kBlock + (LAG - 1 - kk) * kLine) * ES);
                if (kk > 0) rn = lds_v<TS>(rb + (unsigned)(LAG - kk) * ES);
            };
            load_step(0);
#pragma unroll
            for (int kk = 0; kk < LAG; kk++) {
                TS v = shfl_down_v(mine);
#pragma unroll
                for (int k = 0; k < NU + 1; k++) c[k] = cn[k];
                if (lane == 31) v = rn;
                a3 = a2; a2 = a1; a1 = v;
                if (kk > 0) sts_v(fa + (unsigned)(F::kW * kBlock + (LAG - kk) * kLine) * ES, pz);
                if (kk + 1 < LAG) load_step(kk + 1);
                // (the channel's first batch was armed before the loop)
                if (kk == LAG / 2 && in && comes(b - 1 - P)) ch_bw.arm(ch_bw.in + 1, timed_out);
                if (kk == LAG - 3) {
                    const bool more = comes(b - 1 - P);
                    ready = __all_sync(kFull, q + 1 < nb && frame_ready(f_full[fw], use + q + 1) &&
                                                  (!more || ch_bw.arrived(ch_bw.in + (in ? 1 : 0))));
                }
                // z = w - du1 z_E - du2 z_NW - du3 z_N [- du4 z_NE]
                TS z;
                if constexpr (EXACT) {
                    if (ND == 9) z = c[0] - c[1] * mine - c[2] * a1 - c[3] * a2 - c[4] * a3;
                    else z = c[0] - c[1] * mine - c[2] * a1 - c[3] * a2;
                } else {
                    z = fmaf(-c[3], a2, fmaf(-c[2], a1, fmaf(-c[1], mine, c[0])));
                    if (ND == 9) z = fmaf(-c[4], a3, z);
                }
                mine = pz = z;
            }
            sts_v(fa + (unsigned)(F::kW * kBlock) * ES, pz);
            carry = lds_v<TS>(rb);
            fence_async_shared();
            __syncwarp();
            if (in) ch_bw.release(ch_bw.in++);
            if (lane == 0) mbar_arrive(&f_done[fw][(use + q) % NF]);
        }
    };

    // ---- mover warp: frames in, finished planes out, one plane per lane, and
    // the sweep's hand-off values on to the next group.  A
    // frame goes out when the sweep is done with it and comes back with the
    // batch NF later.  Reads cover whole batches (lines behind a group are the
    // next group's, or the next plane's, and reach no valid cell); writes stop
    // at the group's last line.  The lanes that wrote a frame each fence their
    // stores against the copies out before they hand it on; a fence here alone
    // let copies overtake the last stores of a batch now and then, with many
    // instances on the GPU.  track: publish the batches that have arrived
    // in global memory, for the checking warps.
    auto move = [&](const TS *src, int ipos, int nload, TS *dst, int opos, bool down, bool track) {
        constexpr unsigned kBytes = kBlock * ES;
        for (int t = 0; t < nb + NF; t++) {
            if (t >= NF) {
                const int q = t - NF, b = down ? nb - 1 - q : q;
                const unsigned fr = frames + (unsigned)((use + q) % NF) * kFrameBytes;
                wait_frame(f_done[fw], use + q);
                if (down) {
                    if (has_below && b <= dn_top_out) {
                        ch_bw.wait_free(ch_bw.out, timed_out);
                        ch_bw.send(ch_bw.out++, fr + F::kW * kBytes, 0u);
                    }
                } else if (sends_up(b)) {
                    ch_fw.wait_free(ch_fw.out, timed_out);
                    ch_fw.send(ch_fw.out++, fr + F::kW * kBytes + 31u * ES, 0u);
                }
                fence_async_shared();   // this warp's reads precede the copies in
                const int lines = min(LAG, SW - b * LAG);
                if (dst && lines > 0)
                    bulk_s2g(dst + (long long)b * kBlock, fr + (unsigned)opos * kBytes, (unsigned)lines * kLine * ES);
                bulk_commit();
                if (track) {
                    bulk_wait<1>();     // batches before this one have arrived
                    __syncwarp();
                    if (lane == 0) st_cluster_release(smem_u32(&prog[fw]), (unsigned)q);
                }
                bulk_wait_read();
                __syncwarp();
            }
            if (t < nb) {
                const int b = down ? nb - 1 - t : t, f = (use + t) % NF;
                if (lane == 0) mbar_arrive_tx(&f_full[fw][f], (unsigned)nload * kBytes);
                __syncwarp();
                if (src) {
                    const unsigned to = frames + (unsigned)f * kFrameBytes + (unsigned)ipos * kBytes;
                    bulk_g2s(to, src + (long long)b * kBlock, kBytes, &f_full[fw][f]);
                }
            }
        }
        bulk_wait<0>();
        fence_async_global();
        __syncwarp();
        if (track && lane == 0) st_cluster_release(smem_u32(&prog[fw]), (unsigned)nb);
    };
    // a lane's plane in and out: l1 (FP64 only), l2.., u.., 1/l1, and r or w
    auto factor_plane = [&](int k, TS *&p, int &pos) {
        if (k < 4) { p = dlp + k * PS; pos = F::kL + k; if (!EXACT && k == 0) p = nullptr; }
        else if (k < 4 + NU) { p = dup + (k - 4) * PS; pos = F::kU + k - 4; }
        else if (k == 4 + NU) { p = rl1; pos = F::kY; }
        if (p) p += line0 * kLine;
    };
    auto run_mover = [&](bool fused) {
        TS *src = nullptr, *dst = nullptr;
        int ipos = 0, opos = 0, nload;
        if (fused) {
            if (lane < ND) { src = asp + lane * PS + line0 * kLine; ipos = F::kA + lane; }
            if (lane == ND) { src = rp + line0 * kLine; ipos = F::kR; }
            nload = ND + 1;
            factor_plane(lane, dst, opos);
            if (lane == 5 + NU) { dst = wp + line0 * kLine; opos = F::kW; }
        } else {
            if (lane < 4 || lane == 4 + NU) factor_plane(lane, src, ipos);
            if (lane == 5 + NU) { src = rp + line0 * kLine; ipos = F::kR; dst = wp + line0 * kLine; opos = F::kW; }
            if (ND == 9 && lane == 6 + NU) { src = asp + line0 * kLine; ipos = F::kA; }
            nload = 3 + (EXACT ? 1 : 0) + 1 + 1 + (ND == 9 ? 1 : 0);
        }
        move(src, ipos, nload, dst, opos, false, fused && EXACT);
        use += nb;
        src = dst = nullptr;
        if (lane >= 4 && lane < 4 + NU) factor_plane(lane, src, ipos);
        if (lane == 5 + NU) { src = dst = wp + line0 * kLine; ipos = opos = F::kW; }
        move(src, ipos, NU + 1, dst, opos, true, false);
        use += nb;
    };

    // ---- checking warps: parts of batches in order, dealt by a shared
    // counter (small parts, so that the last batch does not keep one warp
    // busy after the sweeps); a part waits until its batch's factors and those
    // it reads of the group below are in global memory
    auto run_check = [&]() {
        constexpr int kParts = LAG / 4;
        unsigned seen[2] = {0u, 0u}, seen_below[2] = {0u, 0u};   // progress known, per group of this CTA
        const int most = batches(rank * WPC);
        bool ok = true;
        for (;;) {
            int n = 0;
            if (lane == 0) n = atomicAdd(&chk_next, 1);
            n = __shfl_sync(kFull, n, 0);
            const int part = n % kParts, f = n / kParts % WPC, b = n / (kParts * WPC), g = rank * WPC + f;
            if (b >= most) break;
            if (g >= NG || b >= batches(g)) continue;
            auto arrived = [&](unsigned &known, unsigned addr, unsigned need) {
                if (known >= need) return;
                const unsigned long long t0 = gtimer();
                while (!timed_out && (known = ld_cluster_acquire(addr)) < need) {
                    __nanosleep(200);
                    if (gtimer() - t0 > kWaitLimitNs) timed_out = true;
                }
            };
            arrived(f ? seen[1] : seen[0], smem_u32(&prog[f]), (unsigned)b + 1u);
            if (g > 0)
                arrived(f ? seen_below[1] : seen_below[0],
                        f > 0 ? smem_u32(&prog[f - 1]) : cluster_addr(&prog[WPC - 1], rank - 1),
                        (unsigned)min(b + P, batches(g - 1) - 1) + 1u);
            __syncwarp();
            const int s = b * LAG + 4 * part;
#pragma unroll 1
            for (int q = 0; q < 4; q++)
                ok = ok & (s + q >= SW || line_ok<ND>((const double *)asp, (const double *)dlp, (const double *)dup,
                                                      (const double *)rl1, nx, ny, SW, PS, g, s + q));
        }
        if (!ok) atomicOr(&vbad, 1u);
    };

    // one sweep pair, with a factorisation in front when `fused`
    auto sweeps = [&](auto ieee_tag, bool fused, bool check) {
        if (front) {
            if (fused) { run_lu(ieee_tag); lu_uses += nb; }
            use += nb;
            if (nit_first) { stamp(L, rank, 1); stamp(L, rank, 2); }
            // also keeps this warp's frame phases with the forward warp's
            mbar_wait(&f_turn[fw], (unsigned)turns & 1u, timed_out);
            run_bw();
            use += nb;
        } else if (fwd) {
            run_fw(fused, fused && !decltype(ieee_tag)::value);
            if (lane == 0) mbar_arrive(&f_turn[fw]);
            if (fused) lu_uses += nb;
            use += 2 * nb;
        } else if (mover) {
            run_mover(fused);
        }
        if constexpr (EXACT) {
            // (WPC = 1: warp 4 shares the front warp's sub-partition)
            if (check && !front && !mover && (WPC == 2 || wl != 4)) run_check();
        }
        turns++;
    };

    // ---- the iteration (fb2d9 msi2d9-v03.f90:42-262, fb2d5 msi2d5-v03.f90:42-233)
    double rr0 = rr0_s;
    const double gammarp = L.tol * sqrt(rr0);
    const int cap = (L.nitm > 0) ? L.nitm : kMaxIterUnbounded;
    int nit = L.nit0;
    double rr = cont ? S.rr[1] : rr0;
    bool factorise = !reuse;
    for (;;) {
        nit = nit + 1;
        // test hook: row group 0's front warp waits, bounded by L.hook_ns, on
        // a barrier that nothing completes, then goes on as usual (its
        // neighbours' own waits are bounded far above that, so every real
        // hand-off still completes and no copy is left in flight)
        if (L.hook_ns && nit == 1 && rank == 0 && wl == 0) {
            if (!mbar_wait_for(&idle_bar, 0u, L.hook_ns)) hook_ran_out = true;
            __syncwarp();
        }
        nit_first = nit == 1;
        sweeps(std::false_type{}, factorise, factorise);
        if constexpr (EXACT) {
            if (factorise) {
                // the findings of the checks, before x changes: the factorisation
                // and its sweep pair again, with IEEE division (A's planes and r
                // are untouched)
                cl.sync();
                unsigned any = 0;
                for (int c = 0; c < C; c++) any |= *cl.map_shared_rank(&vbad, c);
                if (any) {
                    cl.sync();   // every CTA has read the findings
                    bad_pivot = false;   // the repeat decides
                    if (rank == 0 && threadIdx.x == 0) atomicAdd(&g_lu_redo, 1ull);
                    sweeps(std::true_type{}, true, false);
                }
            }
        }
        factorise = false;
        if (nit == 1) stamp(L, rank, 4);
        if (L.apply_only) break;   // x += z by k_unskew_add after the launch
        if (L.ext == 1) break;     // x += z, the residual and the test on the whole GPU
        rr = cluster_residual<ND, TS>(cl, a, S.b, x, wp, rp, nx, ny, SW, red, part);
        if (nit == 1) stamp(L, rank, 5);
        if (sqrt(rr) < gammarp) break;
        if (nit == cap) {
            if (L.nitm <= 0 && L.err && rank == 0 && threadIdx.x == 0) atomicOr(L.err, ERR_WAIT_TIMEOUT);
            break;
        }
    }
    if (bad_pivot && L.err) atomicOr(L.err, ERR_NONFINITE_PIVOT);
    if (mover && use > 0) {
        // every copy into this group's frames has landed (it has, unless a
        // wait ran out before), so that shared memory may go away
        for (int u = max(0, use - NF); u < use; u++)
            (void)mbar_wait_for(&f_full[fw][u % NF], (unsigned)(u / NF) & 1u, kWaitLimitNs);
    }
    if ((timed_out || hook_ran_out) && L.err) atomicOr(L.err, ERR_SPIN_TIMEOUT);
    if (L.ext == 1) {
        // what the whole-GPU passes and the continuation need to know
        if (timed_out || hook_ran_out) atomicOr(ew.status, kExtTimedOut);
        if (bad_pivot) atomicOr(ew.status, kExtBadPivot);
        if (lagged && rank == 0 && threadIdx.x == 0) atomicOr(ew.status, kExtLagged);
    }
    if (rank == 0 && threadIdx.x == 0 && !L.apply_only) {
        if (S.nit) *S.nit = nit;
        if (S.rr) { S.rr[0] = rr0; if (L.ext != 1) S.rr[1] = rr; }
        if (!EXACT && L.lag_max > 0 && S.lag && !L.reuse_lu && L.ext != 1) {
            // the record for the next solve: fresh factors are one solve old;
            // reused ones age, and are renewed next time once they needed a
            // second iteration (or anything went wrong)
            const int st = cont ? *ew.status : 0;
            const bool lag_solve = cont ? (st & kExtLagged) != 0 : lagged;
            const bool renew = timed_out || hook_ran_out || bad_pivot || (st & (kExtTimedOut | kExtBadPivot)) ||
                               (lag_solve && nit > 1);
            S.lag[0] = S.tag;
            S.lag[1] = renew ? L.lag_max : (lag_solve ? lag_age + 1 : 1);
        }
    }
    cl.sync();   // no CTA leaves while another may still write into its shared memory
    stamp(L, rank, 6);
}

bool msi_warp_supported(int ny) { return ny <= 1024; }

long long msi_lu_redo_count()
{
    unsigned long long v = 0;
    if (cudaMemcpyFromSymbol(&v, g_lu_redo, sizeof v) != cudaSuccess) return -1;
    return (long long)v;
}

// launches one cluster per system if the cluster shape can be scheduled;
// *fits = false (and nothing launched) otherwise
template <int ND, int WPC, int NF, typename TS, int LAG>
static cudaError_t launch_cluster(const MsiLaunch &L, int nsys, cudaStream_t st, bool *fits)
{
    *fits = false;
    const int ngroups = (L.ny + 31) / 32;
    const int C = (ngroups + WPC - 1) / WPC;
    if (C > kMaxCluster) return cudaSuccess;
    auto kern = k_msi_c<ND, WPC, NF, TS, LAG>;
    const size_t smem = (size_t)WPC * NF * Frame<ND, LAG>::kPlanes * Frame<ND, LAG>::kBlock * sizeof(TS);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(C * nsys));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    e = cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg);
    if (e != cudaSuccess || nclusters < 1) {
        (void)cudaGetLastError();
        return cudaSuccess;
    }
    *fits = true;
    const bool apply = L.apply_only && L.reuse_lu && L.dev == nullptr && nsys <= 2;
    const long long N = (long long)L.nx * L.ny;
    const dim3 cg((unsigned)((N + 255) / 256 < 1184 ? (N + 255) / 256 : 1184), (unsigned)nsys);
    // the passes over all cells on the whole GPU (grids of kExtMinCells and
    // more, where they outweigh three extra launches)
    bool ext = !L.apply_only && !L.reuse_lu && L.dev == nullptr && nsys <= 2 && N >= kExtMinCells;
    for (int k = 0; k < nsys && ext; k++) ext = L.s[k].rr != nullptr && L.s[k].nit != nullptr;
    MsiLaunch La = L;
    La.apply_only = apply ? 1 : 0;
    if (apply) La.nitm = 1;
    La.ext = ext ? 1 : 0;
    La.nit0 = 0;
    // A (unless its factors are reused) into wavefront-major order and the
    // initial residual first: all systems, whole GPU
    const dim3 sg((unsigned)skew_blocks(L.nx, L.ny), (unsigned)ngroups, (unsigned)nsys);
    La.nparts = (int)(sg.x * sg.y);
    k_skew<ND, TS><<<sg, 256, 0, st>>>(La);
    int launches = 2;
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaLaunchKernelEx(&cfg, kern, La);
    if (e != cudaSuccess) return e;
    if (apply) {
        k_unskew_add<ND, TS><<<cg, 256, 0, st>>>(La);
        launches++;
    } else if (ext) {
        // two iterations with whole-GPU passes, then whatever else it takes
        MsiLaunch Lc = La;
        for (int it = 0; it < 2 && e == cudaSuccess; it++) {
            k_ext_update<ND, TS><<<cg, 256, 0, st>>>(Lc);
            k_ext_resid<ND, TS><<<dim3(kExtBlocks, (unsigned)nsys), 256, 0, st>>>(Lc);
            launches += 2;
            e = cudaGetLastError();
            Lc.nit0 = it + 1;
            if (L.nitm == Lc.nit0 && !L.prof) break;   // (the last launch also stamps the end)
            if (it == 1) Lc.ext = 2;
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, Lc);
            launches++;
        }
    }
    msi_note_launches(launches);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// one row group per SM where the cluster fits, else two, unless the caller
// asked for one schedule.  Batches of 16 lines in four frames per group (8 for
// two FP64 groups, so that both fit in shared memory): a batch costs 300 to
// 400 cycles on top of its steps, and each hop of the wavefront waits for one.
// FP32 solves that reuse factors have the shortest steps, and from
// kLongLagCells on run batches of 32: forward and backward sweep of 514x258
// cells take 97 us with them and 107 with 16, but a fresh FP32 solve 224 us
// against 211 (and one of 82x42 cells 62 against 59); 8 lose everywhere (a
// FP64 sweep pair 201 us against 163).
constexpr long long kLongLagCells = 1LL << 16;
template <int ND, typename TS>
static cudaError_t launch_schedules(const MsiLaunch &L, int nsys, cudaStream_t st, bool *done)
{
    constexpr bool FP64 = std::is_same<TS, double>::value;
    cudaError_t e = cudaSuccess;
    if (L.variant != 2) {
        const bool long_lag = (L.lag_max > 0 || L.reuse_lu) && (long long)L.nx * L.ny >= kLongLagCells;
        if (!FP64 && long_lag) e = launch_cluster<ND, 1, 4, float, 32>(L, nsys, st, done);
        else e = launch_cluster<ND, 1, 4, TS, 16>(L, nsys, st, done);
        if (e != cudaSuccess || *done || L.variant == 1) return e;
    }
    return launch_cluster<ND, 2, 4, TS, FP64 ? 8 : 16>(L, nsys, st, done);
}

template <int ND, typename TS>
static cudaError_t launch_nd(const MsiLaunch &L, int nsys, cudaStream_t st, bool *done)
{
    // the bulk copies need 16-byte aligned scratch (systems given through a
    // device array cannot be checked here) and the wavefront-major layout
    // must fit in the scratch
    *done = false;
    bool aligned = L.dev == nullptr;
    for (int k = 0; k < nsys && aligned; k++) aligned = ((uintptr_t)L.s[k].ws % 16) == 0;
    const bool room = L.ws_cap == 0 || L.ws_cap >= msi_cluster_work_doubles(ND, L.nx, L.ny);
    const bool small = (long long)L.nx * L.ny < (1LL << 31);   // 32-bit cell indices in the passes
    if (!(aligned && room && small)) return cudaSuccess;
    return launch_schedules<ND, TS>(L, nsys, st, done);
}

// m2d_test_wait_hook's setting for the cluster kernel (0: off)
static unsigned long long g_msi_hook_ns = 0;
void set_msi_wait_hook(unsigned long long ns) { g_msi_hook_ns = ns; }

cudaError_t launch_msi_warp(int nd, const MsiLaunch &L0, int nsys, cudaStream_t st)
{
    MsiLaunch L = L0;
    L.hook_ns = g_msi_hook_ns;
    bool done = false;
    cudaError_t e;
    if (L.prec == 1)
        e = nd == 9 ? launch_nd<9, float>(L, nsys, st, &done) : launch_nd<5, float>(L, nsys, st, &done);
    else
        e = nd == 9 ? launch_nd<9, double>(L, nsys, st, &done) : launch_nd<5, double>(L, nsys, st, &done);
    if (e != cudaSuccess || done) return e;
    return launch_msi_generic(nd, L0, nsys, st);
}

}  // namespace m2d
