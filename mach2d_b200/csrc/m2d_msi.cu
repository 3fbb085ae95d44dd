// m2d_msi.cu -- MSI wavefront kernels (lu2d9/fb2d9, lu2d5/fb2d5) and line TDMA.
//
// Dependency structure.  The incomplete factorisation and the forward sweep
// of cell (i,j) read (i-1,j), (i-1,j-1), (i,j-1) and (i+1,j-1)
// (src/solvers/msi2d9-v03.f90:155,357-366); the backward sweep reads the
// mirror image.  Cells on the hyperplane t = i + 2j are therefore mutually
// independent and the whole grid is swept in nx + 2(ny-1) steps.
//
// Execution.  One CTA per linear system.  Thread t owns rows j = t, t+T, ...
// and at step s processes column i = s - 2j of each owned row, so a row lags
// the one below it by two columns.  The factor values a row produces are
// published in a 4-step shared-memory ring [slot][value][row] (conflict-free:
// consecutive threads read consecutive rows); one __syncthreads per step.
// Residuals and the L2 norm of the stopping test run over all cells with
// coalesced accesses and a fixed-order block tree.
//
// Parity.  The reference's special cases for the first/last rows and columns
// are the general formula with out-of-grid neighbours taken as zero and the
// relaxation alpha = 0 there; under the reference's own precondition (no
// coupling to neighbours outside the grid, msi2d9-v03.f90:16-17) the zero
// terms add exact zeros, so with -fmad=false every factor and every sweep
// value is bitwise equal to the lexicographic reference loop.  Only the
// stopping test's sum of squares is ordered differently.
#include "m2d_div.cuh"
#include "m2d_solvers.cuh"

namespace m2d {

static const int kMaxThreads = 1024;
static const int kRingSlots = 4;
static const int kMaxIterUnbounded = 10000;   // nitm <= 0: loop until converged, bounded

int msi_block_threads(int ny)
{
    int t = ((ny + 31) / 32) * 32;
    return t > kMaxThreads ? kMaxThreads : t;
}
size_t msi_smem_bytes(int nd, int ny)
{
    int nu = (nd == 9) ? 4 : 3;
    return (size_t)kRingSlots * nu * ny * sizeof(double) + (size_t)msi_block_threads(ny) * sizeof(double);
}
size_t msi_skew_plane(int nx, int ny)
{
    return (size_t)((ny + 31) / 32) * (size_t)(nx + 62) * 32;
}
size_t msi_generic_work_doubles(int nd, int nx, int ny)
{
    return (size_t)(nd == 9 ? 10 : 8) * (size_t)nx * ny;                 // dl, du, residual
}
size_t msi_cluster_work_doubles(int nd, int nx, int ny)
{
    // dl, du, 1/dl1, residual, correction and A, wavefront-major, then the
    // scratch of the whole-GPU residual passes
    return (size_t)(nd == 9 ? 21 : 15) * msi_skew_plane(nx, ny) + kMsiExtScratch;
}
size_t msi_work_doubles(int nd, int nx, int ny)
{
    const size_t g = msi_generic_work_doubles(nd, nx, ny), c = msi_cluster_work_doubles(nd, nx, ny);
    return g > c ? g : c;
}
int msi_max_ny()
{
    // 227 KB of opt-in shared memory per CTA on sm_100
    int ny = 16;
    while (msi_smem_bytes(9, ny + 16) <= 227 * 1024) ny += 16;
    return ny;
}

#define RING(slot, k, row) ring[((size_t)(slot) * NU + (k)) * ny + (row)]
#define PL(p, k, np) (p)[(long long)((k) - 1) * N + (np)]

// fixed-order block sum for any blockDim.x (a multiple of 32): fold the
// tail onto the largest power of two, then a binary tree
template <int ND>
__device__ double block_sum(double v, double *red)
{
    const int T = blockDim.x;
    int P = 1;
    while (P * 2 <= T) P *= 2;
    red[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < T - P) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + P];
    __syncthreads();
    for (int s = P / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + s];
        __syncthreads();
    }
    double r = red[0];
    __syncthreads();
    return r;
}

// r = A x - b over all cells, in-range neighbours only, in ascending diagonal
// order (msi2d9-v03.f90:61-131 / msi2d5-v03.f90:61-119); returns this
// thread's partial sum of r^2.
template <int ND>
__device__ double residual(const double *__restrict__ a, const double *__restrict__ b,
                           const double *x, double *r, int nx, int ny)
{
    const long long N = (long long)nx * ny;
    double acc = 0.0;
    for (long long np = threadIdx.x; np < N; np += blockDim.x) {
        const int i = (int)(np % nx), j = (int)(np / nx);
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
        r[np] = v;
        acc = acc + v * v;
    }
    return acc;
}

template <int ND>
__global__ void __launch_bounds__(kMaxThreads) k_msi(MsiLaunch L)
{
    constexpr int NU = (ND == 9) ? 4 : 3;
    extern __shared__ double smem[];
    const MsiSys S = L.dev ? L.dev[blockIdx.x] : L.s[blockIdx.x];
    const int nx = L.nx, ny = L.ny;
    const long long N = (long long)nx * ny;
    const int T = blockDim.x;
    const int nsteps = nx + 2 * (ny - 1);
    double *ring = smem;
    double *red = smem + (size_t)kRingSlots * NU * ny;
    const double *__restrict__ a = S.a;
    // plain plane-major scratch: dl planes, du planes, one residual plane
    double *__restrict__ dl = S.ws;
    double *__restrict__ du = S.ws + (ND == 9 ? 5 : 4) * N;
    double *wk = du + NU * N;
    double *x = S.x;
    bool bad_pivot = false;

    // ---- incomplete LU (lu2d9 msi2d9-v03.f90:277-432, lu2d5 msi2d5-v03.f90:247-330)
    for (int s = 0; s < nsteps; s++) {
        const int c0 = s & 3, c1 = (s + 3) & 3, c2 = (s + 2) & 3, c3 = (s + 1) & 3;
        for (int j = threadIdx.x; j < ny; j += T) {
            const int i = s - 2 * j;
            if (i < 0 || i >= nx) continue;
            const long long np = (long long)j * nx + i;
            const bool hw = i > 0, hs = j > 0, hsw = hs && i > 0, hse = hs && i < nx - 1;
            const double alpha = (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2) ? 0.5 : 0.0;
            if (ND == 9) {
                double w1 = hw ? RING(c1, 0, j) : 0.0, w2 = hw ? RING(c1, 1, j) : 0.0;
                double w3 = hw ? RING(c1, 2, j) : 0.0, w4 = hw ? RING(c1, 3, j) : 0.0;
                double s1 = hs ? RING(c2, 0, j - 1) : 0.0, s2 = hs ? RING(c2, 1, j - 1) : 0.0;
                double s3 = hs ? RING(c2, 2, j - 1) : 0.0, s4 = hs ? RING(c2, 3, j - 1) : 0.0;
                double sw1 = hsw ? RING(c3, 0, j - 1) : 0.0, sw2 = hsw ? RING(c3, 1, j - 1) : 0.0;
                double sw3 = hsw ? RING(c3, 2, j - 1) : 0.0, sw4 = hsw ? RING(c3, 3, j - 1) : 0.0;
                double se1 = hse ? RING(c1, 0, j - 1) : 0.0, se2 = hse ? RING(c1, 1, j - 1) : 0.0;
                double se3 = hse ? RING(c1, 2, j - 1) : 0.0, se4 = hse ? RING(c1, 3, j - 1) : 0.0;
                const double b1 = PL(a, 1, np), b2 = PL(a, 2, np), b3 = PL(a, 3, np);
                const double b4 = PL(a, 4, np), b5 = PL(a, 5, np), b6 = PL(a, 6, np);
                const double b7 = PL(a, 7, np), b8 = PL(a, 8, np), b9 = PL(a, 9, np);
                double l5 = b1;
                double l4 = (b2 - l5 * sw1 - alpha * b3 * se1) / (1.0 - alpha * s1 * se1);
                double l3 = b3 - l4 * s1;
                double l2 = (b4 - l4 * s2 - l5 * sw3 - 2.0 * alpha * l5 * sw2) / (1 + 2.0 * alpha * w2);
                double phi1 = l3 * se1, phi2 = l5 * sw2, phi3 = l3 * se4, phi4 = l2 * w2;
                double l1 = b5 - l2 * w1 - l3 * se2 - l4 * s3 - l5 * sw4
                          + alpha * (2.0 * phi1 + phi2 + phi3 + 2.0 * phi4);
                double u1 = (b6 - l3 * se3 - l4 * s4 - 2.0 * alpha * (phi1 + phi3)) / l1;
                double u2 = (b7 - l2 * w3) / l1;
                double u3 = (b8 - l2 * w4 - alpha * phi4) / l1;
                double u4 = b9 / l1;
                if (!(fabs(l1) > 0.0) || !isfinite(l1)) bad_pivot = true;
                PL(dl, 1, np) = l1; PL(dl, 2, np) = l2; PL(dl, 3, np) = l3; PL(dl, 4, np) = l4; PL(dl, 5, np) = l5;
                PL(du, 1, np) = u1; PL(du, 2, np) = u2; PL(du, 3, np) = u3; PL(du, 4, np) = u4;
                RING(c0, 0, j) = u1; RING(c0, 1, j) = u2; RING(c0, 2, j) = u3; RING(c0, 3, j) = u4;
            } else {
                double w1 = hw ? RING(c1, 0, j) : 0.0, w2 = hw ? RING(c1, 1, j) : 0.0;
                double w3 = hw ? RING(c1, 2, j) : 0.0;
                double s1 = hs ? RING(c2, 0, j - 1) : 0.0, s2 = hs ? RING(c2, 1, j - 1) : 0.0;
                double s3 = hs ? RING(c2, 2, j - 1) : 0.0;
                double se1 = hse ? RING(c1, 0, j - 1) : 0.0, se2 = hse ? RING(c1, 1, j - 1) : 0.0;
                double se3 = hse ? RING(c1, 2, j - 1) : 0.0;
                (void)hsw;
                const double b1 = PL(a, 1, np), b2 = PL(a, 2, np), b3 = PL(a, 3, np);
                const double b4 = PL(a, 4, np), b5 = PL(a, 5, np);
                double l4 = b1 / (1.0 - alpha * s1 * se1);
                double l3 = -l4 * s1;
                double l2 = (b2 - l4 * s2) / (1.0 + 2.0 * alpha * w2);
                double phi1 = l3 * se1, phi4 = l2 * w2;
                double l1 = b3 - l2 * w1 - l3 * se2 - l4 * s3 + 2.0 * alpha * (phi1 + phi4);
                double u1 = (b4 - l3 * se3 - 2.0 * alpha * phi1) / l1;
                double u2 = -l2 * w3 / l1;
                double u3 = (b5 - alpha * phi4) / l1;
                if (!(fabs(l1) > 0.0) || !isfinite(l1)) bad_pivot = true;
                PL(dl, 1, np) = l1; PL(dl, 2, np) = l2; PL(dl, 3, np) = l3; PL(dl, 4, np) = l4;
                PL(du, 1, np) = u1; PL(du, 2, np) = u2; PL(du, 3, np) = u3;
                RING(c0, 0, j) = u1; RING(c0, 1, j) = u2; RING(c0, 2, j) = u3;
            }
        }
        __syncthreads();
    }
    if (bad_pivot && L.err) atomicOr(L.err, ERR_NONFINITE_PIVOT);

    // ---- fb2d9 / fb2d5 (msi2d9-v03.f90:42-262, msi2d5-v03.f90:42-233)
    double rr0 = block_sum<ND>(residual<ND>(a, S.b, x, wk, nx, ny), red);
    const double gammarp = L.tol * sqrt(rr0);
    const int cap = (L.nitm > 0) ? L.nitm : kMaxIterUnbounded;
    int nit = 0;
    double rr = rr0;
    for (;;) {
        nit = nit + 1;
        // forward: L w = -r, w overwrites r in wk
        for (int s = 0; s < nsteps; s++) {
            const int c0 = s & 3, c1 = (s + 3) & 3, c2 = (s + 2) & 3, c3 = (s + 1) & 3;
            for (int j = threadIdx.x; j < ny; j += T) {
                const int i = s - 2 * j;
                if (i < 0 || i >= nx) continue;
                const long long np = (long long)j * nx + i;
                const bool hw = i > 0, hs = j > 0;
                const double ww = hw ? RING(c1, 0, j) : 0.0;
                const double wse = (hs && i < nx - 1) ? RING(c1, 0, j - 1) : 0.0;
                const double ws = hs ? RING(c2, 0, j - 1) : 0.0;
                double w;
                if (ND == 9) {
                    const double wsw = (hs && hw) ? RING(c3, 0, j - 1) : 0.0;
                    w = -(wk[np] + PL(dl, 2, np) * ww + PL(dl, 3, np) * wse + PL(dl, 4, np) * ws
                          + PL(dl, 5, np) * wsw) / PL(dl, 1, np);
                } else {
                    w = -(wk[np] + PL(dl, 2, np) * ww + PL(dl, 3, np) * wse + PL(dl, 4, np) * ws)
                        / PL(dl, 1, np);
                }
                wk[np] = w;
                RING(c0, 0, j) = w;
            }
            __syncthreads();
        }
        // backward: U z = w, var = z + var
        for (int s = 0; s < nsteps; s++) {
            const int c0 = s & 3, c1 = (s + 3) & 3, c2 = (s + 2) & 3, c3 = (s + 1) & 3;
            for (int j = threadIdx.x; j < ny; j += T) {
                const int i = nx - 1 - (s - 2 * (ny - 1 - j));
                if (i < 0 || i >= nx) continue;
                const long long np = (long long)j * nx + i;
                const bool he = i < nx - 1, hn = j < ny - 1;
                const double ze = he ? RING(c1, 0, j) : 0.0;
                const double znw = (hn && i > 0) ? RING(c1, 0, j + 1) : 0.0;
                const double zn = hn ? RING(c2, 0, j + 1) : 0.0;
                double z;
                if (ND == 9) {
                    const double zne = (hn && he) ? RING(c3, 0, j + 1) : 0.0;
                    z = wk[np] - PL(du, 1, np) * ze - PL(du, 2, np) * znw - PL(du, 3, np) * zn
                        - PL(du, 4, np) * zne;
                } else {
                    z = wk[np] - PL(du, 1, np) * ze - PL(du, 2, np) * znw - PL(du, 3, np) * zn;
                }
                x[np] = z + x[np];
                RING(c0, 0, j) = z;
            }
            __syncthreads();
        }
        rr = block_sum<ND>(residual<ND>(a, S.b, x, wk, nx, ny), red);
        if (sqrt(rr) < gammarp) break;
        if (nit == cap) {
            if (L.nitm <= 0 && L.err && threadIdx.x == 0) atomicOr(L.err, ERR_WAIT_TIMEOUT);
            break;
        }
    }
    if (threadIdx.x == 0) {
        if (S.nit) *S.nit = nit;
        if (S.rr) { S.rr[0] = rr0; S.rr[1] = rr; }
    }
}

static thread_local int g_msi_launches = 0;
void msi_note_launches(int n) { g_msi_launches = n; }
int msi_last_launch_count() { return g_msi_launches; }

cudaError_t launch_msi(int nd, const MsiLaunch &L, int nsys, cudaStream_t st)
{
    if (L.ny > msi_max_ny() || L.nx < 3 || L.ny < 3) return cudaErrorInvalidValue;
    if (L.variant == 3 && L.prec == 0) return launch_msi_generic(nd, L, nsys, st);
    if (msi_warp_supported(L.ny)) return launch_msi_warp(nd, L, nsys, st);
    return launch_msi_generic(nd, L, nsys, st);
}

cudaError_t launch_msi_generic(int nd, const MsiLaunch &L, int nsys, cudaStream_t st)
{
    if (L.ny > msi_max_ny() || L.nx < 3 || L.ny < 3) return cudaErrorInvalidValue;
    const int T = msi_block_threads(L.ny);
    const size_t sm = msi_smem_bytes(nd, L.ny);
    // the limit is the kernel's, shared by every thread that launches it: the
    // largest grid's, always the same value (set to each launch's own, another
    // thread's smaller one in between made the launch fail)
    const size_t sm_max = msi_smem_bytes(nd, msi_max_ny());
    if (nd == 9) {
        cudaError_t e = cudaFuncSetAttribute(k_msi<9>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_max);
        if (e != cudaSuccess) return e;
        k_msi<9><<<nsys, T, sm, st>>>(L);
    } else {
        cudaError_t e = cudaFuncSetAttribute(k_msi<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_max);
        if (e != cudaSuccess) return e;
        k_msi<5><<<nsys, T, sm, st>>>(L);
    }
    msi_note_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// line TDMA (src/solvers/tdma2d9.f90:38-322, tdma2d5.f90:38-241).  A phase
// (every x line, or every y line) is one launch; the right-hand sides of a
// line read the old values of its neighbours (the reference's separate
// loops), so a phase writes its result to another buffer.
//
// A CTA takes LPC lines.  Lane l of warp 0 runs the recurrence of line l,
//   P = -e / (c + w P'),  Q = (D - w Q') / (c + w P'),
// while the other warps bring the next chunk of kTdmaChunk elements into
// shared memory (coalesced, right-hand sides D included) and check the
// quotients of the previous one (quot_ok); a quotient that is not IEEE
// division's repeats the CTA's lines with '/', so P and Q are the reference's
// bit for bit.  P and Q stay in shared
// memory, the back-substitution overwrites Q with x, and the lines are
// written once.  Bound by the latency of the recurrence, about 70 cycles a
// step for the division without a branch.  Four outer iterations on 203x77
// cells (200 line iterations) take 6.0 ms; one thread per line walking global
// memory, 1.1 us a step, took 85 ms.
namespace {
constexpr int kTdmaThreads = 128, kTdmaChunk = 64;
constexpr int kTdmaSmem = 220 * 1024;   // a CTA's dynamic limit (one value: threads share it, see launch_msi_generic)
enum { TDMA_X9, TDMA_X5, TDMA_Y9, TDMA_Y5, TDMA_LINES };
struct TdmaArgs {
    int nx, ny;                  // TDMA_LINES: line length and number of lines
    const double *a, *b, *x;     // TDMA_LINES: a = {aw, ap, ae} in a, b, x and d in rhs
    const double *rhs;
    double *out;                 // result (not x)
    double *P, *Q;               // scratch of N doubles each (Q may be out), used when in_smem == 0
    int in_smem;                 // P and Q of a CTA's lines fit in shared memory
};
// one element: w x_{i-1} + c x_i + e x_{i+1} = d, the terms of the other
// direction moved to d in the reference's order
struct TdmaRow { double w, c, e, d; };
template <int KIND>
__device__ __forceinline__ TdmaRow tdma_row(const TdmaArgs &A, int l, int q)
{
    TdmaRow r;
    if (KIND == TDMA_LINES) {
        const long long o = (long long)l * A.nx + q;
        r.w = A.a[o]; r.c = A.b[o]; r.e = A.x[o]; r.d = A.rhs[o];
    } else {
        constexpr bool X = KIND == TDMA_X9 || KIND == TDMA_X5, NINE = KIND == TDMA_X9 || KIND == TDMA_Y9;
        const int nx = A.nx, ny = A.ny, i = X ? q : l, j = X ? l : q;
        const long long N = (long long)nx * ny, np = (long long)j * nx + i;
        const double *__restrict__ a = A.a;
        const double *__restrict__ x = A.x;
        const bool hw = i > 0, he = i < nx - 1, hs = j > 0, hn = j < ny - 1;
        double d = A.b[np];
        if (NINE) {
            r.w = PL(a, X ? 4 : 2, np); r.c = PL(a, 5, np); r.e = PL(a, X ? 6 : 8, np);
            if (X) {
                if (hs && hw) d = d - PL(a, 1, np) * x[np - nx - 1];
                if (hs) d = d - PL(a, 2, np) * x[np - nx];
                if (hs && he) d = d - PL(a, 3, np) * x[np - nx + 1];
                if (hn && hw) d = d - PL(a, 7, np) * x[np + nx - 1];
                if (hn) d = d - PL(a, 8, np) * x[np + nx];
                if (hn && he) d = d - PL(a, 9, np) * x[np + nx + 1];
            } else {
                if (hw && hs) d = d - PL(a, 1, np) * x[np - nx - 1];
                if (hw) d = d - PL(a, 4, np) * x[np - 1];
                if (hw && hn) d = d - PL(a, 7, np) * x[np + nx - 1];
                if (he && hs) d = d - PL(a, 3, np) * x[np - nx + 1];
                if (he) d = d - PL(a, 6, np) * x[np + 1];
                if (he && hn) d = d - PL(a, 9, np) * x[np + nx + 1];
            }
        } else {
            r.w = PL(a, X ? 2 : 1, np); r.c = PL(a, 3, np); r.e = PL(a, X ? 4 : 5, np);
            if (X) {
                if (hn) d = d - PL(a, 5, np) * x[np + nx];
                if (hs) d = d - PL(a, 1, np) * x[np - nx];
            } else {
                if (hw) d = d - PL(a, 2, np) * x[np - 1];
                if (he) d = d - PL(a, 4, np) * x[np + 1];
            }
        }
        r.d = d;
    }
    if (q == 0) r.w = -0.0;      // no predecessor (P = 0, Q = -0): c + w P = c and d - w Q = d, zeros of either sign too
    return r;
}

template <int KIND, int LPC>
__global__ void __launch_bounds__(kTdmaThreads) k_tdma(TdmaArgs A)
{
    constexpr bool X = KIND != TDMA_Y9 && KIND != TDMA_Y5;
    constexpr int CH = kTdmaChunk, E = CH * LPC;
    extern __shared__ double smem[];
    __shared__ int bad;
    double *buf = smem;                              // 3 chunks x {w, c, e, d} x E, element-major
    const int n = X ? A.nx : A.ny, m = X ? A.ny : A.nx;
    const int l0 = blockIdx.x * LPC, nl = min(LPC, m - l0);
    // P, Q of element q of line l0 + l
    double *Pp, *Qp;
    long long si, sl;
    if (A.in_smem) {
        Pp = buf + 12 * E; Qp = Pp + (long long)n * LPC;
        si = LPC; sl = 1;
    } else {
        si = X ? 1 : A.nx; sl = X ? A.nx : 1;
        Pp = A.P + l0 * sl; Qp = A.Q + l0 * sl;
    }
    const int nch = (n + CH - 1) / CH;
    auto load = [&](int c, int t, int T) {           // chunk c by threads t of T
        double *d = buf + (c % 3) * 4 * E;
        for (int k = t; k < E; k += T) {
            // consecutive threads along memory: elements of an x line, the
            // LPC neighbours of a y line
            const int l = X ? k / CH : k % LPC, e = X ? k % CH : k / LPC, q = c * CH + e;
            if (q >= n || l >= nl) continue;
            const TdmaRow r = tdma_row<KIND>(A, l0 + l, q);
            const int o = e * LPC + l;
            d[o] = r.w; d[E + o] = r.c; d[2 * E + o] = r.e; d[3 * E + o] = r.d;
        }
    };
    auto check = [&](int c, int t, int T) {
        const double *d = buf + (c % 3) * 4 * E;
        bool ok = true;
        for (int k = t; k < E; k += T) {
            const int e = k / LPC, l = k % LPC, q = c * CH + e;
            if (q >= n || l >= nl) continue;
            const double pw = q > 0 ? Pp[(q - 1) * si + l * sl] : 0.0, qw = q > 0 ? Qp[(q - 1) * si + l * sl] : -0.0;
            const double rhs = d[3 * E + k], den = d[E + k] + d[k] * pw, num = rhs - d[k] * qw;
            double &pv = Pp[q * si + l * sl], &qv = Qp[q * si + l * sl];
            ok = ok & quot_ok(-d[2 * E + k], den, pv) & quot_ok(num, den, qv);
            // The sign of a zero is set here: the recurrence's other values do
            // not depend on it, nor does num's unless -0 - w Q has a zero Q,
            // whose own sign may be set at this moment.
            const bool ps = quot_sign_ok(-d[2 * E + k], den, pv), qs = quot_sign_ok(num, den, qv);
            const bool minus0 = ((__double2hiint(rhs) ^ (int)0x80000000) | __double2loint(rhs)) == 0;
            if (!(ps & qs & !minus0)) {
                if (!ps) pv = -pv;
                if (!qs) qv = -qv;
                ok = ok & !(minus0 && q > 0 && qw == 0.0);
            }
        }
        if (!ok) bad = 1;
    };
    const int lane = threadIdx.x;
    auto forward = [&](auto ieee_tag, bool checked) {
        constexpr bool IEEE = decltype(ieee_tag)::value;
        double p = 0.0, v = -0.0;
        load(0, threadIdx.x, kTdmaThreads);
        for (int c = 0; c <= nch; c++) {
            __syncthreads();
            if (threadIdx.x >= 32) {
                if (c + 1 < nch) load(c + 1, threadIdx.x - 32, kTdmaThreads - 32);
                if (checked && c > 0) check(c - 1, threadIdx.x - 32, kTdmaThreads - 32);
            } else if (c < nch && lane < nl) {
                const double *d = buf + (c % 3) * 4 * E + lane;
                const int cnt = min(CH, n - c * CH);
                double *pp = Pp + (long long)c * CH * si + lane * sl, *qq = Qp + (long long)c * CH * si + lane * sl;
                double w = d[0], cc = d[E], ee = d[2 * E], dd = d[3 * E];
#pragma unroll 4
                for (int e = 0; e < cnt; e++) {
                    const double w1 = w, c1 = cc, e1 = ee, d1 = dd;
                    const int o = min(e + 1, CH - 1) * LPC;   // the next element, loaded a step ahead
                    w = d[o]; cc = d[E + o]; ee = d[2 * E + o]; dd = d[3 * E + o];
                    const double den = c1 + w1 * p;
                    const double num = d1 - w1 * v;
                    if (IEEE) {
                        p = -e1 / den;
                        v = num / den;
                    } else {
                        const Rcp r = rcp_start(den);
                        p = div_plus(-e1, den, r);
                        v = div_plus(num, den, r);
                    }
                    pp[e * si] = p;
                    qq[e * si] = v;
                }
            }
        }
        __syncthreads();
    };
    if (threadIdx.x == 0) bad = 0;
    forward(std::false_type{}, true);
    if (bad) forward(std::true_type{}, false);
    if (lane < nl) {
        double *pp = Pp + lane * sl, *qq = Qp + lane * sl;
        double v = qq[(n - 1) * si];
#pragma unroll 8
        for (int q = n - 2; q >= 0; q--) {
            v = pp[q * si] * v + qq[q * si];
            qq[q * si] = v;
        }
    }
    __syncthreads();
    const int total = n * nl;
    for (int k = threadIdx.x; k < total; k += kTdmaThreads) {
        const int l = X ? k / n : k % nl, q = X ? k % n : k / nl;
        const long long o = X ? (long long)(l0 + l) * A.nx + q : (long long)q * A.nx + l0 + l;
        A.out[o] = Qp[q * si + l * sl];
    }
}

template <int KIND, int LPC>
cudaError_t launch_tdma_phase(TdmaArgs A, cudaStream_t st, size_t limit = kTdmaSmem)
{
    constexpr bool X = KIND != TDMA_Y9 && KIND != TDMA_Y5;
    const int n = X ? A.nx : A.ny, m = X ? A.ny : A.nx;
    const size_t chunks = (size_t)12 * kTdmaChunk * LPC * sizeof(double);
    const size_t lines = (size_t)2 * n * LPC * sizeof(double);
    A.in_smem = chunks + lines <= limit;             // longer lines keep P and Q in global memory
    const size_t sm = chunks + (A.in_smem ? lines : 0);
    const cudaError_t e = cudaFuncSetAttribute(k_tdma<KIND, LPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTdmaSmem);
    if (e != cudaSuccess) return e;
    k_tdma<KIND, LPC><<<(m + LPC - 1) / LPC, kTdmaThreads, sm, st>>>(A);
    return cudaGetLastError();
}

// One thread per line, for batches so large that many threads hide the
// memory's latency better than CTAs with a recurrence on a few lanes.
__global__ void k_tdma_batch(TdmaArgs A)
{
    const int l = blockIdx.x * blockDim.x + threadIdx.x, n = A.nx;
    if (l >= A.ny) return;
    const long long o = (long long)l * n;
    const double *__restrict__ w = A.a + o, *__restrict__ c = A.b + o, *__restrict__ e = A.x + o;
    const double *__restrict__ d = A.rhs + o;
    double *P = A.P + o, *Q = A.Q + o, *out = A.out + o;
    double p = -e[0] / c[0], v = d[0] / c[0];
    P[0] = p; Q[0] = v;
    for (int q = 1; q < n; q++) {
        const double den = c[q] + w[q] * p;
        p = -e[q] / den;
        v = (d[q] - w[q] * v) / den;
        P[q] = p; Q[q] = v;
    }
    out[n - 1] = v;
    for (int q = n - 2; q >= 0; q--) {
        v = P[q] * v + Q[q];
        out[q] = v;
    }
}
}  // namespace

cudaError_t launch_tdma(int nd, int nx, int ny, int nitm, const double *a, const double *b,
                        double *x, double *P, double *Q, cudaStream_t st)
{
    cudaError_t e = cudaSuccess;
    for (int it = 0; it < nitm && e == cudaSuccess; it++) {
        // x lines: x -> Q, y lines: Q -> x.  A row's loads are coalesced with
        // one line per CTA; four columns make the 32-byte sectors of a y line.
        TdmaArgs A = {nx, ny, a, b, x, nullptr, Q, P, Q, 0};
        e = nd == 9 ? launch_tdma_phase<TDMA_X9, 1>(A, st) : launch_tdma_phase<TDMA_X5, 1>(A, st);
        A.x = Q;
        A.out = A.Q = x;
        if (e == cudaSuccess)
            e = nd == 9 ? launch_tdma_phase<TDMA_Y9, 4>(A, st) : launch_tdma_phase<TDMA_Y5, 4>(A, st);
    }
    return e;
}

// independent lines: P = -ae/(ap + aw P_w), Q = (d - aw Q_w)/(ap + aw P_w)
cudaError_t launch_tdma_lines(int n, int nlines, const double *aw, const double *ap,
                              const double *ae, const double *d, double *x, double *P,
                              double *Q, cudaStream_t st)
{
    const TdmaArgs A = {n, nlines, aw, ap, ae, d, x, P, Q, 0};
    // One line per CTA is the fastest way through a few lines.  From about
    // 1000 on CTAs queue for the SMs, and four lines share one warp's
    // instructions: 300 elements, 512 lines 32.9 us with one and 34.6 with four,
    // 2400 75 and 50, 10000 250 and 132.  A CTA's P and Q stay in shared memory
    // while three CTAs fit in an SM, to 768 elements; past that four lines gain
    // only from about 1200 on, in global memory (1000 elements, 5000 lines 409
    // and 438 us; 2000, 2400 lines 607 and 458).  Where a batch moves many MB,
    // or lines are short beside a CTA's start-up, one thread per line is the
    // faster: 30000 lines of 8 elements 17.8 us against 29 with four per CTA, of
    // 30 40.7 and 47, of 1000 1400 and 2140; but of 100 141 and 120.
    if ((nlines >= 4096 && n <= 16) || (nlines >= 20000 && (n < 64 || n >= 700))) {
        k_tdma_batch<<<(nlines + 63) / 64, 64, 0, st>>>(A);
        return cudaGetLastError();
    }
    if ((nlines >= 1000 && n <= 768) || (nlines >= 2400 && n >= 1200))
        return launch_tdma_phase<TDMA_LINES, 4>(A, st, kTdmaSmem / 3);
    return launch_tdma_phase<TDMA_LINES, 1>(A, st);
}

// Parallel cyclic reduction, one CTA per line, the line's four coefficient
// arrays in shared memory (ping-pong between two copies).  With the line
// written aw_i x_{i-1} + ap_i x_i + ae_i x_{i+1} = d_i, a step of stride s
// eliminates x_{i-s} and x_{i+s} from row i with rows i-s and i+s:
//   k1 = aw_i / ap_{i-s},  k2 = ae_i / ap_{i+s}   (0 past the line's ends)
//   aw'_i = -aw_{i-s} k1,  ae'_i = -ae_{i+s} k2
//   ap'_i = ap_i - ae_{i-s} k1 - aw_{i+s} k2
//   d'_i  = d_i - d_{i-s} k1 - d_{i+s} k2
// so after ceil(log2 n) steps every row holds one unknown: x_i = d_i / ap_i
// (Hockney's cyclic reduction in its parallel form).  Global loads and
// stores are whole coalesced lines.  The rounding differs from the
// sequential Thomas algorithm (k_tdma_lines); for diagonally dominant lines
// the two agree to about 1e-15 relative.
constexpr int kPcrThreads = 256;
constexpr int kPcrMaxN = 2048;

__global__ void __launch_bounds__(kPcrThreads) k_tdma_lines_pcr(int n, int nlines, const double *__restrict__ aw,
                                                                const double *__restrict__ ap,
                                                                const double *__restrict__ ae,
                                                                const double *__restrict__ d, double *x)
{
    extern __shared__ double pcr[];   // 2 copies x {aw, ap, ae, d} x n
    const int l = blockIdx.x;
    if (l >= nlines) return;
    const long long o = (long long)l * n;
    double *A0 = pcr, *B0 = A0 + n, *C0 = B0 + n, *D0 = C0 + n;
    double *A1 = D0 + n, *B1 = A1 + n, *C1 = B1 + n, *D1 = C1 + n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        A0[i] = aw[o + i]; B0[i] = ap[o + i]; C0[i] = ae[o + i]; D0[i] = d[o + i];
    }
    __syncthreads();
    for (int sft = 1; sft < n; sft <<= 1) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int im = i - sft, ip = i + sft;
            const double k1 = im >= 0 ? A0[i] / B0[im] : 0.0;
            const double k2 = ip < n ? C0[i] / B0[ip] : 0.0;
            const double am = im >= 0 ? A0[im] : 0.0, cm = im >= 0 ? C0[im] : 0.0, dm = im >= 0 ? D0[im] : 0.0;
            const double ap_ = ip < n ? A0[ip] : 0.0, cp = ip < n ? C0[ip] : 0.0, dp = ip < n ? D0[ip] : 0.0;
            A1[i] = -am * k1;
            C1[i] = -cp * k2;
            B1[i] = B0[i] - cm * k1 - ap_ * k2;
            D1[i] = D0[i] - dm * k1 - dp * k2;
        }
        __syncthreads();
        double *t;
        t = A0; A0 = A1; A1 = t;
        t = B0; B0 = B1; B1 = t;
        t = C0; C0 = C1; C1 = t;
        t = D0; D0 = D1; D1 = t;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) x[o + i] = D0[i] / B0[i];
}

bool tdma_lines_pcr_supported(int n) { return n >= 1 && n <= kPcrMaxN; }

cudaError_t launch_tdma_lines_pcr(int n, int nlines, const double *aw, const double *ap, const double *ae,
                                  const double *d, double *x, cudaStream_t st)
{
    if (!tdma_lines_pcr_supported(n) || nlines < 1) return cudaErrorInvalidValue;
    const size_t smem = (size_t)8 * n * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_tdma_lines_pcr, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(8 * kPcrMaxN * sizeof(double)));
    if (e != cudaSuccess) return e;
    k_tdma_lines_pcr<<<nlines, kPcrThreads, smem, st>>>(n, nlines, aw, ap, ae, d, x);
    return cudaGetLastError();
}

}  // namespace m2d
