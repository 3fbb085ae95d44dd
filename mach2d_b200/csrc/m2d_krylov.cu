// m2d_krylov.cu -- flexible GMRES around the MSI preconditioner and the
// learned p' correction.  No counterpart in the reference: MACH-2D iterates
// MSI as a stationary method (fb2d9 / fb2d5, src/solvers/msi2d9-v03.f90:
// 42-262).  This solver keeps MSI's incomplete factorisation (lu2d9 /
// lu2d5, computed once per solve, as the reference computes it once per
// call) and uses it as the right preconditioner of Saad's flexible GMRES
// (SIAM J. Sci. Comput. 14, 1993), so the Krylov space replaces the fixed
// point iteration x += (LU)^-1 (b - A x).  The preconditioner may change
// from one Krylov step to the next, which lets the learned correction (a
// nonlinear map) act as a preconditioner too: z = N(v), then one MSI step
// from it, z += (LU)^-1 (v - A z).
//
// Device work per step: one MSI application (the cluster kernel with
// reused factors: forward and backward sweeps only), one product A z, two
// passes of classical Gram-Schmidt (h = V^T w in one launch, w -= V h in
// another, done twice for orthogonality), a norm.  The FP64 dot products use
// a fixed per-block order and a fixed final order, so a solve is bitwise
// reproducible.  The small Hessenberg least-squares problem (Givens
// rotations) lives on the host.
#include <cmath>
#include <cstring>
#include <vector>
#include "m2d_solvers.cuh"
#include "../../include/mach2d_b200.h"

void m2d_set_last_error_msg(const char *);

namespace m2d {
// the learned correction x_out = x + N(b - A x) (m2d_unet.cu), no acceptance test
cudaError_t unet_correct(m2d_unet *n, int nx, int ny, const double *d_a, const double *d_b, const double *d_x,
                         double *d_xout, const double *d_Jp, cudaStream_t st);
}

using namespace m2d;

namespace {

constexpr int kThreads = 256;
constexpr int kBlocks = 296;          // 2 per SM
constexpr int kMaxRestart = 32;       // accumulators per thread in the multi-dot

#define PLK(a, k, np) (a)[(long long)(k) * N + (np)]

// r = b - A x (sign 1) or w = A x (sign 0, b unused), every cell; couplings
// to cells outside the grid are dropped, as in the MSI residual.  One block per
// 128 cells of a row: bandwidth bounds it, and a thread that took its cell's
// row and column out of one 64-bit index spent longer on that division than on
// its 19 loads (1026x514: 15.0 us so, 9.9 now; 46 MB).
template <int ND>
__global__ void k_apply_a(int nx, int ny, const double *__restrict__ a, const double *__restrict__ b,
                          const double *__restrict__ x, double *y, int residual)
{
    const long long N = (long long)nx * ny;
    const int j = blockIdx.y, i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < nx) {
        const long long np = (long long)j * nx + i;
        const bool w = i > 0, e = i < nx - 1, s = j > 0, n = j < ny - 1;
        double v = 0.0;
        if (ND == 9) {
            if (s && w) v = v + PLK(a, 0, np) * x[np - nx - 1];
            if (s) v = v + PLK(a, 1, np) * x[np - nx];
            if (s && e) v = v + PLK(a, 2, np) * x[np - nx + 1];
            if (w) v = v + PLK(a, 3, np) * x[np - 1];
            v = v + PLK(a, 4, np) * x[np];
            if (e) v = v + PLK(a, 5, np) * x[np + 1];
            if (n && w) v = v + PLK(a, 6, np) * x[np + nx - 1];
            if (n) v = v + PLK(a, 7, np) * x[np + nx];
            if (n && e) v = v + PLK(a, 8, np) * x[np + nx + 1];
        } else {
            if (s) v = v + PLK(a, 0, np) * x[np - nx];
            if (w) v = v + PLK(a, 1, np) * x[np - 1];
            v = v + PLK(a, 2, np) * x[np];
            if (e) v = v + PLK(a, 3, np) * x[np + 1];
            if (n) v = v + PLK(a, 4, np) * x[np + nx];
        }
        y[np] = residual ? b[np] - v : v;
    }
}

// out[i] = sum_c V_i[c] w[c] over c < N, i < k (k <= kMaxRestart, rows of V ld
// doubles apart).  Block (x, y) sums rows R y ... of slice x, a contiguous one
// of kBlocks, into part[i * kBlocks + x]; the last block of a y (counted in
// count[y], left at zero) adds its rows' parts in slice order.  The order of
// the additions does not depend on k or R.
//
// Bandwidth bounds it: R rows at a time keep R loads in flight per thread and
// the blocks of all rows on the GPU at once, where a thread with an
// accumulator for every row waited for one load after the other; the parts'
// sum in the same launch saves a second one of a single warp.  1026x514, the
// mean over a 20-vector cycle: 34 us with the second launch, 11.5 now.
template <int R>
__global__ void __launch_bounds__(kThreads) k_multidot(int k, long long N, long long ld, const double *__restrict__ V,
                                                       const double *__restrict__ w, double *part, unsigned *count,
                                                       double *out)
{
    const int i0 = blockIdx.y * R, rows = k - i0 < R ? k - i0 : R;
    const double *v[R];
    double acc[R];
#pragma unroll
    for (int q = 0; q < R; q++) {
        v[q] = V + (long long)(i0 + (q < rows ? q : rows - 1)) * ld;   // (rows past the last repeat it)
        acc[q] = 0.0;
    }
    const long long per = (N + gridDim.x - 1) / gridDim.x;
    const long long lo = per * blockIdx.x, hi = lo + per < N ? lo + per : N;
#pragma unroll 4
    for (long long c = lo + threadIdx.x; c < hi; c += kThreads) {
        const double wc = w[c];
#pragma unroll
        for (int q = 0; q < R; q++) acc[q] = acc[q] + v[q][c] * wc;
    }
    __shared__ double red[kThreads / 32][R];
    __shared__ double parts[R * kBlocks];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < R; q++) {
        double t = acc[q];
        for (int o = 16; o > 0; o >>= 1) t = t + __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) red[wp][q] = t;
    }
    __syncthreads();
    if ((int)threadIdx.x < rows) {
        double t = 0.0;
        for (int q = 0; q < kThreads / 32; q++) t = t + red[q][threadIdx.x];
        part[(long long)(i0 + threadIdx.x) * kBlocks + blockIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(count + blockIdx.y, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int t = threadIdx.x; t < rows * kBlocks; t += kThreads) parts[t] = __ldcg(part + (long long)i0 * kBlocks + t);
    __syncthreads();
    if ((int)threadIdx.x < rows) {
        double t = 0.0;
#pragma unroll 8
        for (int q = 0; q < kBlocks; q++) t = t + parts[threadIdx.x * kBlocks + q];
        out[i0 + threadIdx.x] = t;
    }
    if (threadIdx.x == 0) count[blockIdx.y] = 0;
}

// y += sign * sum_{i < k} h[i] X_i over c < N (rows of X ld apart, h in
// device memory)
__global__ void k_multi_axpy(int k, long long N, long long ld, const double *__restrict__ X,
                             const double *__restrict__ h, double sign, double *y)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N;
         c += (long long)gridDim.x * blockDim.x) {
        double v = y[c];
        for (int i = 0; i < k; i++) v = v + sign * h[i] * X[(long long)i * ld + c];
        y[c] = v;
    }
}

// y = x / |x|, where *ss = |x|^2
__global__ void k_normalise(long long N, const double *__restrict__ x, const double *ss, double *y)
{
    const double f = 1.0 / sqrt(*ss);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N;
         c += (long long)gridDim.x * blockDim.x)
        y[c] = x[c] * f;
}

int fail(int code, const char *msg)
{
    m2d_set_last_error_msg(msg);
    return code;
}

struct Layout {
    long long N;
    double *V, *Z, *w, *t, *ws, *part, *h;
    size_t ws_doubles;
};

// slots of Layout::h: the two passes' dots, |w|^2, a constant 1, and the
// multi-dot's block counters
constexpr int kH2 = kMaxRestart, kHw = 2 * kMaxRestart, kHOne = kHw + 1, kHCount = kHw + 2;
constexpr int kRows = 4;      // rows per block of the multi-dot
static_assert(kHCount * sizeof(double) + (kMaxRestart / kRows) * sizeof(unsigned) <= (2 * kMaxRestart + 8) * sizeof(double),
              "the counters fit");

size_t align32(size_t n) { return (n + 31) / 32 * 32; }

Layout layout(int nd, int nx, int ny, int m, double *base)
{
    Layout L;
    L.N = (long long)nx * ny;
    const size_t Na = align32((size_t)L.N);
    double *p = base;
    L.V = p; p += (size_t)(m + 1) * Na;
    L.Z = p; p += (size_t)m * Na;
    L.w = p; p += Na;
    L.t = p; p += Na;
    L.ws_doubles = align32(msi_work_doubles(nd, nx, ny) + 4);
    L.ws = p; p += L.ws_doubles;
    L.part = p; p += align32((size_t)kMaxRestart * kBlocks);
    L.h = p; p += align32(2 * kMaxRestart + 8);
    return L;
}

size_t workspace_doubles(int nd, int nx, int ny, int m)
{
    const size_t Na = align32((size_t)nx * ny);
    return (size_t)(2 * m + 3) * Na + align32(msi_work_doubles(nd, nx, ny) + 4) + align32((size_t)kMaxRestart * kBlocks)
           + align32(2 * kMaxRestart + 8);
}

}  // namespace

extern "C" long m2d_fgmres_workspace_doubles(int nd, int nx, int ny, int restart)
{
    if ((nd != 9 && nd != 5) || nx < 4 || ny < 4 || restart < 1 || restart > kMaxRestart) return -1;
    return (long)workspace_doubles(nd, nx, ny, restart);
}

extern "C" int m2d_fgmres_solve(int nd, int nx, int ny, int restart, int maxit, double tol, const double *d_a,
                                const double *d_b, double *d_x, int prec, m2d_unet *net, const double *d_Jp,
                                double *d_work, void *stream, m2d_fgmres_report *rep)
{
    if ((nd != 9 && nd != 5) || nx < 4 || ny < 4 || restart < 1 || restart > kMaxRestart || maxit < 1 ||
        !(tol > 0.0) || !d_a || !d_b || !d_x || !d_work || prec < 0 || prec > 2)
        return fail(M2D_ERR_ARG, "m2d_fgmres_solve: bad arguments");
    if (prec == 2 && (nd != 5 || !net || !d_Jp))
        return fail(M2D_ERR_ARG, "m2d_fgmres_solve: the learned preconditioner needs nd = 5, a network and Jp");
    if (ny > msi_max_ny()) return fail(M2D_ERR_TOO_LARGE, "m2d_fgmres_solve: ny exceeds m2d_msi_max_ny()");
    if (((uintptr_t)d_work) % 16) return fail(M2D_ERR_ARG, "m2d_fgmres_solve: d_work must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const int m = restart;
    Layout W = layout(nd, nx, ny, m, d_work);
    const long long N = W.N;
    const size_t Na = align32((size_t)N);
    const unsigned g = (unsigned)((N + kThreads - 1) / kThreads < 1184 ? (N + kThreads - 1) / kThreads : 1184);
    cudaError_t e = cudaSuccess;
    int msi_apps = 0, net_apps = 0, total = 0, restarts = 0;
    bool factored = false, converged = false;
    std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), gv(m + 1), hcol(m + 2);
    double bnorm = 0.0, resid = 0.0;

    auto apply_a = [&](const double *x, double *y, const double *b, int residual) {
        const dim3 ga((unsigned)((nx + 127) / 128), (unsigned)ny);   // (ny <= msi_max_ny())
        if (nd == 9) k_apply_a<9><<<ga, 128, 0, st>>>(nx, ny, d_a, b, x, y, residual);
        else k_apply_a<5><<<ga, 128, 0, st>>>(nx, ny, d_a, b, x, y, residual);
    };
    // dots of the first k rows of X with y into W.h[at..at + k)
    auto dots = [&](int k, const double *X, const double *y, int at) -> cudaError_t {
        unsigned *count = (unsigned *)(W.h + kHCount);
        if (k == 1) k_multidot<1><<<kBlocks, kThreads, 0, st>>>(1, N, (long long)Na, X, y, W.part, count, W.h + at);
        else k_multidot<kRows><<<dim3(kBlocks, (unsigned)((k + kRows - 1) / kRows)), kThreads, 0, st>>>(
                 k, N, (long long)Na, X, y, W.part, count, W.h + at);
        return cudaGetLastError();
    };
    auto to_host = [&](double *host, int at, int n) -> cudaError_t {
        cudaError_t ee = cudaMemcpyAsync(host, W.h + at, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, st);
        if (ee == cudaSuccess) ee = cudaStreamSynchronize(st);
        return ee;
    };
    // |x|^2 into W.h[kHw] and to the host
    auto square = [&](const double *x, double *host) -> cudaError_t {
        const cudaError_t ee = dots(1, x, x, kHw);
        return ee == cudaSuccess ? to_host(host, kHw, 1) : ee;
    };
    // one application of the factors: y = (LU)^-1 rhs, y zeroed here; the
    // first call of a solve also factorises (and runs the full iteration
    // step, which from y = 0 gives the same y)
    auto apply_factors = [&](const double *rhs, double *y) -> cudaError_t {
        cudaError_t ee = cudaMemsetAsync(y, 0, (size_t)N * sizeof(double), st);
        if (ee != cudaSuccess) return ee;
        MsiLaunch L;
        memset(&L, 0, sizeof L);
        L.nx = nx; L.ny = ny; L.nitm = 1; L.tol = 0.0;
        L.prec = (prec >= 1) ? 1 : 0;
        L.reuse_lu = factored ? 1 : 0;
        L.apply_only = factored ? 1 : 0;
        L.s[0].a = d_a; L.s[0].b = rhs; L.s[0].x = y;
        L.s[0].ws = W.ws;
        L.s[0].rr = W.ws + (W.ws_doubles - 4);
        L.ws_cap = W.ws_doubles - 4;
        ee = launch_msi(nd, L, 1, st);
        factored = true;
        msi_apps++;
        return ee;
    };
    // the preconditioner: z = P(v)
    auto precondition = [&](const double *v, double *z) -> cudaError_t {
        if (prec != 2) return apply_factors(v, z);
        // z = N(v) from the zero guess, then z += (LU)^-1 (v - A z)
        cudaError_t ee = cudaMemsetAsync(W.w, 0, (size_t)N * sizeof(double), st);
        if (ee == cudaSuccess) ee = unet_correct(net, nx, ny, d_a, v, W.w, z, d_Jp, st);
        if (ee != cudaSuccess) return ee;
        net_apps++;
        apply_a(z, W.t, v, 1);
        ee = apply_factors(W.t, W.w);
        if (ee != cudaSuccess) return ee;
        const double one = 1.0;
        ee = cudaMemcpyAsync(W.h + kHOne, &one, sizeof(double), cudaMemcpyHostToDevice, st);
        if (ee != cudaSuccess) return ee;
        k_multi_axpy<<<g, kThreads, 0, st>>>(1, N, (long long)Na, W.w, W.h + kHOne, 1.0, z);
        return cudaGetLastError();
    };

    e = cudaMemsetAsync(W.h + kHCount, 0, (kMaxRestart / kRows) * sizeof(unsigned), st);
    {
        // |b|
        double hb = 0.0;
        if (e == cudaSuccess) e = square(d_b, &hb);
        bnorm = std::sqrt(hb);
    }
    while (e == cudaSuccess && !converged && total < maxit) {
        // r = b - A x into V_0, beta = |r|
        apply_a(d_x, W.V, d_b, 1);
        double hb = 0.0;
        e = square(W.V, &hb);
        if (e != cudaSuccess) break;
        const double beta = std::sqrt(hb);
        resid = beta;
        if (!(beta > tol * bnorm)) { converged = std::isfinite(beta); break; }
        k_normalise<<<g, kThreads, 0, st>>>(N, W.V, W.h + kHw, W.V);
        std::fill(gv.begin(), gv.end(), 0.0);
        gv[0] = beta;
        int jdone = 0;
        for (int j = 0; j < m && total < maxit; j++) {
            double *Vj = W.V + (size_t)j * Na, *Zj = W.Z + (size_t)j * Na, *Vn = W.V + (size_t)(j + 1) * Na;
            e = precondition(Vj, Zj);
            if (e != cudaSuccess) break;
            apply_a(Zj, W.w, nullptr, 0);
            // classical Gram-Schmidt, twice, and the new vector; the host reads
            // the column once they are all queued (read pass by pass the GPU
            // waited for it three times an iteration: 1026x514, 18 iterations
            // 14.0 ms so, 11.7 now with the dots above)
            for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
                const int at = pass ? kH2 : 0;
                e = dots(j + 1, W.V, W.w, at);
                if (e != cudaSuccess) break;
                k_multi_axpy<<<g, kThreads, 0, st>>>(j + 1, N, (long long)Na, W.V, W.h + at, -1.0, W.w);
            }
            if (e == cudaSuccess) e = dots(1, W.w, W.w, kHw);
            if (e != cudaSuccess) break;
            k_normalise<<<g, kThreads, 0, st>>>(N, W.w, W.h + kHw, Vn);
            double hh[kHw + 1];
            e = to_host(hh, 0, kHw + 1);
            if (e != cudaSuccess) break;
            for (int i = 0; i <= j; i++) hcol[i] = hh[i] + hh[kH2 + i];
            hcol[j + 1] = std::sqrt(hh[kHw]);
            // Givens rotations on the new column
            for (int i = 0; i < j; i++) {
                const double t = cs[i] * hcol[i] + sn[i] * hcol[i + 1];
                hcol[i + 1] = -sn[i] * hcol[i] + cs[i] * hcol[i + 1];
                hcol[i] = t;
            }
            const double den = std::hypot(hcol[j], hcol[j + 1]);
            cs[j] = den > 0.0 ? hcol[j] / den : 1.0;
            sn[j] = den > 0.0 ? hcol[j + 1] / den : 0.0;
            hcol[j] = den;
            hcol[j + 1] = 0.0;
            gv[j + 1] = -sn[j] * gv[j];
            gv[j] = cs[j] * gv[j];
            for (int i = 0; i <= j; i++) H[(size_t)i * m + j] = hcol[i];
            total++;
            jdone = j + 1;
            resid = std::fabs(gv[j + 1]);
            if (!std::isfinite(resid)) { e = cudaErrorUnknown; break; }
            if (resid <= tol * bnorm) break;
        }
        if (e != cudaSuccess || jdone == 0) break;
        // y = H^-1 g, x += Z y
        std::vector<double> y(jdone);
        for (int i = jdone - 1; i >= 0; i--) {
            double s = gv[i];
            for (int k = i + 1; k < jdone; k++) s -= H[(size_t)i * m + k] * y[k];
            y[i] = s / H[(size_t)i * m + i];
        }
        e = cudaMemcpyAsync(W.h, y.data(), (size_t)jdone * sizeof(double), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) break;
        k_multi_axpy<<<g, kThreads, 0, st>>>(jdone, N, (long long)Na, W.Z, W.h, 1.0, d_x);
        restarts++;
        if (resid <= tol * bnorm) converged = true;
    }
    if (e == cudaErrorUnknown) return fail(M2D_ERR_NAN, "m2d_fgmres_solve: non-finite residual");
    if (e != cudaSuccess) {
        m2d_set_last_error(e, "m2d_fgmres_solve", __FILE__, __LINE__);
        return M2D_ERR_CUDA;
    }
    // the true residual of the result
    double rr = 0.0;
    apply_a(d_x, W.w, d_b, 1);
    e = square(W.w, &rr);
    if (e != cudaSuccess) {
        m2d_set_last_error(e, "m2d_fgmres_solve", __FILE__, __LINE__);
        return M2D_ERR_CUDA;
    }
    if (rep) {
        rep->iterations = total;
        rep->msi_applications = msi_apps;
        rep->learned_applications = net_apps;
        rep->cycles = restarts;
        rep->converged = converged ? 1 : 0;
        rep->rel_residual = bnorm > 0.0 ? std::sqrt(rr) / bnorm : std::sqrt(rr);
    }
    return converged ? M2D_OK : M2D_ERR_TIMEOUT;
}
