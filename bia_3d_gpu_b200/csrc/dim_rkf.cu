// dim_rkf.cu -- the direct-integration (DIM) FP64 reference solver on the device.
//
// Rebuilds dim/rkf_kernel.cu: all 6n equations y' = (v, a) with the direct-sum
// acceleration a_i = eps sum_j (r_i - r_j) / (|r_ij|^2 + 1e-99)^{3/2}
// (dim/rkf_kernel.cu:29-53) integrated from x0 to xe by the Fehlberg 4(5) pair with
// step doubling and the reference's adaptive control (dim/rkf_kernel.cu:194-495):
// the "low" track advances by one step h with the embedded error estimate, the "high"
// track by two steps h/2; a step is accepted when max_i |er_i| / et_i <= 1.
//
// Differences from the reference, none of which changes the scheme:
//  * the state stays on the device for the whole integration; per attempted step the
//    host reads one double (the error norm) instead of copying the 11*6n work array
//    both ways (dim/rkf_kernel.cu:290-292,485-489);
//  * the acceleration sum over j is split into 8 fixed chunks whose partial sums are
//    added in order (deterministic; the association differs from the reference's single
//    running sum by rounding only);
//  * errors set IER (10000 too many steps, 20000 zero tolerance, 30000 step underflow)
//    and return instead of calling exit(0) (dim/rkf_kernel.cu:298-315,491-494).
// Layout: SoA, component-major, 6 arrays of n (x, y, z, u, v, w).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "bia_internal.cuh"

namespace bia {

constexpr int kDimChunks = 8;
constexpr int kDimParticlesPerBlock = 32;

// Fehlberg coefficients (dim/rkf_kernel.cu:161-168); stage s (1..5) forms
// w_s = y0 + h * sum_m B[s][m] k_m, the 6th line forms yn with GA, the 7th er with DA.
__constant__ double c_fehl[7][6] = {
    {1.0 / 4, 0, 0, 0, 0, 0},
    {3.0 / 32, 9.0 / 32, 0, 0, 0, 0},
    {1932.0 / 2197, -7200.0 / 2197, 7296.0 / 2197, 0, 0, 0},
    {439.0 / 216, -8.0, 3680.0 / 513, -845.0 / 4104, 0, 0},
    {-8.0 / 27, 2.0, -3544.0 / 2565, 1859.0 / 4104, -11.0 / 40, 0},
    {16.0 / 135, 0, 6656.0 / 12825, 28561.0 / 56430, -9.0 / 50, 2.0 / 55},
    {1.0 / 360, 0, -128.0 / 4275, -2197.0 / 75240, 1.0 / 50, 2.0 / 55},
};

// k_out = (v, a)(y_in).  Block: 32 particles x 8 j-chunks; the chunk partial sums are
// added in chunk order.
__global__ void __launch_bounds__(kDimParticlesPerBlock * kDimChunks) dim_accel_kernel(
    int n, double eps, const double *__restrict__ yin, double *__restrict__ kout)
{
    __shared__ double part[kDimChunks][3][kDimParticlesPerBlock];
    const int lane = threadIdx.x % kDimParticlesPerBlock;
    const int chunk = threadIdx.x / kDimParticlesPerBlock;
    const int i = blockIdx.x * kDimParticlesPerBlock + lane;
    const double *X = yin, *Y = yin + n, *Z = yin + 2 * (size_t)n;
    double ax = 0.0, ay = 0.0, az = 0.0;
    if (i < n) {
        const double xi = X[i], yi = Y[i], zi = Z[i];
        const int per = (n + kDimChunks - 1) / kDimChunks;
        const int j0 = chunk * per;
        const int j1 = min(n, j0 + per);
        for (int j = j0; j < j1; j++) {
            const double xij = xi - X[j], yij = yi - Y[j], zij = zi - Z[j];
            const double rsq = xij * xij + yij * yij + zij * zij + 1e-99;
            const double eee = eps / (rsq * sqrt(rsq));
            ax += xij * eee;
            ay += yij * eee;
            az += zij * eee;
        }
    }
    part[chunk][0][lane] = ax;
    part[chunk][1][lane] = ay;
    part[chunk][2][lane] = az;
    __syncthreads();
    if (chunk == 0 && i < n) {
        double s[3] = {0.0, 0.0, 0.0};
        for (int c = 0; c < kDimChunks; c++)
            for (int d = 0; d < 3; d++) s[d] += part[c][d][lane];
        kout[i] = yin[3 * (size_t)n + i];
        kout[(size_t)n + i] = yin[4 * (size_t)n + i];
        kout[2 * (size_t)n + i] = yin[5 * (size_t)n + i];
        kout[3 * (size_t)n + i] = s[0];
        kout[4 * (size_t)n + i] = s[1];
        kout[5 * (size_t)n + i] = s[2];
    }
}

// out = y0 + h * sum_{m < nk} c_fehl[row][m] k_m  (row 0..5), or er = h * sum (row 6)
__global__ void __launch_bounds__(256) dim_combine_kernel(int len, int row, int nk, bool add_y0,
                                                          const double *__restrict__ hdev,
                                                          const double *__restrict__ y0,
                                                          const double *__restrict__ k, double *__restrict__ out)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= len) return;
    const double h = *hdev;
    double acc;
    if (row == 0) {
        acc = h * c_fehl[0][0] * k[e];  // (h * B21) * k1, dim/rkf_kernel.cu:82
    } else {
        acc = 0.0;
        for (int m = 0; m < nk; m++) acc += c_fehl[row][m] * k[(size_t)m * len + e];
        acc = h * acc;
    }
    out[e] = add_y0 ? y0[e] + acc : acc;
}

// per-block max of |er| / et with et = relerr (|yl0| + |yln|) / 2 + abserr; a zero et
// is flagged by a negative result
__global__ void __launch_bounds__(256) dim_errnorm_kernel(int len, double relerr, double abserr,
                                                          const double *__restrict__ yl0,
                                                          const double *__restrict__ yln,
                                                          const double *__restrict__ er, double *__restrict__ blockmax)
{
    __shared__ double sh[256];
    double m = 0.0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < len; e += gridDim.x * blockDim.x) {
        const double et = relerr * (fabs(yl0[e]) + fabs(yln[e])) / 2 + abserr;
        if (et == 0.0) m = -1.0e300;
        else if (m >= 0.0) m = fmax(m, fabs(er[e]) / et);
    }
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            const double a = sh[threadIdx.x], b = sh[threadIdx.x + s];
            sh[threadIdx.x] = (a < 0.0 || b < 0.0) ? -1.0e300 : fmax(a, b);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) blockmax[blockIdx.x] = sh[0];
}

// min over i with |k1_i| > 0 of |(relerr |y_i| + abserr) / k1_i| (initial step size,
// dim/rkf_kernel.cu:248-261); +inf when no k1_i is nonzero
__global__ void __launch_bounds__(256) dim_toldy_kernel(int len, double relerr, double abserr,
                                                        const double *__restrict__ y, const double *__restrict__ k1,
                                                        double *__restrict__ blockmin)
{
    __shared__ double sh[256];
    double m = INFINITY;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < len; e += gridDim.x * blockDim.x) {
        if (fabs(k1[e]) > 0.0) m = fmin(m, fabs((relerr * fabs(y[e]) + abserr) / k1[e]));
    }
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] = fmin(sh[threadIdx.x], sh[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) blockmin[blockIdx.x] = sh[0];
}

__global__ void dim_final_reduce_kernel(int count, bool take_max, const double *__restrict__ in, double *out)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double m = take_max ? 0.0 : INFINITY;
    for (int b = 0; b < count; b++) {
        const double v = in[b];
        if (take_max) m = (m < 0.0 || v < 0.0) ? -1.0e300 : fmax(m, v);
        else m = fmin(m, v);
    }
    *out = m;
}

__global__ void __launch_bounds__(256) dim_esterr_kernel(int len, const double *__restrict__ yln,
                                                         const double *__restrict__ yhn, double *__restrict__ ese)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < len) ese[e] = (yln[e] - yhn[e]) / 31;
}

constexpr int kDimReduceBlocks = 148;
constexpr int kDimCoopMaxBlocks = 1024;  // partials of the cooperative solver's reductions

// Device buffers of one integration: 6n doubles each for yl0, yln, yh0, yhm, yhn, er, w
// and 6 x 6n for k1..k6; plus reduction scratch and the step size.
struct DimBuffers {
    double *yl0, *yln, *yh0, *yhm, *yhn, *er, *w, *wb, *k, *red, *h, *scal, *io;
    double *pos;  // the resident kernel's stage positions, [2 tracks][2 parities][3][n rounded up to even]: over k
};

struct DimRun {
    int n, len;
    bool fast_inv = false;  // the cooperative solver's rsqrt-based inverse cube
    double eps, relerr, abserr;
    cudaStream_t st;
    DimBuffers B;
    double *h_pinned;  // [0] h to upload, [1] reduction result read back
};

static unsigned grid_of(int len) { return (unsigned)((len + 255) / 256); }

// One Fehlberg step of size *hdev from y0: yn and (want_er) er (dim/rkf_kernel.cu fehl).
static cudaError_t dim_fehl(const DimRun &R, const double *y0, double *yn, bool want_er)
{
    const int n = R.n, len = R.len;
    const unsigned ga = (unsigned)((n + kDimParticlesPerBlock - 1) / kDimParticlesPerBlock);
    const unsigned threads = kDimParticlesPerBlock * kDimChunks;
    double *k = R.B.k;
    dim_accel_kernel<<<ga, threads, 0, R.st>>>(n, R.eps, y0, k);
    for (int s = 0; s < 5; s++) {
        dim_combine_kernel<<<grid_of(len), 256, 0, R.st>>>(len, s, s + 1, true, R.B.h, y0, k, R.B.w);
        dim_accel_kernel<<<ga, threads, 0, R.st>>>(n, R.eps, R.B.w, k + (size_t)(s + 1) * len);
    }
    dim_combine_kernel<<<grid_of(len), 256, 0, R.st>>>(len, 5, 6, true, R.B.h, y0, k, yn);
    if (want_er) dim_combine_kernel<<<grid_of(len), 256, 0, R.st>>>(len, 6, 6, false, R.B.h, y0, k, R.B.er);
    return cudaGetLastError();
}

static cudaError_t set_h(const DimRun &R, double h)
{
    R.h_pinned[0] = h;
    return cudaMemcpyAsync(R.B.h, R.h_pinned, sizeof(double), cudaMemcpyHostToDevice, R.st);
}

static cudaError_t read_scalar(const DimRun &R, double *out)
{
    cudaError_t e = cudaMemcpyAsync(R.h_pinned + 1, R.B.scal, sizeof(double), cudaMemcpyDeviceToHost, R.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(R.st);
    if (e == cudaSuccess) *out = R.h_pinned[1];
    return e;
}

// The adaptive loop of dim/rkf_kernel.cu:194-495 (INIT = 1 computes the first step).
// y (device SoA 6n) holds the state at *x0 on entry and the high track at xe on exit;
// ese (optional device 6n) the final (yln - yhn)/31.  Returns ier.
static int dim_integrate(DimRun &R, double *y, double *x0, double xe, int init, double *H, int *nde,
                         long long *accepted, long long *rejected, double *ese, int *status)
{
    const double EPSMIN = 1e-15;
    const int ITEMAX = 10000;
    const size_t bytes = (size_t)R.len * sizeof(double);
    cudaError_t e;
    *status = BIA_OK;
#define DIM_CHECK(x)                          \
    do {                                      \
        e = (x);                              \
        if (e != cudaSuccess) {               \
            *status = cuda_status(e);         \
            return 0;                         \
        }                                     \
    } while (0)
    DIM_CHECK(cudaMemcpyAsync(R.B.yh0, y, bytes, cudaMemcpyDeviceToDevice, R.st));
    DIM_CHECK(cudaMemcpyAsync(R.B.yl0, y, bytes, cudaMemcpyDeviceToDevice, R.st));
    *nde = 0;
    if (init == 1) {
        const unsigned ga = (unsigned)((R.n + kDimParticlesPerBlock - 1) / kDimParticlesPerBlock);
        dim_accel_kernel<<<ga, kDimParticlesPerBlock * kDimChunks, 0, R.st>>>(R.n, R.eps, R.B.yl0, R.B.k);
        dim_toldy_kernel<<<kDimReduceBlocks, 256, 0, R.st>>>(R.len, R.relerr, R.abserr, R.B.yl0, R.B.k, R.B.red);
        dim_final_reduce_kernel<<<1, 32, 0, R.st>>>(kDimReduceBlocks, false, R.B.red, R.B.scal);
        double toldy = 0.0;
        DIM_CHECK(read_scalar(R, &toldy));
        *H = std::isinf(toldy) ? EPSMIN * (xe - *x0) : fmin((xe - *x0) / 100e0, pow(toldy, 0.2));
        *nde = 1;
    }
    double X = *x0;
    int ier = 10000;
    for (int iter = 0; iter < ITEMAX; iter++) {
        DIM_CHECK(set_h(R, *H));
        DIM_CHECK(dim_fehl(R, R.B.yl0, R.B.yln, true));
        *nde += 6;
        dim_errnorm_kernel<<<kDimReduceBlocks, 256, 0, R.st>>>(R.len, R.relerr, R.abserr, R.B.yl0, R.B.yln,
                                                                 R.B.er, R.B.red);
        dim_final_reduce_kernel<<<1, 32, 0, R.st>>>(kDimReduceBlocks, true, R.B.red, R.B.scal);
        double erret = 0.0;
        DIM_CHECK(read_scalar(R, &erret));
        if (erret < 0.0) {
            ier = 20000;
            break;
        }
        if (erret > 1) {
            (*rejected)++;
            if (erret >= 59049) *H *= 0.1;
            else *H *= 0.9 / pow(erret, 0.2);
            if (*H <= EPSMIN) {
                ier = 30000;
                break;
            }
        } else if (X + *H < xe) {
            // two half steps on the high track (fhstep, dim/rkf_kernel.cu:318-362)
            DIM_CHECK(set_h(R, *H / 2));
            DIM_CHECK(dim_fehl(R, R.B.yh0, R.B.yhm, false));
            DIM_CHECK(dim_fehl(R, R.B.yhm, R.B.yhn, false));
            *nde += 12;
            X += *H;
            *x0 = X;
            DIM_CHECK(cudaMemcpyAsync(R.B.yl0, R.B.yln, bytes, cudaMemcpyDeviceToDevice, R.st));
            DIM_CHECK(cudaMemcpyAsync(R.B.yh0, R.B.yhn, bytes, cudaMemcpyDeviceToDevice, R.st));
            (*accepted)++;
            if (erret <= 1.889568e-4) *H *= 5.0;
            else *H *= 0.9 / pow(erret, 0.2);
        } else {
            // last step to xe (dim/rkf_kernel.cu:386-483)
            *H = xe - X;
            DIM_CHECK(set_h(R, *H));
            DIM_CHECK(dim_fehl(R, R.B.yl0, R.B.yln, true));
            DIM_CHECK(set_h(R, *H / 2));
            DIM_CHECK(dim_fehl(R, R.B.yh0, R.B.yhm, false));
            DIM_CHECK(dim_fehl(R, R.B.yhm, R.B.yhn, false));
            *nde += 18;
            if (ese) dim_esterr_kernel<<<grid_of(R.len), 256, 0, R.st>>>(R.len, R.B.yln, R.B.yhn, ese);
            DIM_CHECK(cudaMemcpyAsync(y, R.B.yhn, bytes, cudaMemcpyDeviceToDevice, R.st));
            DIM_CHECK(cudaMemcpyAsync(R.B.yl0, R.B.yln, bytes, cudaMemcpyDeviceToDevice, R.st));
            *x0 = xe;
            (*accepted)++;
            ier = 0;
            break;
        }
    }
    if (ier != 0) {  // leave the last accepted high-track state in y
        DIM_CHECK(cudaMemcpyAsync(y, R.B.yh0, bytes, cudaMemcpyDeviceToDevice, R.st));
    }
    DIM_CHECK(cudaStreamSynchronize(R.st));
#undef DIM_CHECK
    return ier;
}

static size_t dim_buffer_doubles(int n)
{
    const size_t len = (size_t)6 * n;
    return 8 * len + 6 * len + kDimCoopMaxBlocks + 16;
}

static void dim_carve(double *base, int n, DimBuffers &B)
{
    const size_t len = (size_t)6 * n;
    B.yl0 = base;
    B.yln = base + len;
    B.yh0 = base + 2 * len;
    B.yhm = base + 3 * len;
    B.yhn = base + 4 * len;
    B.er = base + 5 * len;
    B.w = base + 6 * len;
    B.k = base + 7 * len;
    // 16-byte aligned (base is, 7 len is even); 12 (n + 1) <= 36 n doubles
    B.pos = B.k;
    B.wb = base + 13 * len;
    B.red = base + 14 * len;
    B.h = B.red + kDimCoopMaxBlocks;
    B.scal = B.h + 1;
    B.io = B.scal + 2;  // 6 doubles of the cooperative solver's inputs and outputs
}



// ---------------------------------------------------------------------------------------
// The whole adaptive integration in one cooperative kernel: the same stages, arithmetic
// and acceptance rule as dim_integrate below, with the step control on the device.  Every
// block computes the decisions from the same grid-wide reductions (bitwise the same
// values), so all blocks take the same path and meet at the same grid-wide barriers; the
// loop is bounded by ITEMAX attempted steps.  Tracks are swapped, not copied.
namespace cg = cooperative_groups;

struct DimCoopArgs {
    int n, len, init, itemax;
    double eps, relerr, abserr, xe;
    DimBuffers B;   // B.red holds >= gridDim.x doubles
    double *y;      // state in (at io[0]) and out
    double *ese;    // optional (yln - yhn) / 31 of the last step
    double *io;     // in: [0] x0, [1] H; out: [0] x reached, [1] H, [2] nde, [3] accepted,
                    // [4] rejected, [5] ier
};

// Fused stage of the cooperative solver: k_s = (v, a)(win) for a group of P particles, and
// right away, by the thread that owns particle i, the next stage's input for particle i:
// w = y0 + h sum_m c_fehl[s][m] k_m (s < 5), or yn (row 5) and er (row 6) after the last
// stage.  The combination is per particle, so only the next stage needs a grid-wide
// barrier.
//
// j-tiles: the block's 256 threads load the positions of 256 particles j at a time into
// shared memory (coalesced structure-of-arrays loads, one element per thread and
// component); thread (particle lane, chunk c) of the block's P x C threads (C = 256 / P)
// adds the tile's entries c, c + C, ..., and the C chunk sums of a particle are added in
// chunk order at the end (deterministic).  P = 32: each tile serves 32 particles, 32 entries per
// thread.  It takes the sizes beyond the resident kernel below (more than 224 particles a CTA, 33152 on 148 SMs).
//
// Inverse cube: kFastInv (bia_dim_integrate) eps r^-3 from one rsqrt (r^-1, then its cube;
// rsqrt is within 1 ulp, the product within ~4 ulp of eps / r^3); otherwise the
// reference's eps / (rsq sqrt(rsq)) (dim/rkf_kernel.cu:44-46), the form rkf_c_ keeps.
constexpr int kCoopTile = 256;
template <int P>
struct CoopShared {
    double part[256 / P][3][P];
    double tile[3][kCoopTile];
};

template <int P, bool kFastInv>
__device__ void coop_stage(const DimCoopArgs &A, int s, double h, const double *__restrict__ y0,
                           const double *__restrict__ win, double *__restrict__ wout, double *__restrict__ yn,
                           bool want_er, CoopShared<P> &sh)
{
    constexpr int C = 256 / P;
    const int n = A.n;
    const size_t len = (size_t)A.len;
    const int lane = threadIdx.x % P;
    const int chunk = threadIdx.x / P;
    const int ngroups = (n + P - 1) / P;
    const double *X = win, *Y = win + n, *Z = win + 2 * (size_t)n;
    double *k = A.B.k;
    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const int i = grp * P + lane;
        const bool live = i < n;
        const double xi = live ? X[i] : 0.0, yi = live ? Y[i] : 0.0, zi = live ? Z[i] : 0.0;
        double ax = 0.0, ay = 0.0, az = 0.0;
        for (int jt = 0; jt < n; jt += kCoopTile) {
            __syncthreads();  // the previous tile (or group) is consumed
            const int jl = jt + (int)threadIdx.x;
            if (jl < n) {
                sh.tile[0][threadIdx.x] = X[jl];
                sh.tile[1][threadIdx.x] = Y[jl];
                sh.tile[2][threadIdx.x] = Z[jl];
            }
            __syncthreads();
            const int cnt = min(kCoopTile, n - jt);
            if (live) {
                for (int q = chunk; q < cnt; q += C) {
                    const double xij = xi - sh.tile[0][q], yij = yi - sh.tile[1][q], zij = zi - sh.tile[2][q];
                    const double rsq = xij * xij + yij * yij + zij * zij + 1e-99;
                    double eee;
                    if (kFastInv) {
                        const double ir = rsqrt(rsq);
                        eee = A.eps * (ir * ir * ir);
                    } else {
                        eee = A.eps / (rsq * sqrt(rsq));
                    }
                    ax += xij * eee;
                    ay += yij * eee;
                    az += zij * eee;
                }
            }
        }
        sh.part[chunk][0][lane] = ax;
        sh.part[chunk][1][lane] = ay;
        sh.part[chunk][2][lane] = az;
        __syncthreads();
        if (chunk == 0 && live) {
            double a3[3] = {0.0, 0.0, 0.0};
            for (int c = 0; c < C; c++)
                for (int d = 0; d < 3; d++) a3[d] += sh.part[c][d][lane];
            double *ks = k + (size_t)s * len;
            for (int c = 0; c < 3; c++) {
                ks[(size_t)c * n + i] = win[(size_t)(3 + c) * n + i];
                ks[(size_t)(3 + c) * n + i] = a3[c];
            }
            for (int c = 0; c < 6; c++) {
                const size_t e = (size_t)c * n + i;
                if (s < 5) {
                    double acc;
                    if (s == 0) {
                        acc = h * c_fehl[0][0] * k[e];
                    } else {
                        acc = 0.0;
                        for (int m = 0; m <= s; m++) acc += c_fehl[s][m] * k[(size_t)m * len + e];
                        acc = h * acc;
                    }
                    wout[e] = y0[e] + acc;
                } else {
                    double acc = 0.0;
                    for (int m = 0; m < 6; m++) acc += c_fehl[5][m] * k[(size_t)m * len + e];
                    yn[e] = y0[e] + h * acc;
                    if (want_er) {
                        double ae = 0.0;
                        for (int m = 0; m < 6; m++) ae += c_fehl[6][m] * k[(size_t)m * len + e];
                        A.B.er[e] = h * ae;
                    }
                }
            }
        }
    }
    __syncthreads();
}

// One Fehlberg step of size h: six fused stages, one grid-wide barrier after each.
template <int P, bool kFastInv>
__device__ void coop_fehl(const DimCoopArgs &A, cg::grid_group &grid, double h, const double *y0, double *yn,
                          bool want_er, CoopShared<P> &part)
{
    // stage inputs alternate between two scratch vectors so a stage never overwrites the
    // input other blocks are still reading: w_a for even stages' output, w_b for odd
    double *wa = A.B.w, *wb = A.B.wb;
    const double *win = y0;
    for (int st = 0; st < 6; st++) {
        double *wout = (st % 2 == 0) ? wa : wb;
        coop_stage<P, kFastInv>(A, st, h, y0, win, wout, yn, want_er, part);
        grid.sync();
        win = wout;
    }
}

// grid-wide max of |er| / et (negative when an et is zero), the same on every block
__device__ double coop_errnorm(const DimCoopArgs &A, cg::grid_group &grid, const double *yl0, const double *yln,
                               double *sh)
{
    double m = 0.0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < A.len; e += gridDim.x * blockDim.x) {
        const double et = A.relerr * (fabs(yl0[e]) + fabs(yln[e])) / 2 + A.abserr;
        if (et == 0.0) m = -1.0e300;
        else if (m >= 0.0) m = fmax(m, fabs(A.B.er[e]) / et);
    }
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int s2 = 128; s2 > 0; s2 >>= 1) {
        if (threadIdx.x < s2) {
            const double a = sh[threadIdx.x], b = sh[threadIdx.x + s2];
            sh[threadIdx.x] = (a < 0.0 || b < 0.0) ? -1.0e300 : fmax(a, b);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) A.B.red[blockIdx.x] = sh[0];
    grid.sync();
    __shared__ double total;
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int b = 0; b < (int)gridDim.x; b++) {
            const double v = A.B.red[b];
            t = (t < 0.0 || v < 0.0) ? -1.0e300 : fmax(t, v);
        }
        total = t;
    }
    __syncthreads();
    const double r = total;
    __syncthreads();
    return r;
}

template <int P, bool kFastInv>
__global__ void __launch_bounds__(256) dim_coop_kernel(const DimCoopArgs A)
{
    cg::grid_group grid = cg::this_grid();
    __shared__ CoopShared<P> part;
    __shared__ double sh[256];
    __shared__ double total;
    const double EPSMIN = 1e-15;
    const int len = A.len;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, gsz = gridDim.x * blockDim.x;
    double *yl0 = A.B.yl0, *yln = A.B.yln, *yh0 = A.B.yh0, *yhn = A.B.yhn;
    for (int e = gid; e < len; e += gsz) {
        yh0[e] = A.y[e];
        yl0[e] = A.y[e];
    }
    double X = A.io[0], H = A.io[1];
    int nde = 0;
    grid.sync();
    if (A.init == 1) {
        coop_stage<P, kFastInv>(A, 0, 0.0, yl0, yl0, A.B.wb, nullptr, false, part);  // k1 only (w unused)
        grid.sync();
        double m = INFINITY;
        for (int e = gid; e < len; e += gsz)
            if (fabs(A.B.k[e]) > 0.0) m = fmin(m, fabs((A.relerr * fabs(yl0[e]) + A.abserr) / A.B.k[e]));
        sh[threadIdx.x] = m;
        __syncthreads();
        for (int s2 = 128; s2 > 0; s2 >>= 1) {
            if (threadIdx.x < s2) sh[threadIdx.x] = fmin(sh[threadIdx.x], sh[threadIdx.x + s2]);
            __syncthreads();
        }
        if (threadIdx.x == 0) A.B.red[blockIdx.x] = sh[0];
        grid.sync();
        if (threadIdx.x == 0) {
            double t = INFINITY;
            for (int b = 0; b < (int)gridDim.x; b++) t = fmin(t, A.B.red[b]);
            total = t;
        }
        __syncthreads();
        const double toldy = total;
        H = isinf(toldy) ? EPSMIN * (A.xe - X) : fmin((A.xe - X) / 100e0, pow(toldy, 0.2));
        nde = 1;
        grid.sync();  // the reduction scratch is reused below
    }
    long long acc = 0, rej = 0;
    int ier = 10000;
    for (int iter = 0; iter < A.itemax; iter++) {
        coop_fehl<P, kFastInv>(A, grid, H, yl0, yln, true, part);
        nde += 6;
        const double erret = coop_errnorm(A, grid, yl0, yln, sh);
        if (erret < 0.0) {
            ier = 20000;
            break;
        }
        if (erret > 1) {
            rej++;
            if (erret >= 59049) H *= 0.1;
            else H *= 0.9 / pow(erret, 0.2);
            if (H <= EPSMIN) {
                ier = 30000;
                break;
            }
        } else if (X + H < A.xe) {
            coop_fehl<P, kFastInv>(A, grid, H / 2, yh0, A.B.yhm, false, part);
            coop_fehl<P, kFastInv>(A, grid, H / 2, A.B.yhm, yhn, false, part);
            nde += 12;
            X += H;
            double *t1 = yl0; yl0 = yln; yln = t1;  // accepted: the new tracks become the old ones
            double *t2 = yh0; yh0 = yhn; yhn = t2;
            acc++;
            if (erret <= 1.889568e-4) H *= 5.0;
            else H *= 0.9 / pow(erret, 0.2);
        } else {
            H = A.xe - X;
            coop_fehl<P, kFastInv>(A, grid, H, yl0, yln, true, part);
            coop_fehl<P, kFastInv>(A, grid, H / 2, yh0, A.B.yhm, false, part);
            coop_fehl<P, kFastInv>(A, grid, H / 2, A.B.yhm, yhn, false, part);
            nde += 18;
            X = A.xe;
            acc++;
            ier = 0;
            break;
        }
    }
    // outputs: the state (the high track at xe, or the last accepted one), the low track
    // in B.yl0, (yln - yhn) / 31
    const double *yout = (ier == 0) ? yhn : yh0;
    const double *lout = (ier == 0) ? yln : yl0;
    for (int e = gid; e < len; e += gsz) {
        if (A.ese && ier == 0) A.ese[e] = (yln[e] - yhn[e]) / 31;
        A.y[e] = yout[e];
    }
    grid.sync();
    if (lout != A.B.yl0)
        for (int e = gid; e < len; e += gsz) A.B.yl0[e] = lout[e];
    if (gid == 0) {
        A.io[0] = X;
        A.io[1] = H;
        A.io[2] = nde;
        A.io[3] = (double)acc;
        A.io[4] = (double)rej;
        A.io[5] = ier;
    }
}

// ---------------------------------------------------------------------------------------
// The resident solver: the same integration with every particle's whole state (tracks, stage derivatives)
// in the shared memory of the CTA that owns it, one CTA per SM.  Between stages only the stage
// positions cross the device: a CTA publishes its particles' (24 bytes each), the grid meets, and
// every CTA streams all positions through shared memory in double-buffered tiles.
//
// A derivative of dim_coop_kernel took 6 us at n = 200 and 12 at 1332, mostly latency: stage sums through
// global memory, 8 warps per SM on the forces, a serial loop over the blocks' error norms.  Here
// * 16 warps share a CTA's particles: lanes hold P x R of them (R in registers, P across lanes) and the
//   32/P lane groups of the 16 warps split the tile's positions (dim_shape picks P and R);
// * the low track's step and the high track's first half step do not depend on one another and run their
//   stages together while a stage is mostly latency (dual): 12 grid-wide barriers a step instead of
//   18.  An attempt that is rejected has done the half step for nothing (rejections are rare);
// * the error norm's partials travel with the last stage and are read by one warp;
// * the integration is one loop over stages, so that nothing lives in local memory across a barrier (its
//   fence empties L1).
// Forces: eps r^-3 by the reciprocal square root's approximation and one third-order step, 15 FP64
// operations an interaction (the sum takes eps once); a particle whose sum is not finite (positions
// beyond 1e154) is summed again with rsqrt.
//
// Measured, a derivative: n = 200 3.1 us (dim_coop_kernel 6.0), 1332 7.4 (11.9), 4096 26 (56), 6000 54 (97), 32768
// 1183 (2204).  What bounds it: at n = 32768 the interactions (35 cycles of register reads each, 85 % of
// the stage); at 1332 they are 9200 of a stage's 21000 cycles, the barrier 3600, fetching the
// positions 3400, the sums 3300; at 200 latency throughout.
constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxR = 7;

struct DimResArgs {
    int n, npad, own;  // own: particles per CTA (the last may have fewer)
    int P, init, itemax;
    int dual;          // low step and first half step together
    int tile;          // positions per tile
    int rows;          // rows of warp sums kept at a time: 16, 8 or 4
    double eps, relerr, abserr, xe;
    double *pos;  // [2 tracks][2 parities][3][npad]
    double *red;  // [gridDim.x]
    double *y, *ese, *yl0, *er, *io;  // as DimCoopArgs
};

// shared memory, in doubles: two tiles, the warps' partial sums, the forces of two tracks, their stage velocities
// (two parities), five state vectors, the error, the stage derivatives of one or two tracks
static size_t res_smem_doubles(int own, int slots, int tile, int rows, bool dual)
{
    return 2 * 3 * (size_t)tile + (size_t)rows * 3 * slots + (6 + 12 + 36 + (dual ? 72 : 36)) * (size_t)own;
}

__device__ __forceinline__ void cp_async16(double *dst, const double *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// force on a particle whose sum overflowed: every position again, rsqrt's full range
static __device__ __noinline__ double dim_force_again(const double *pos, int n, int npad, int i, int c, double eps)
{
    const double xi = __ldcg(pos + i), yi = __ldcg(pos + npad + i), zi = __ldcg(pos + 2 * (size_t)npad + i);
    double a = 0.0;
    for (int j = 0; j < n; j++) {
        const double d[3] = {xi - __ldcg(pos + j), yi - __ldcg(pos + npad + j), zi - __ldcg(pos + 2 * (size_t)npad + j)};
        const double rsq = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + 1e-99;
        const double ir = rsqrt(rsq);
        a += d[c] * (eps * (ir * ir * ir));
    }
    return a;
}

// maximum (negative wins) or minimum
__device__ __forceinline__ double res_pick(double a, double b, bool take_max)
{
    return take_max ? ((a < 0.0 || b < 0.0) ? -1.0e300 : fmax(a, b)) : fmin(a, b);
}

extern __shared__ __align__(16) double res_smem[];

// What a pass over six stages is: the first step size, an attempted low step (with the first half step when
// dual), the half steps of an accepted one, and the same to the end.
enum ResPhase { kResInit, kResTry, kResHalf1, kResHalf2, kResLast, kResLastHalf1, kResLastHalf2, kResDone };

template <int R, bool kFastInv>
__global__ void __launch_bounds__(kResThreads, 1) dim_resident_kernel(const DimResArgs A)
{
    cg::grid_group grid = cg::this_grid();
    __shared__ double s_red[kResWarps];
    __shared__ double s_total;
    const double EPSMIN = 1e-15;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int own = A.own, P = A.P, slots = P * R, npad = A.npad;
    const int first = blockIdx.x * own, mine = min(own, A.n - first);
    const int ntiles = (A.n + A.tile - 1) / A.tile;
    double *const tiles = res_smem;                 // [2][3][tile]
    double *const part = tiles + 2 * 3 * A.tile;    // [rows][3][slots]
    double *const force = part + A.rows * 3 * slots;  // [2][3][own]
    double *const vel = force + 6 * own;            // [2 tracks][2 stage parities][3][own]
    double *const vec = vel + 12 * own;             // the state vectors, [6][own] each
    const int vlen = 6 * own;
    double *yl0 = vec, *yln = vec + vlen, *yh0 = vec + 2 * vlen, *yhn = vec + 3 * vlen;
    double *const yhm = vec + 4 * vlen, *const er = vec + 5 * vlen;
    double *const kbuf = vec + 6 * vlen;            // [1 or 2][6 stages][6][own]
    const size_t track = 6 * (size_t)npad, half = 3 * (size_t)npad;

    // positions of state vector y as track t's next stage input
    auto publish = [&](int t, const double *y, int parity) {
        double *dst = A.pos + t * track + parity * half + first;
        for (int e = tid; e < 96; e += kResThreads) {  // three warps, one a component
            for (int i = lane; i < mine; i += 32) dst[(size_t)warp * npad + i] = y[warp * own + i];
        }
    };
    // the block's value over its threads' v, into its slot of A.red, before a barrier
    auto block_value = [&](double v, bool take_max) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = res_pick(v, __shfl_xor_sync(0xffffffffu, v, o), take_max);
        if (lane == 0) s_red[warp] = v;
        __syncthreads();
        if (tid == 0) {
            double m = s_red[0];
            for (int w = 1; w < kResWarps; w++) m = res_pick(m, s_red[w], take_max);
            A.red[blockIdx.x] = m;
        }
    };
    // the grid's value, after the barrier: every CTA reads the same partials
    auto grid_value = [&](bool take_max) {
        if (warp == 0) {
            double m = take_max ? 0.0 : INFINITY;
            for (int b = lane; b < (int)gridDim.x; b += 32) m = res_pick(m, __ldcg(A.red + b), take_max);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = res_pick(m, __shfl_xor_sync(0xffffffffu, m, o), take_max);
            if (lane == 0) s_total = m;
        }
        __syncthreads();
        return s_total;
    };

    for (int c = warp; c < 6; c += kResWarps)
        for (int i = lane; i < mine; i += 32)
            yl0[c * own + i] = yh0[c * own + i] = A.y[(size_t)c * A.n + first + i];
    double X = A.io[0], H = A.io[1];
    int nde = 0, acc = 0, rej = 0, iter = 0, ier = 10000, parity = 0, s = 0;
    int phase = A.init == 1 ? kResInit : kResTry;
    bool to_end = false;  // the attempted step reaches xe
    __syncthreads();
    publish(0, yl0, parity);
    publish(1, yh0, parity);
    grid.sync();
    if (phase == kResTry) to_end = !(X + H < A.xe);

#pragma unroll 1
    while (phase != kResDone) {
        // the tracks of this stage: t0 .. t0 + nt - 1, from y0 by h into yn
        const int t0 = (phase == kResHalf1 || phase == kResHalf2 || phase == kResLastHalf1 || phase == kResLastHalf2) ? 1 : 0;
        const int nt = (A.dual && ((phase == kResTry && !to_end) || phase == kResLast)) ? 2 : 1;

        // forces of this CTA's particles in those tracks from their published positions
        {
            const int total = nt * ntiles;
            const double *src0 = A.pos + t0 * track + parity * half;
            auto issue = [&](int q) {
                const int u = q >= ntiles ? 1 : 0, jt = q - u * ntiles;
                const double *src = src0 + u * track + jt * A.tile;
                double *dst = tiles + (q & 1) * 3 * A.tile;
                const int pieces = (min(A.tile, A.n - jt * A.tile) + 1) / 2;  // 16 bytes (npad is even)
                for (int e = tid; e < pieces; e += kResThreads) {
#pragma unroll
                    for (int c = 0; c < 3; c++) cp_async16(dst + c * A.tile + 2 * e, src + (size_t)c * npad + 2 * e);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            issue(0);
            if (total > 1) issue(1);
            const int pi = lane & (P - 1);
            const int js = lane / P + (32 / P) * warp, nj = kResThreads / P;
            double xi[R], yi[R], zi[R], ax[R], ay[R], az[R];
#pragma unroll 1
            for (int q = 0; q < total; q++) {
                const int u = q >= ntiles ? 1 : 0, jt = q - u * ntiles;
                if (jt == 0) {
                    const double *p = src0 + u * track;
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const int i = min(first + min(r * P + pi, own - 1), A.n - 1);
                        xi[r] = __ldcg(p + i);
                        yi[r] = __ldcg(p + npad + i);
                        zi[r] = __ldcg(p + 2 * (size_t)npad + i);
                        ax[r] = ay[r] = az[r] = 0.0;
                    }
                }
                if (q + 1 < total) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncthreads();
                const double *T = tiles + (q & 1) * 3 * A.tile;
                const int cnt = min(A.tile, A.n - jt * A.tile);
                constexpr int kUnroll = R >= 3 ? 1 : R == 2 ? 2 : 4;  // chains side by side; more spills
#pragma unroll kUnroll
                for (int j = js; j < cnt; j += nj) {
                    const double xj = T[j], yj = T[A.tile + j], zj = T[2 * A.tile + j];
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const double dx = xi[r] - xj, dy = yi[r] - yj, dz = zi[r] - zj;
                        if (kFastInv) {
                            const double rsq = fma(dx, dx, fma(dy, dy, fma(dz, dz, 1e-99)));
                            double y;
                            asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(rsq));
                            const double y2 = y * y;  // exact: the low half of y is zero
                            const double e = fma(-rsq, y2, 1.0);
                            const double y3 = y * y2;
                            const double w = fma(y3 * e, fma(e, 1.875, 1.5), y3);
                            ax[r] = fma(dx, w, ax[r]);
                            ay[r] = fma(dy, w, ay[r]);
                            az[r] = fma(dz, w, az[r]);
                        } else {
                            const double rsq = dx * dx + dy * dy + dz * dz + 1e-99;
                            const double w = A.eps / (rsq * sqrt(rsq));
                            ax[r] += dx * w;
                            ay[r] += dy * w;
                            az[r] += dz * w;
                        }
                    }
                }
                if (jt == ntiles - 1) {
                    // the lane groups' sums, the warps' onto A.rows rows in turn, then the rows in order
                    for (int o = P; o < 32; o <<= 1) {
#pragma unroll
                        for (int r = 0; r < R; r++) {
                            ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
                            ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
                            az[r] += __shfl_xor_sync(0xffffffffu, az[r], o);
                        }
                    }
                    double *pw = part + (warp & (A.rows - 1)) * 3 * slots;
                    for (int w0 = 0; w0 < kResWarps; w0 += A.rows) {
                        if (warp >= w0 && warp < w0 + A.rows && lane < P) {
#pragma unroll
                            for (int r = 0; r < R; r++) {
                                const int sl = r * P + lane;
                                pw[sl] = (w0 == 0 ? 0.0 : pw[sl]) + ax[r];
                                pw[slots + sl] = (w0 == 0 ? 0.0 : pw[slots + sl]) + ay[r];
                                pw[2 * slots + sl] = (w0 == 0 ? 0.0 : pw[2 * slots + sl]) + az[r];
                            }
                        }
                        __syncthreads();
                    }
                    // one lane a row, two sums a warp (rows beyond A.rows add zero)
                    for (int e = 2 * warp + (lane >> 4); e - (lane >> 4) < 3 * mine; e += 2 * kResWarps) {
                        const int c = e < mine ? 0 : e < 2 * mine ? 1 : 2, i = e - c * mine, w = lane & 15;
                        double a = e < 3 * mine && w < A.rows ? part[(w * 3 + c) * slots + i] : 0.0;
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                        if (w == 0 && e < 3 * mine) {
                            if (kFastInv) {
                                a *= A.eps;
                                if (!isfinite(a)) a = dim_force_again(src0 + u * track, A.n, npad, first + i, c, A.eps);
                            }
                            force[((t0 + u) * 3 + c) * own + i] = a;
                        }
                    }
                }
                __syncthreads();  // the tile's buffer is free; the forces are there
                if (q + 2 < total) issue(q + 2);
            }
        }

        if (phase == kResInit) {  // first step size (dim/rkf_kernel.cu:248-261)
            double m = INFINITY;
            for (int c = warp; c < 6; c += kResWarps)
                for (int i = lane; i < mine; i += 32) {
                    const double k1 = c < 3 ? yl0[(3 + c) * own + i] : force[(c - 3) * own + i];
                    if (fabs(k1) > 0.0) m = fmin(m, fabs((A.relerr * fabs(yl0[c * own + i]) + A.abserr) / k1));
                }
            block_value(m, false);
            grid.sync();
            const double toldy = grid_value(false);
            H = isinf(toldy) ? EPSMIN * (A.xe - X) : fmin((A.xe - X) / 100e0, pow(toldy, 0.2));
            nde = 1;
            phase = kResTry;
            to_end = !(X + H < A.xe);
            continue;
        }

        // stage s of those tracks: its derivative, and the next stage's input or, after the sixth, the new state
        double worst = 0.0;
        for (int row = warp; row < 6 * nt; row += kResWarps) {
            const int t = t0 + (row >= 6 ? 1 : 0), c = row >= 6 ? row - 6 : row;
            const double *y0 = t == 0 ? yl0 : (phase == kResHalf2 || phase == kResLastHalf2) ? yhm : yh0;
            double *yn = t == 0 ? yln : (phase == kResHalf2 || phase == kResLastHalf2) ? yhn : yhm;
            const double h = t == 0 ? H : H / 2;
            double *k0 = kbuf + (A.dual ? t : 0) * 6 * vlen + c * own;  // stage m at m vlen
            double *v = vel + t * vlen;                                  // [2 stage parities][3][own]
            for (int i = lane; i < mine; i += 32) {
                double *k = k0 + i;
                k[s * vlen] = c >= 3 ? force[(t * 3 + c - 3) * own + i]
                            : s == 0 ? y0[(3 + c) * own + i]
                                     : v[((s & 1) * 3 + c) * own + i];
                double sum = 0.0;
                if (s == 0) {
                    sum = h * c_fehl[0][0] * k[0];
                } else {
                    for (int m = 0; m <= s; m++) sum += c_fehl[s][m] * k[m * vlen];
                    sum = h * sum;
                }
                const double y = y0[c * own + i], w = y + sum;
                if (s < 5) {
                    if (c < 3) A.pos[t * track + (parity ^ 1) * half + (size_t)c * npad + first + i] = w;
                    else v[(((s + 1) & 1) * 3 + c - 3) * own + i] = w;
                } else {
                    yn[c * own + i] = w;
                    if (t == 0) {
                        double ae = 0.0;
                        for (int m = 0; m < 6; m++) ae += c_fehl[6][m] * k[m * vlen];
                        ae = h * ae;
                        er[c * own + i] = ae;
                        const double et = A.relerr * (fabs(y) + fabs(w)) / 2 + A.abserr;
                        if (et == 0.0) worst = -1.0e300;
                        else if (worst >= 0.0) worst = fmax(worst, fabs(ae) / et);
                    }
                }
            }
        }
        if (s < 5) {
            grid.sync();
            parity ^= 1;
            s++;
            continue;
        }

        // after the sixth stage: publish what comes next, meet, decide
        s = 0;
        if (phase == kResTry) block_value(worst, true);
        __syncthreads();
        if (phase == kResTry || phase == kResLast) {
            publish(1, nt == 2 ? yhm : yh0, parity ^ 1);
        } else if (phase == kResHalf1 || phase == kResLastHalf1) {
            publish(1, yhm, parity ^ 1);
        } else {
            publish(0, yln, parity ^ 1);
            publish(1, yhn, parity ^ 1);
        }
        grid.sync();
        parity ^= 1;
        if (phase == kResTry) {
            nde += 6;
            const double erret = grid_value(true);
            if (erret < 0.0) {
                ier = 20000;
                phase = kResDone;
            } else if (erret > 1) {
                rej++;
                if (erret >= 59049) H *= 0.1;
                else H *= 0.9 / pow(erret, 0.2);
                if (H <= EPSMIN) {
                    ier = 30000;
                    phase = kResDone;
                } else if (++iter >= A.itemax) {
                    phase = kResDone;
                } else {
                    publish(0, yl0, parity);
                    publish(1, yh0, parity);
                    grid.sync();
                    to_end = !(X + H < A.xe);
                }
            } else if (!to_end) {
                // the half steps of the high track (fhstep, dim/rkf_kernel.cu:318-362), and the next step's size
                if (tid == 0) s_red[0] = erret;  // for the end of the second half step
                phase = nt == 2 ? kResHalf2 : kResHalf1;
            } else {
                // last step to xe (dim/rkf_kernel.cu:386-483)
                H = A.xe - X;
                publish(0, yl0, parity);
                publish(1, yh0, parity);
                grid.sync();
                phase = kResLast;
            }
        } else if (phase == kResHalf1) {
            phase = kResHalf2;
        } else if (phase == kResHalf2) {
            const double erret = s_red[0];
            nde += 12;
            X += H;
            double *t1 = yl0; yl0 = yln; yln = t1;  // accepted: the new tracks become the old ones
            double *t2 = yh0; yh0 = yhn; yhn = t2;
            acc++;
            if (erret <= 1.889568e-4) H *= 5.0;
            else H *= 0.9 / pow(erret, 0.2);
            to_end = !(X + H < A.xe);
            phase = ++iter >= A.itemax ? kResDone : kResTry;
        } else if (phase == kResLast) {
            phase = nt == 2 ? kResLastHalf2 : kResLastHalf1;
        } else if (phase == kResLastHalf1) {
            phase = kResLastHalf2;
        } else {
            nde += 18;
            X = A.xe;
            acc++;
            ier = 0;
            phase = kResDone;
        }
    }
    __syncthreads();
    // outputs as dim_coop_kernel's: the state (the high track at xe, or the last accepted one), the low track,
    // (yln - yhn) / 31 and the last error estimate
    const double *yout = (ier == 0) ? yhn : yh0, *lout = (ier == 0) ? yln : yl0;
    for (int c = warp; c < 6; c += kResWarps)
        for (int i = lane; i < mine; i += 32) {
            const int at = c * own + i;
            const size_t g = (size_t)c * A.n + first + i;
            if (A.ese && ier == 0) A.ese[g] = (yln[at] - yhn[at]) / 31;
            A.y[g] = yout[at];
            A.yl0[g] = lout[at];
            A.er[g] = er[at];
        }
    if (blockIdx.x == 0 && tid == 0) {
        A.io[0] = X;
        A.io[1] = H;
        A.io[2] = nde;
        A.io[3] = (double)acc;
        A.io[4] = (double)rej;
        A.io[5] = ier;
    }
}

// Slots of the resident kernel for `own` particles per CTA: P across lanes, R in registers, the cheapest in
// cycles of the SM: 35 register-port cycles an interaction and warp on four schedulers and 12 a position
// read, and 64 for each value and step of the lane groups' sums (two shuffles from each of 16 warps, two
// cycles each).  Measured at n = 1332: P, R = 4, 3 11000 cycles a stage, 16, 1 12500.
static void dim_shape(int n, int own, int *P, int *R)
{
    double best = 0.0;
    *P = *R = 0;
    for (int p = 1, lg = 5; p <= 32; p *= 2, lg--) {
        const int r = (own + p - 1) / p;
        if (r > kResMaxR) continue;
        const double per_warp = (double)r * (double)((n + kResThreads / p - 1) / (kResThreads / p));
        const double cost = (140.0 + 48.0 / r) * per_warp + 192.0 * r * lg;
        if (*R == 0 || cost < best) {
            best = cost;
            *P = p;
            *R = r;
        }
    }
}

template <bool kFastInv>
static const void *dim_resident_form(int R)
{
    switch (R) {
    case 1: return (const void *)dim_resident_kernel<1, kFastInv>;
    case 2: return (const void *)dim_resident_kernel<2, kFastInv>;
    case 3: return (const void *)dim_resident_kernel<3, kFastInv>;
    case 4: return (const void *)dim_resident_kernel<4, kFastInv>;
    case 5: return (const void *)dim_resident_kernel<5, kFastInv>;
    case 6: return (const void *)dim_resident_kernel<6, kFastInv>;
    default: return (const void *)dim_resident_kernel<7, kFastInv>;
    }
}

// The resident kernel's launch for n particles on a device with `sms` SMs: false where the particles do not fit
// (more than kResMaxR x 32 a CTA, or the shared memory).  Larger tiles, more rows of warp sums and both
// tracks at once as far as the shared memory goes; both tracks only while a stage is mostly latency
// (measured at n = 6000 either way the same).
static bool dim_resident_plan(int n, int sms, size_t max_smem, DimResArgs &A, int *G, int *R, size_t *bytes)
{
    A.own = (n + sms - 1) / sms;
    *G = (n + A.own - 1) / A.own;
    if (*G > kDimCoopMaxBlocks) return false;
    dim_shape(n, A.own, &A.P, R);
    if (*R == 0) return false;
    for (int level = n <= 4096 ? 0 : 1; level < 4; level++) {
        A.dual = level == 0;
        A.tile = level < 3 ? 1024 : 512;
        A.rows = level < 2 ? kResWarps : 4;
        *bytes = res_smem_doubles(A.own, A.P * *R, A.tile, A.rows, A.dual != 0) * sizeof(double);
        if (*bytes <= max_smem) return true;
    }
    return false;
}

// The cooperative solver (dim_coop_kernel); *ran = false when the device cannot run it
// (no cooperative launch), and the caller takes the host-controlled loop instead.
static int dim_integrate_coop(DimRun &R, double *y, double *x0, double xe, int init, double *H, int *nde,
                              long long *accepted, long long *rejected, double *ese, int *status, bool *ran)
{
    *ran = false;
    *status = BIA_OK;
    const char *force_host = getenv("BIA_DIM_HOST_CONTROL");
    if (force_host && force_host[0] == '1') return 0;
    int dev = 0, coop = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    int max_smem = 0;
    if (cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    max_smem -= 1024;  // the kernel's static shared memory
    R.h_pinned[0] = *x0;
    R.h_pinned[1] = *H;
    int G = 0, reg = 0;
    size_t bytes = 0;
    const void *kern = nullptr;
    DimResArgs B;
    DimCoopArgs A;
    void *args[1];
    const char *gcap = getenv("BIA_DIM_COOP_BLOCKS");  // a cap on the blocks: the global-memory kernel's
    const int cap = gcap ? atoi(gcap) : 0;
    if (cap <= 0 && dim_resident_plan(R.n, sms, (size_t)max_smem, B, &G, &reg, &bytes)) {
        kern = R.fast_inv ? dim_resident_form<true>(reg) : dim_resident_form<false>(reg);
        // the limit belongs to the process: always the device's own, so that no call takes room from one that
        // another thread is about to launch
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        B.n = R.n;
        B.npad = (R.n + 1) & ~1;
        B.init = init;
        B.itemax = 10000;
        B.eps = R.eps;
        B.relerr = R.relerr;
        B.abserr = R.abserr;
        B.xe = xe;
        B.pos = R.B.pos;
        B.red = R.B.red;
        B.y = y;
        B.ese = ese;
        B.yl0 = R.B.yl0;
        B.er = R.B.er;
        B.io = R.B.io;
        args[0] = (void *)&B;
    } else {
        // too many particles for a CTA per SM (dim_resident_plan): groups of 32, all state in global memory
        kern = R.fast_inv ? (const void *)dim_coop_kernel<32, true> : (const void *)dim_coop_kernel<32, false>;
        bytes = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            return 0;
        }
        G = (R.n + 31) / 32;
        if (G > sms * per_sm) G = sms * per_sm;
        if (G > kDimCoopMaxBlocks) G = kDimCoopMaxBlocks;  // B.red holds kDimCoopMaxBlocks partials
        if (cap > 0 && cap < G) G = cap;
        A.n = R.n;
        A.len = R.len;
        A.init = init;
        A.itemax = 10000;
        A.eps = R.eps;
        A.relerr = R.relerr;
        A.abserr = R.abserr;
        A.xe = xe;
        A.B = R.B;
        A.y = y;
        A.ese = ese;
        A.io = R.B.io;
        args[0] = (void *)&A;
    }
    cudaError_t e = cudaMemcpyAsync(R.B.io, R.h_pinned, 2 * sizeof(double), cudaMemcpyHostToDevice, R.st);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel(kern, dim3(G), dim3(bytes ? kResThreads : 256), args, bytes, R.st);
    double out[6] = {0, 0, 0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(R.h_pinned, R.B.io, 6 * sizeof(double), cudaMemcpyDeviceToHost, R.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(R.st);
    if (e != cudaSuccess) {
        *status = cuda_status(e);
        *ran = true;
        return 0;
    }
    for (int k = 0; k < 6; k++) out[k] = R.h_pinned[k];
    *x0 = out[0];
    *H = out[1];
    *nde = (int)out[2];
    *accepted += (long long)out[3];
    *rejected += (long long)out[4];
    *ran = true;
    return (int)out[5];
}

struct DimDropIn {
    bool ready = false;
    DeviceBuffer buf, state;
    double *h_pinned = nullptr;
};
static thread_local DimDropIn g_dim;

}  // namespace bia

using namespace bia;

extern "C" int bia_dim_integrate(bia_context *ctx, int n, double eps_th, double *y, double x0, double xe,
                                 double relerr, double abserr, bia_dim_stats *stats)
{
    if (!ctx || n < 1 || !y || !(xe > x0)) return BIA_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    cudaError_t e = ctx->dim.reserve(dim_buffer_doubles(n) * sizeof(double));
    if (e != cudaSuccess) return cuda_status(e);
    if (!ctx->h_dim) {
        e = cudaMallocHost((void **)&ctx->h_dim, 8 * sizeof(double));
        if (e != cudaSuccess) return cuda_status(e);
    }
    DimRun R;
    R.n = n;
    R.len = 6 * n;
    R.eps = eps_th;
    R.relerr = relerr;
    R.abserr = abserr;
    R.st = ctx->stream;
    R.h_pinned = ctx->h_dim;
    R.fast_inv = true;
    dim_carve((double *)ctx->dim.ptr, n, R.B);
    double X = x0, H = 0.0;
    int nde = 0, status = BIA_OK;
    long long acc = 0, rej = 0;
    bool ran = false;
    int ier = dim_integrate_coop(R, y, &X, xe, 1, &H, &nde, &acc, &rej, nullptr, &status, &ran);
    if (!ran) ier = dim_integrate(R, y, &X, xe, 1, &H, &nde, &acc, &rej, nullptr, &status);
    if (stats) {
        stats->accepted = acc;
        stats->rejected = rej;
        stats->nde = nde;
        stats->ier = ier;
        stats->h_last = H;
        stats->x_reached = X;
    }
    if (status != BIA_OK) return status;
    return ier == 0 ? BIA_OK : BIA_ERR_NOT_CONVERGED;
}

// Drop-in for rkf_c_ (dim/rkf_kernel.cu:194-495), called from dim/dim_3D.f90:30 as
// RKF_C(%VAL(NEQ), %VAL(eps_th), X0, XE, Y0, INIT, RELERR, ABSERR, YN, ESTERR, NDE, IER,
// WK0, WK1, WK2, WK3, WK4).  Host arrays are AoS (x, y, z, u, v, w per particle).
extern "C" void rkf_c_(const int neq, const double eps_th, double *X0, double *XE, double *YH0, int *INIT,
                       const double *RELERR, const double *ABSERR, double *YHN, double *ESE, int *NDE, int *IER,
                       double *H, double *YL0, double *YLN, double *ERR, double *WRK)
{
    (void)WRK;
    if (neq < 6 || neq % 6 || !X0 || !XE || !YH0 || !INIT || !RELERR || !ABSERR || !YHN || !ESE || !NDE ||
        !IER || !H || !YL0 || !YLN || !ERR || !(*XE > *X0)) {
        set_last_error(BIA_ERR_INVALID_ARGUMENT);
        return;
    }
    const int n = neq / 6;
    DimDropIn &S = g_dim;
    cudaError_t e = cudaSuccess;
    if (!S.ready) {
        e = cudaMallocHost((void **)&S.h_pinned, 8 * sizeof(double));
        if (e != cudaSuccess) {
            set_last_error(cuda_status(e));
            return;
        }
        S.ready = true;
    }
    if ((e = S.buf.reserve(dim_buffer_doubles(n) * sizeof(double))) != cudaSuccess ||
        (e = S.state.reserve((size_t)2 * neq * sizeof(double))) != cudaSuccess) {
        set_last_error(cuda_status(e));
        return;
    }
    double *dy = (double *)S.state.ptr;       // SoA state
    double *dese = dy + neq;                  // SoA esterr
    // AoS host -> SoA device
    double *tmp = (double *)malloc(sizeof(double) * neq);
    if (!tmp) {
        set_last_error(BIA_ERR_OUT_OF_MEMORY);
        return;
    }
    for (int i = 0; i < n; i++)
        for (int c = 0; c < 6; c++) tmp[(size_t)c * n + i] = YH0[6 * (size_t)i + c];
    e = cudaMemcpy(dy, tmp, sizeof(double) * neq, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        free(tmp);
        set_last_error(cuda_status(e));
        return;
    }
    DimRun R;
    R.n = n;
    R.len = neq;
    R.eps = eps_th;
    R.relerr = *RELERR;
    R.abserr = *ABSERR;
    R.st = 0;
    R.h_pinned = S.h_pinned;
    dim_carve((double *)S.buf.ptr, n, R.B);
    int nde = 0, status = BIA_OK;
    long long acc = 0, rej = 0;
    const int init = *INIT;
    bool ran = false;
    int ier = dim_integrate_coop(R, dy, X0, *XE, init, H, &nde, &acc, &rej, dese, &status, &ran);
    if (!ran) ier = dim_integrate(R, dy, X0, *XE, init, H, &nde, &acc, &rej, dese, &status);
    if (init == 1) *INIT = 2;
    *NDE = nde;
    *IER = ier;
    if (status == BIA_OK) {
        // SoA device -> AoS host: YHN (high track), YL0 / YLN (low track), ESE, ERR
        double *outs[4] = {YHN, YLN, ESE, ERR};
        const double *srcs[4] = {dy, R.B.yl0, dese, R.B.er};
        for (int o = 0; o < 4 && e == cudaSuccess; o++) {
            if (ier != 0 && o == 2) continue;
            e = cudaMemcpy(tmp, srcs[o], sizeof(double) * neq, cudaMemcpyDeviceToHost);
            if (e == cudaSuccess)
                for (int i = 0; i < n; i++)
                    for (int c = 0; c < 6; c++) outs[o][6 * (size_t)i + c] = tmp[(size_t)c * n + i];
        }
        if (e == cudaSuccess) {
            memcpy(YL0, YLN, sizeof(double) * neq);  // after the last step YL0 = YLN
            if (ier == 0) memcpy(YH0, YHN, sizeof(double) * neq);
        }
        status = cuda_status(e);
    }
    free(tmp);
    set_last_error(status != BIA_OK ? status : (ier == 0 ? BIA_OK : BIA_ERR_NOT_CONVERGED));
}
