// invariance.cu -- conserved quantities of an N-body state on the device, FP64.
//
// Replaces invariance_gpu_ / inv_device / sum_device (bia/invariance.cu:15-110):
// sum x, sum v, sum L = x cross v, KE = sum |v|^2 (no 1/2) and
// PE = eps_th * sum_{i<j} 1/r_ij (bia/Invariance_CPU.f90:8-19), with optional charges
// (q_i q_j / r_ij).  The reference's inv_device gives thread i the whole row j > i
// (triangular imbalance, uncoalesced) and sum_device runs 11 serial sums on one thread
// each.  Here the pair sum uses the step kernel's 32 x 32 warp-blocks over the upper
// triangle, each CTA's partial goes to a fixed slot, and all partials are added in a
// fixed order, so the result is reproducible; a lane sums 32 pairs of a block, then blocks, then
// lanes, warps and CTAs, so that the rounding error stays far below n ulps.
#include <cuda_runtime.h>

#include "bia_internal.cuh"
#include "bia_pair.cuh"

namespace bia {

constexpr int kInvThreads = 256;
constexpr int kInvWarps = kInvThreads / 32;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    return v;
}

// Unit t of the pair sum: block rows 2 g and 2 g + 1 (as far as they are <= bj) of block column bj; the
// columns before bj hold floor((bj + 1)^2 / 4) units.
__host__ __device__ __forceinline__ long long inv_units_before(long long bj) { return (bj + 1) * (bj + 1) / 4; }

__device__ __forceinline__ void inv_unit_coords(long long t, int &g, int &bj)
{
    long long c = (long long)(2.0 * sqrt((double)t));
    while (inv_units_before(c) > t) c--;
    while (inv_units_before(c + 1) <= t) c++;
    bj = (int)c;
    g = (int)(t - inv_units_before(c));
}

// The lane's pairs of a block with roots and divisions: coincident, subnormal or overflowing separations.
static __device__ __noinline__ double inv_block_again(const double2 *xy, const double2 *zq, double xi, double yi, double zi,
                                                      double qi, int lane, bool diag, bool row_live, int ncols)
{
    double acc = 0.0;
    for (int k = diag ? 1 : 0; k <= (diag ? 16 : 31); k++) {
        const int src = (lane + k) & 31;
        if ((!diag || k < 16 || lane < 16) && row_live && src < ncols) {
            const double dx = xi - xy[src].x, dy = yi - xy[src].y, dz = zi - zq[src].x;
            acc += qi * zq[src].y * (1.0 / sqrt(dx * dx + dy * dy + dz * dz));
        }
    }
    return acc;
}

// The invariants in one launch: every CTA takes its share of the particles (the ten one-body sums) and of the
// pair sum (q_i q_j) / r_ij over i<j (one warp a unit of two 32 x 32 blocks of one block column), leaves its
// twelve sums in part[blockIdx.x][12], and the CTA that arrives last adds them up, one warp a sum, in block
// order: the result does not depend on which CTA that is.  out[12], order {KE, -, Lx, Ly, Lz, Ua, Va, Wa,
// Xa, Ya, Za, pair sum}.
//
// A pair is a distance and a reciprocal square root, 12 FP64 operations (28 register-read cycles a warp).
// Its column comes from two 16-byte shared-memory rows, eight cycles of the SM's one shared-memory port per
// scheduler, so a lane keeps two rows and reads a column once for both.  n = 32768: 1.46 ms with shuffled
// columns, 1/sqrt and one partial per 8 blocks added by a single CTA, 0.70 with one row a lane, 0.57 so.
__global__ void __launch_bounds__(kInvThreads) inv_kernel(int n, long long units, const double *x, const double *y,
                                                          const double *z, const double *u, const double *v,
                                                          const double *w, const double *q, double *part,
                                                          unsigned int *arrived, double *out)
{
    __shared__ double sh[kInvWarps][12];
    __shared__ double2 s_xy[kInvWarps][32], s_zq[kInvWarps][32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double2 *xy = s_xy[wid], *zq = s_zq[wid];
    double pairs = 0.0;
    for (long long t = (long long)blockIdx.x * kInvWarps + wid; t < units; t += (long long)gridDim.x * kInvWarps) {
        int g, bj;
        inv_unit_coords(t, g, bj);
        const int jo = bj * 32 + lane, ncols = n - bj * 32;
        const bool jv = jo < n;
        double xi[2], yi[2], zi[2], qi[2];
        bool iv[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = (2 * g + h) * 32 + lane;
            iv[h] = 2 * g + h <= bj && i < n;
            xi[h] = iv[h] ? x[i] : 0.0;
            yi[h] = iv[h] ? y[i] : 0.0;
            zi[h] = iv[h] ? z[i] : 0.0;
            qi[h] = iv[h] ? (q ? q[i] : 1.0) : 0.0;
        }
        __syncwarp();
        xy[lane] = make_double2(jv ? x[jo] : 0.0, jv ? y[jo] : 0.0);
        zq[lane] = make_double2(jv ? z[jo] : 0.0, jv ? (q ? q[jo] : 1.0) : 0.0);
        __syncwarp();
        double a[2] = {0.0, 0.0};
        if (2 * g + 1 < bj && ncols >= 32) {  // two blocks off the diagonal, every pair there
#pragma unroll 4
            for (int k = 0; k < 32; k++) {
                const int src = (lane + k) & 31;
                const double2 cxy = xy[src], czq = zq[src];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const double dx = xi[h] - cxy.x, dy = yi[h] - cxy.y, dz = zi[h] - czq.x;
                    a[h] = fma(czq.y, rsqrt_normal(fma(dz, dz, fma(dy, dy, dx * dx))), a[h]);
                }
            }
        } else {
            for (int h = 0; h < 2; h++) {
                const bool diag = 2 * g + h == bj;
                for (int k = diag ? 1 : 0; k <= (diag ? 16 : 31); k++) {
                    const int src = (lane + k) & 31;
                    const double2 cxy = xy[src], czq = zq[src];
                    const double dx = xi[h] - cxy.x, dy = yi[h] - cxy.y, dz = zi[h] - czq.x;
                    const double r = rsqrt_normal(fma(dz, dz, fma(dy, dy, dx * dx)));
                    if ((!diag || k < 16 || lane < 16) && iv[h] && src < ncols) a[h] = fma(czq.y, r, a[h]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            double acc = qi[h] * a[h];
            if (!isfinite(acc))
                acc = inv_block_again(xy, zq, xi[h], yi[h], zi[h], qi[h], lane, 2 * g + h == bj, iv[h], ncols);
            pairs += acc;
        }
    }
    double s[12];
#pragma unroll
    for (int k = 0; k < 12; k++) s[k] = 0.0;
    s[11] = pairs;
    for (int p = blockIdx.x * kInvThreads + threadIdx.x; p < n; p += gridDim.x * kInvThreads) {
        const double X = x[p], Y = y[p], Z = z[p], U = u[p], V = v[p], W = w[p];
        s[0] += U * U + V * V + W * W;
        s[2] += Y * W - Z * V;
        s[3] += Z * U - X * W;
        s[4] += X * V - Y * U;
        s[5] += U; s[6] += V; s[7] += W;
        s[8] += X; s[9] += Y; s[10] += Z;
    }
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const double t = warp_sum(s[k]);
        if (lane == 0) sh[wid][k] = t;
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        double t = 0.0;
        for (int k = 0; k < kInvWarps; k++) t += sh[k][threadIdx.x];
        part[(size_t)blockIdx.x * 12 + threadIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int k = wid; k < 12; k += kInvWarps) {
        double t = 0.0;
        for (unsigned int b = lane; b < gridDim.x; b += 32) t += __ldcg(part + (size_t)b * 12 + k);
        t = warp_sum(t);
        if (lane == 0) out[k] = t;
    }
}

// Grid: enough CTAs for the pair units, at most what is resident (4 per SM).
static int inv_grid(int n)
{
    const long long blocks = (inv_units_before((n + 31) / 32) + kInvWarps - 1) / kInvWarps;
    const int sms = device_sm_count();
    const long long cap = sms > 0 ? 4LL * sms : 592;
    return (int)(blocks < cap ? blocks : cap);
}

// Enqueue the invariants of device SoA state into out_dev[12] (11 values, slot 1 = 0, slot 11 = raw
// pair sum before the eps_th factor).  scratch must hold inv_scratch_doubles(n).
size_t inv_scratch_doubles(int n) { return (size_t)inv_grid(n) * 12 + 1; }

cudaError_t enqueue_invariance(cudaStream_t st, int n, const double *x, const double *y, const double *z,
                               const double *u, const double *v, const double *w, const double *q,
                               double *scratch, double *out_dev)
{
    const int grid = inv_grid(n);
    unsigned int *arrived = (unsigned int *)(scratch + (size_t)grid * 12);
    cudaError_t e = cudaMemsetAsync(arrived, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    inv_kernel<<<grid, kInvThreads, 0, st>>>(n, inv_units_before((n + 31) / 32), x, y, z, u, v, w, q, scratch, arrived, out_dev);
    return cudaGetLastError();
}

struct InvDropInState {
    int ready = 0;
    DeviceBuffer state, scratch;
    double *h_out = nullptr;
};
static thread_local InvDropInState g_inv;

}  // namespace bia

using namespace bia;

extern "C" int bia_invariance(bia_context *ctx, int n, double eps_th, const double *x, const double *y,
                              const double *z, const double *u, const double *v, const double *w,
                              const double *q, double out[11])
{
    if (!ctx || n < 1 || !x || !y || !z || !u || !v || !w || !out) return BIA_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    const size_t need = inv_scratch_doubles(n) + 12;
    cudaError_t e = ctx->inv.reserve(need * sizeof(double));
    if (e != cudaSuccess) return cuda_status(e);
    double *scratch = (double *)ctx->inv.ptr;
    double *res = scratch + inv_scratch_doubles(n);
    e = enqueue_invariance(ctx->stream, n, x, y, z, u, v, w, q, scratch, res);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ctx->h_inv, res, 12 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_status(e);
    for (int k = 0; k < 11; k++) out[k] = ctx->h_inv[k];
    out[1] = eps_th * ctx->h_inv[11];
    return BIA_OK;
}

extern "C" void invariance_gpu_(const int N, const double eps_th, double *X, double *Y, double *Z, double *U,
                                double *V, double *W, double *KE, double *PE, double *Lx, double *Ly,
                                double *Lz, double *Ua, double *Va, double *Wa, double *Xa, double *Ya,
                                double *Za)
{
    if (N < 1 || !X || !Y || !Z || !U || !V || !W || !KE || !PE || !Lx || !Ly || !Lz || !Ua || !Va || !Wa ||
        !Xa || !Ya || !Za) {
        set_last_error(BIA_ERR_INVALID_ARGUMENT);
        return;
    }
    InvDropInState &S = g_inv;
    cudaError_t e = cudaSuccess;
    if (!S.ready) {
        e = cudaMallocHost((void **)&S.h_out, 12 * sizeof(double));
        if (e != cudaSuccess) {
            set_last_error(cuda_status(e));
            return;
        }
        S.ready = 1;
    }
    const size_t need = inv_scratch_doubles(N) + 12;
    if ((e = S.state.reserve((size_t)6 * N * sizeof(double))) != cudaSuccess ||
        (e = S.scratch.reserve(need * sizeof(double))) != cudaSuccess) {
        set_last_error(cuda_status(e));
        return;
    }
    double *d = (double *)S.state.ptr;
    double *host[6] = {X, Y, Z, U, V, W};
    for (int k = 0; k < 6 && e == cudaSuccess; k++)
        e = cudaMemcpy(d + (size_t)k * N, host[k], N * sizeof(double), cudaMemcpyHostToDevice);
    double *scratch = (double *)S.scratch.ptr;
    double *res = scratch + inv_scratch_doubles(N);
    if (e == cudaSuccess)
        e = enqueue_invariance(0, N, d, d + N, d + 2 * (size_t)N, d + 3 * (size_t)N, d + 4 * (size_t)N,
                               d + 5 * (size_t)N, nullptr, scratch, res);
    if (e == cudaSuccess) e = cudaMemcpy(S.h_out, res, 12 * sizeof(double), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        set_last_error(cuda_status(e));
        return;
    }
    const double *o = S.h_out;
    *KE = o[0];
    *PE = eps_th * o[11];
    *Lx = o[2]; *Ly = o[3]; *Lz = o[4];
    *Ua = o[5]; *Va = o[6]; *Wa = o[7];
    *Xa = o[8]; *Ya = o[9]; *Za = o[10];
    set_last_error(BIA_OK);
}
