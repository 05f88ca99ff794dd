// bia_row.cu -- drop-in replacement of the reference's per-particle entry
// find_dxyuv_kernel_ (bia/find_dXYUV_kernel.cu:526-561), called once per particle i
// by bia/bia.f90:135,138.
//
// Semantics kept: for the fixed 1-based particle I and every j > I the pair given by
// the host AoS array RXYZUVW (x_i-x_j, ..., w_i-w_j) is solved, dXYZUVW[6j+k] receives
// the half-displacement and the host arrays dX..dW are accumulated in place
// (dX[i] += h_j, dX[j] -= h_j).  Entries j <= i of dXYZUVW are zero.
//
// What bounds a call is latency: it moves 96 bytes a pair, and at N = 1332 the pairs of one
// row are 42 warps.  So the rows j > i alone go through one pinned buffer that the kernel
// reads and writes over PCIe itself, and a call is one launch and one wait.  With three
// blocking copies back, one to the device and a memset it took 102 us at N = 1332 (mean
// over all I, from Python), now 45.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <mutex>

#include "bia_internal.cuh"
#include "bia_pair.cuh"

namespace bia {

constexpr int kRowPart = 8;  // doubles a warp leaves for the host: six sums, its non-finite pairs, 0

struct RowArgs {
    const double *rel;  // AoS [6m], pinned host memory: the m rows j > i
    double *out;        // AoS [6m], pinned host memory
    double *part;       // [warps][kRowPart], pinned host memory: sum over the warp's j of h_j
    int m;
    double eps_th;
    PairParams P;
};

// One warp a block: the pairs of a row are too few to fill the SMs, and a warp that has an SM's
// FP64 pipes and PCIe requests to itself is back first.  The AoS rows pass through shared memory
// so that each 256 bytes of host memory are one request.
template <int M>
__global__ void __launch_bounds__(32) bia_row_kernel(const RowArgs A)
{
    __shared__ double sh[6 * 32];
    const int lane = threadIdx.x;
    const int base = blockIdx.x * 32;
    const int words = 6 * min(32, A.m - base);
    const double *src = A.rel + (size_t)6 * base;
    double *dst = A.out + (size_t)6 * base;
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (lane + 32 * k < words) sh[lane + 32 * k] = src[lane + 32 * k];
    __syncwarp();
    PairCounters cnt;
    counters_zero(cnt);
    double h[6] = {0, 0, 0, 0, 0, 0};
    double *s = sh + 6 * lane;
    if (base + lane < A.m) {
        const double r[3] = {s[0], s[1], s[2]};
        const double g[3] = {s[3], s[4], s[5]};
        pair_halfdisp<M>(A.P, A.eps_th, r, g, h, cnt);
#pragma unroll
        for (int c = 0; c < 6; c++) s[c] = h[c];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (lane + 32 * k < words) dst[lane + 32 * k] = sh[lane + 32 * k];
    const unsigned full = 0xffffffffu;
    double *part = A.part + (size_t)kRowPart * blockIdx.x;
#pragma unroll
    for (int c = 0; c < 6; c++) {
        double v = h[c];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(full, v, off);
        if (lane == 0) part[c] = v;
    }
    const int nonfinite = __reduce_add_sync(full, cnt.nonfinite);
    if (lane == 0) part[6] = nonfinite;
}

// A host thread's pinned buffer, grown on demand.  A thread that ends leaves it to the next one that
// starts: at most as many are held as threads have used the entry at the same time.  They die with
// the process; freeing them here could run after the CUDA runtime has shut down.  What is known of a
// buffer lies beside it, so that a buffer that died early (a device reset) is never read here.
struct RowBuffer {
    RowBuffer *next;
    double *ptr;
    size_t bytes;
};
static std::mutex g_idle_lock;
static RowBuffer *g_idle = nullptr;

struct RowState {
    RowBuffer *buf = nullptr;
    ~RowState()
    {
        if (!buf) return;
        std::lock_guard<std::mutex> g(g_idle_lock);
        buf->next = g_idle;
        g_idle = buf;
    }
    cudaError_t reserve(size_t want)
    {
        if (!buf) {
            std::lock_guard<std::mutex> g(g_idle_lock);
            if (g_idle) {
                buf = g_idle;
                g_idle = buf->next;
            }
        }
        if (!buf) buf = (RowBuffer *)calloc(1, sizeof(RowBuffer));
        if (!buf) return cudaErrorMemoryAllocation;
        if (want <= buf->bytes) return cudaSuccess;
        if (buf->ptr && cudaFreeHost(buf->ptr) != cudaSuccess) cudaGetLastError();  // clear
        buf->ptr = nullptr;
        buf->bytes = 0;
        cudaError_t e = cudaHostAlloc((void **)&buf->ptr, want, cudaHostAllocMapped | cudaHostAllocPortable);
        if (e == cudaSuccess) buf->bytes = want;
        return e;
    }
};
static thread_local RowState g_row;

}  // namespace bia

using namespace bia;

extern "C" void find_dxyuv_kernel_(const int METHOD, const int N, const int I, const double EPS,
                                   const double DT, const int ITR, double *dX, double *dY, double *dZ,
                                   double *dU, double *dV, double *dW, double *RXYZUVW,
                                   double *dXYZUVW)
{
    const int i = I - 1;
    if (N < 1 || i < 0 || i >= N || !RXYZUVW || !dXYZUVW || !dX || !dY || !dZ || !dU || !dV || !dW ||
        (METHOD != 0 && METHOD != 1) || ITR < 1 || ITR > 62) {
        set_last_error(BIA_ERR_INVALID_ARGUMENT);
        return;
    }
    RowState &S = g_row;
    const size_t below = (size_t)6 * (i + 1);    // doubles of the rows j <= i
    const size_t words = (size_t)6 * N - below;  // doubles of the rows j > i
    const int m = N - 1 - i, warps = (m + 31) / 32;
    // sized for the longest row of N particles; each part starts on a 256-byte boundary
    const size_t span = ((size_t)6 * N + 31) / 32 * 32;
    cudaError_t e = S.reserve((2 * span + (size_t)kRowPart * ((N + 31) / 32)) * sizeof(double));
    double *d_buf = nullptr;
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&d_buf, S.buf->ptr, 0);
    if (e != cudaSuccess) {
        set_last_error(cuda_status(e));
        return;
    }
    double *const rel = S.buf->ptr;
    const double *out = rel + span, *part = rel + 2 * span;
    if (m > 0) {
        memcpy(rel, RXYZUVW + below, words * sizeof(double));
        RowArgs A;
        A.rel = d_buf;
        A.out = d_buf + span;
        A.part = d_buf + 2 * span;
        A.m = m;
        A.eps_th = EPS;
        A.P.dt = DT;
        A.P.err = 1e-12;
        A.P.relerr = 0.0;
        A.P.abserr = 1e-16;
        A.P.itr = ITR;
        A.P.method = METHOD;
        if (METHOD == 0)
            bia_row_kernel<kMethodRkf><<<warps, 32>>>(A);
        else
            bia_row_kernel<kMethodAlg><<<warps, 32>>>(A);
        e = cudaGetLastError();
    }
    // on the null stream, so that a call waits for what the program's other streams have queued,
    // as blocking copies do
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    if (e != cudaSuccess) {
        set_last_error(cuda_status(e));
        return;
    }
    memset(dXYZUVW, 0, below * sizeof(double));
    memcpy(dXYZUVW + below, out, words * sizeof(double));
    double *acc[6] = {dX, dY, dZ, dU, dV, dW};
    double sum[6] = {0, 0, 0, 0, 0, 0};
    bool nonfinite = false;
    for (int w = 0; w < warps; w++, part += kRowPart) {
        for (int c = 0; c < 6; c++) sum[c] += part[c];
        nonfinite |= part[6] != 0.0;
    }
    for (int c = 0; c < 6; c++) acc[c][i] += sum[c];
    for (int j = i + 1; j < N; j++) {
        const double *h = dXYZUVW + (size_t)6 * j;
        for (int c = 0; c < 6; c++) acc[c][j] -= h[c];
    }
    set_last_error(nonfinite ? BIA_ERR_NONFINITE : BIA_OK);
}
