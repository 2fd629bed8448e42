// A linear solve for callers that cannot allocate device memory.
//
// tf_solve_bsr_static solves A x = b for a caller-owned 3x3 block-sparse
// matrix with block-Jacobi preconditioned BiCGStab in FP64, like the solve
// behind tf_solve, but it calls no cudaMalloc, cudaFree or other allocating
// routine.  Its work vectors, reduction partials and scalars live in one
// file-scope device array, g_static_scratch, sized for at most
// kStaticMaxNodes block rows.  Every GPU that loads this library holds that
// array (about 4.6 MB) until the process exits.
//
// Host code cannot use the array's name as a device address, so the first
// call on each device looks the address up with cudaGetSymbolAddress while
// that device is current, and caches it together with the CUDA context it
// came from; a call in another context (after cudaDeviceReset, say) looks it
// up again.  Every call synchronises its stream and reads scalars back to the
// host, so no call may be made on a stream that is being captured: such a call
// returns TF_BAD_INPUT and leaves the capture untouched.  All calls on a device
// share the one array: calls that overlap on the GPU (two streams, two host
// threads) race on it and give wrong results or an error, so serialise them.
// Each call sets the count of the CTAs' meetings before its kernel, and writes
// the scalars and every work vector before reading it, so nothing carries
// over from the previous call.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "tf_count.h"
#include "tf_internal.cuh"

namespace tf {
namespace {

constexpr int kStaticMaxNodes = 16384;
constexpr int kStaticThreads = 512;
constexpr int kStaticWarps = kStaticThreads / 32;
constexpr int kStaticMaxGrid = kStaticMaxNodes / 32;
constexpr size_t kVecLen = 4 * (size_t)kStaticMaxNodes;  // a row's three entries in one 32-byte load
// phat and shat, which all CTAs read; then 27 doubles per row that only the
// row's CTA uses (its vectors and inverse diagonal block), where they do not
// fit its shared memory
constexpr size_t kOffLocal = 2 * kVecLen;
constexpr int kLocal = 27;
constexpr size_t kOffPart = kOffLocal + kLocal * (size_t)kStaticMaxNodes;
constexpr int kMaxSums = 2;
constexpr int kNumSums = 4;                   // reductions of an iteration and the start
constexpr size_t kOffScal = kOffPart + kNumSums * kMaxSums * (size_t)kStaticMaxGrid;
constexpr size_t kNumScal = 16;
constexpr size_t kOffBar = kOffScal + kNumScal;
constexpr size_t kScratchDoubles = kOffBar + 2;
constexpr int kStaticSmem = 200 * 1024;
constexpr int kStaticPolls = 1 << 22;         // a wait for the other CTAs gives up after some seconds
// The count of the CTAs' arrivals wraps after 5.65 M iterations on 152 SMs.  It
// starts one below the wrap (a memset's pattern), so every solve crosses it.
constexpr unsigned kCountStart = 0xffffffffu;

__device__ __align__(256) double g_static_scratch[kScratchDoubles];

enum { Q_BB = 0, Q_RR, Q_ITER, Q_FLAG };
enum { QF_RUNNING = 0, QF_CONVERGED = 1, QF_BREAKDOWN = 2, QF_NAN = 3, QF_STUCK = 4 };

struct SCtx {
    int n;
    int rows;  // per CTA
    int meet;  // CTAs at a meeting
    int max_iter;
    double tol2;
    const int* __restrict__ rowptr;
    const int* __restrict__ colidx;
    const double* __restrict__ val;
    double* base;  // device address of g_static_scratch
    __device__ double* phat() const { return base; }
    __device__ double* shat() const { return base + kVecLen; }
    __device__ double* part(int k) const { return base + kOffPart + k * kMaxSums * (size_t)kStaticMaxGrid; }
    __device__ double* q() const { return base + kOffScal; }
    __device__ unsigned* bar() const { return reinterpret_cast<unsigned*>(base + kOffBar); }
};

struct SShared {
    double sums[kMaxSums][kStaticWarps];
    double rho, rr, bb, alpha, omega, beta;  // the recurrence's scalars
    int it, flag;
    double y[kStaticWarps][3][32];
    int stuck;
};

// All CTAs meet (they are resident together: a cooperative launch).  False when
// the wait ran out.
__device__ __forceinline__ bool s_barrier(const SCtx& c, SShared& sh, unsigned& goal) {
    goal += c.meet;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned* bar = c.bar();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned seen;
        int polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
        } while (!count_reached(seen, goal) && ++polls < kStaticPolls);
        if (!count_reached(seen, goal)) sh.stuck = 1;
    }
    __syncthreads();
    return !sh.stuck;
}

// Sums over all CTAs in a fixed order; thread 0 of every CTA then takes them to
// the next scalars (`then`), which all threads find in sh.  One thread: a
// division by all 512 keeps the FP64 pipe busy for 3 us.  `slot`: where this warp's
// values enter (-1: it has none), `slots`: how many warps have some.  It is a
// meeting of the CTAs as well.  Reduction k of an iteration has its own partials:
// they are rewritten an iteration later.
template <int NV, class F>
__device__ __forceinline__ bool s_reduce(const SCtx& c, SShared& sh, unsigned& goal, int k, int slot, int slots,
                                         double (&v)[NV], F then) {
    const int lane = threadIdx.x & 31;
    if (slot >= 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < NV; ++u) v[u] += __shfl_down_sync(0xffffffffu, v[u], o);
        if (lane == 0)
#pragma unroll
            for (int u = 0; u < NV; ++u) sh.sums[u][slot] = v[u];
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            double s = sh.sums[u][0];
            for (int w = 1; w < slots; ++w) s += sh.sums[u][w];
            c.part(k)[u * kStaticMaxGrid + blockIdx.x] = s;
        }
    if (!s_barrier(c, sh, goal)) return false;
    if (threadIdx.x < 32) {
        double s[NV];
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            s[u] = 0.0;
#pragma unroll 8
            for (int b = lane; b < (int)gridDim.x; b += 32) s[u] += __ldcg(&c.part(k)[u * kStaticMaxGrid + b]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < NV; ++u) s[u] += __shfl_down_sync(0xffffffffu, s[u], o);
        if (lane == 0) then(s);
    }
    __syncthreads();
    return true;
}

// The rows of a CTA: its blocks, in shared memory as far as they fit; a group of
// warps for 32 rows, each warp a share of every row's blocks.
struct SRows {
    int nr, groups, share;  // rows, groups of 32, warps per group
    int row0;
    const int* ptr;         // positions of the rows' blocks from the CTA's first (shared)
    const int* col;
    const double* val;
    const double* staged;   // the first nstaged blocks, in shared memory
    int nstaged;
};

// The entries of a row of phat or shat, written by any CTA before the last meeting
__device__ __forceinline__ void load_row(const double* x, double (&v)[3]) {
    double pad;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(pad) : "l"(x) : "memory");
}

// y = A x for the rows of a group, summed over its warps, on the group's first
// warp (returns true there; lane = row of the group).  Every thread calls it.
__device__ __forceinline__ bool s_rows(const SRows& R, SShared& sh, int g, const double* x, double (&y)[3]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = warp % R.share;
    const int i = 32 * g + lane;
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
    if (g < R.groups && i < R.nr) {
        const int p1 = R.ptr[i + 1];
        for (int pb = R.ptr[i] + w; pb < p1; pb += 4 * R.share) {  // four blocks' columns, then their x, then the sums
            const double* xj[4];
            double v[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u) xj[u] = pb + u * R.share < p1 ? x + 4 * (size_t)R.col[pb + u * R.share] : nullptr;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (xj[u]) load_row(xj[u], v[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!xj[u]) continue;
                const int p = pb + u * R.share;
                const double* a = (p < R.nstaged ? R.staged : R.val) + 9 * (size_t)p;
                y0 = fma(a[0], v[u][0], fma(a[1], v[u][1], fma(a[2], v[u][2], y0)));
                y1 = fma(a[3], v[u][0], fma(a[4], v[u][1], fma(a[5], v[u][2], y1)));
                y2 = fma(a[6], v[u][0], fma(a[7], v[u][1], fma(a[8], v[u][2], y2)));
            }
        }
    }
    sh.y[warp][0][lane] = y0;
    sh.y[warp][1][lane] = y1;
    sh.y[warp][2][lane] = y2;
    __syncthreads();
    // pairs of warps, then pairs of pairs: a chain of additions waits for each
    for (int k = 1; k < R.share; k *= 2) {
        if (g < R.groups && w % (2 * k) == 0 && w + k < R.share)
#pragma unroll
            for (int d = 0; d < 3; ++d) sh.y[warp][d][lane] += sh.y[warp + k][d][lane];
        __syncthreads();
    }
    if (w != 0 || g >= R.groups) return false;
#pragma unroll
    for (int d = 0; d < 3; ++d) y[d] = sh.y[warp][d][lane];
    return i < R.nr;
}

__device__ __forceinline__ void s_prec(const double* D, const double r[3], double z[3]) {
    z[0] = fma(D[0], r[0], fma(D[1], r[1], D[2] * r[2]));
    z[1] = fma(D[3], r[0], fma(D[4], r[1], D[5] * r[2]));
    z[2] = fma(D[6], r[0], fma(D[7], r[1], D[8] * r[2]));
}

// Inverse of a block row's diagonal block (identity where it has none or it is singular)
__device__ __forceinline__ void s_diag_inverse(const SCtx& c, int i, double* inv) {
    const double* M = nullptr;
    for (int p = c.rowptr[i]; p < c.rowptr[i + 1]; ++p)
        if (c.colidx[p] == i) M = c.val + 9 * (size_t)p;
    for (int k = 0; k < 9; ++k) inv[k] = k % 4 == 0 ? 1.0 : 0.0;
    if (!M) return;
    const double c0 = M[4] * M[8] - M[5] * M[7], c1 = M[5] * M[6] - M[3] * M[8], c2 = M[3] * M[7] - M[4] * M[6];
    const double det = M[0] * c0 + M[1] * c1 + M[2] * c2;
    if (det == 0.0) return;
    const double r = 1.0 / det;
    inv[0] = c0 * r;
    inv[1] = (M[2] * M[7] - M[1] * M[8]) * r;
    inv[2] = (M[1] * M[5] - M[2] * M[4]) * r;
    inv[3] = c1 * r;
    inv[4] = (M[0] * M[8] - M[2] * M[6]) * r;
    inv[5] = (M[2] * M[3] - M[0] * M[5]) * r;
    inv[6] = c2 * r;
    inv[7] = (M[1] * M[6] - M[0] * M[7]) * r;
    inv[8] = (M[0] * M[4] - M[1] * M[3]) * r;
}

// The whole solve: block-Jacobi BiCGStab over all CTAs, each with the rows
// blockIdx.x * rows ...  Bound by the meetings of the CTAs (five an iteration, 1.4
// us each, three of them with a sum) and the FP64 pipe (two products of 27 blocks
// a row: 4 us each at 56 rows per SM, half the lanes of the last group idle).  As
// five launches an iteration with a thread per row, 33 of them on 8,405 rows,
// the products waited for memory: 70 us an iteration against 30 now (19.1 -> 8.3
// ms to 1e-12; 105 rows 5.0 -> 1.5, 1,200 12.9 -> 4.4, 16,200 19.5 -> 9.8).  The
// matrix stays in shared memory between the iterations: nothing is allocated.
__global__ void __launch_bounds__(kStaticThreads, 1) ks_solve(SCtx c, const double* b, double* x) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SShared sh;
    const int t = threadIdx.x, warp = t >> 5;
    SRows R;
    R.row0 = blockIdx.x * c.rows;
    R.nr = min(c.rows, c.n - R.row0);
    const int all = (c.rows + 31) / 32;           // groups of 32 rows
    R.share = max(1, kStaticWarps / all);         // warps on a group
    R.groups = (R.nr + 31) / 32;
    const int passes = (all * R.share + kStaticWarps - 1) / kStaticWarps;  // groups a warp serves in turn
    const int p0 = c.rowptr[R.row0], nb = c.rowptr[R.row0 + R.nr] - p0;
    if (t == 0) sh.stuck = 0;
    // shared memory: row positions, then the CTA's vectors, blocks and columns as far as they fit
    int* ptr = reinterpret_cast<int*>(smem);
    size_t used = ((R.nr + 1) * sizeof(int) + 15) / 16 * 16;
    for (int k = t; k <= R.nr; k += kStaticThreads) ptr[k] = c.rowptr[R.row0 + k] - p0;
    R.ptr = ptr;
    double* loc = c.base + kOffLocal + (size_t)kLocal * R.row0;
    if (used + sizeof(double) * kLocal * R.nr <= kStaticSmem) {
        loc = reinterpret_cast<double*>(smem + used);
        used += (sizeof(double) * kLocal * R.nr + 15) / 16 * 16;
    }
    R.col = c.colidx + p0;
    R.val = c.val + 9 * (size_t)p0;
    if (used + sizeof(int) * nb <= kStaticSmem / 4) {
        int* col = reinterpret_cast<int*>(smem + used);
        for (int k = t; k < nb; k += kStaticThreads) col[k] = R.col[k];
        R.col = col;
        used += (sizeof(int) * nb + 15) / 16 * 16;
    }
    double* staged = reinterpret_cast<double*>(smem + used);
    R.staged = staged;
    R.nstaged = min(nb, (int)((kStaticSmem - used) / (9 * sizeof(double))));
#pragma unroll 8
    for (int k = t; k < 9 * R.nstaged; k += kStaticThreads) staged[k] = R.val[k];
    const int n3 = 3 * R.nr;
    double *r = loc, *rhat = r + n3, *p = rhat + n3, *v = p + n3, *s = v + n3, *tv = s + n3, *dinv = tv + n3;
    double *phat = c.phat() + 4 * R.row0, *shat = c.shat() + 4 * R.row0;
    x += 3 * (size_t)R.row0;
    b += 3 * (size_t)R.row0;
    // a thread per row, but for the products
    const int slots_row = min(kStaticWarps, R.groups), slot_row = warp < slots_row ? warp : -1;
    const int par = kStaticWarps / R.share, slots_mul = min(par, R.groups);
    const int slot_mul = warp % R.share == 0 && warp / R.share < slots_mul ? warp / R.share : -1;
    double bb[1] = {0.0};
    for (int i = t; i < R.nr; i += kStaticThreads) {
        s_diag_inverse(c, R.row0 + i, dinv + 9 * (size_t)i);
        for (int d = 3 * i; d < 3 * i + 3; ++d) {
            const double bk = b[d];
            r[d] = rhat[d] = bk;
            p[d] = v[d] = 0.0;
            x[d] = 0.0;
            bb[0] = fma(bk, bk, bb[0]);
        }
    }
    unsigned goal = kCountStart;
    bool ok = s_reduce<1>(c, sh, goal, 0, slot_row, slots_row, bb, [&](const double* q) {
        sh.rho = sh.rr = sh.bb = q[0];
        sh.alpha = sh.omega = 1.0;
        sh.beta = 0.0;
        sh.it = 0;
        sh.flag = q[0] == 0.0 ? QF_CONVERGED : (isfinite(q[0]) ? QF_RUNNING : QF_NAN);
    });
    while (ok && sh.flag == QF_RUNNING && sh.it < c.max_iter) {
        // p = r + beta (p - omega v); phat = M^-1 p
        const double beta = sh.beta, omega0 = sh.omega;
        for (int i = t; i < R.nr; i += kStaticThreads) {
            double pp[3], z[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int k = 3 * i + d;
                pp[d] = fma(beta, fma(-omega0, v[k], p[k]), r[k]);
                p[k] = pp[d];
            }
            s_prec(dinv + 9 * (size_t)i, pp, z);
#pragma unroll
            for (int d = 0; d < 3; ++d) phat[4 * i + d] = z[d];
        }
        if (!(ok = s_barrier(c, sh, goal))) break;
        // v = A phat; alpha = rho / (rhat, v)
        double rv[1] = {0.0}, y[3];
        for (int k = 0; k < passes; ++k) {
            const int g = warp / R.share + k * par;
            if (s_rows(R, sh, g, c.phat(), y))
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int e = 3 * (32 * g + (t & 31)) + d;
                    v[e] = y[d];
                    rv[0] = fma(rhat[e], y[d], rv[0]);
                }
            if (k + 1 < passes) __syncthreads();
        }
        ok = s_reduce<1>(c, sh, goal, 1, slot_mul, slots_mul, rv, [&](const double* q) {
            if (q[0] == 0.0 || !isfinite(q[0])) sh.flag = isfinite(q[0]) ? QF_BREAKDOWN : QF_NAN;
            else sh.alpha = sh.rho / q[0];
        });
        if (!ok || sh.flag != QF_RUNNING) break;
        // s = r - alpha v; shat = M^-1 s
        const double alpha = sh.alpha;
        for (int i = t; i < R.nr; i += kStaticThreads) {
            double ss[3], z[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int k = 3 * i + d;
                ss[d] = fma(-alpha, v[k], r[k]);
                s[k] = ss[d];
            }
            s_prec(dinv + 9 * (size_t)i, ss, z);
#pragma unroll
            for (int d = 0; d < 3; ++d) shat[4 * i + d] = z[d];
        }
        if (!(ok = s_barrier(c, sh, goal))) break;
        // t = A shat; omega = (t, s) / (t, t)
        double ts[2] = {0.0, 0.0};
        for (int k = 0; k < passes; ++k) {
            const int g = warp / R.share + k * par;
            if (s_rows(R, sh, g, c.shat(), y))
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int e = 3 * (32 * g + (t & 31)) + d;
                    tv[e] = y[d];
                    ts[0] = fma(y[d], s[e], ts[0]);
                    ts[1] = fma(y[d], y[d], ts[1]);
                }
            if (k + 1 < passes) __syncthreads();
        }
        ok = s_reduce<2>(c, sh, goal, 2, slot_mul, slots_mul, ts, [&](const double* q) {
            if (!isfinite(q[0]) || !isfinite(q[1])) sh.flag = QF_NAN;
            else sh.omega = q[1] > 0.0 ? q[0] / q[1] : 0.0;
        });
        if (!ok || sh.flag != QF_RUNNING) break;
        // x += alpha phat + omega shat; r = s - omega t; rho' = (rhat, r)
        const double omega = sh.omega;
        double ro[2] = {0.0, 0.0};
        if (t == kStaticThreads - 1) sh.beta = alpha / omega;  // beside the others' work
        for (int i = t; i < R.nr; i += kStaticThreads)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int k = 3 * i + d;
                x[k] = fma(omega, shat[4 * i + d], fma(alpha, phat[4 * i + d], x[k]));
                const double rk = fma(-omega, tv[k], s[k]);
                r[k] = rk;
                ro[0] = fma(rhat[k], rk, ro[0]);
                ro[1] = fma(rk, rk, ro[1]);
            }
        ok = s_reduce<2>(c, sh, goal, 3, slot_row, slots_row, ro, [&](const double* q) {
            sh.beta *= q[0] / sh.rho;
            sh.rho = q[0];
            sh.rr = q[1];
            ++sh.it;
            if (!isfinite(q[1])) sh.flag = QF_NAN;
            else if (q[1] <= c.tol2 * sh.bb) sh.flag = QF_CONVERGED;
            else if (sh.omega == 0.0 || q[0] == 0.0) sh.flag = QF_BREAKDOWN;
        });
    }
    if (t == 0 && !ok) c.q()[Q_FLAG] = QF_STUCK;
    if (t != 0 || blockIdx.x != 0 || !ok) return;
    double* q = c.q();
    q[Q_BB] = sh.bb;
    q[Q_RR] = sh.rr;
    q[Q_ITER] = sh.it;
    q[Q_FLAG] = sh.flag;
}

std::mutex g_addr_mutex;
struct ScratchAddr {
    CUcontext ctx;
    double* ptr;
};
ScratchAddr g_addr[64] = {};
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
CtxGetCurrentFn g_ctx_get = nullptr;

// The current CUDA context, through the driver entry point the runtime hands
// out (the library does not link the driver library itself).
tf_status current_context(CUcontext* ctx) {
    if (!g_ctx_get) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetDriverEntryPointByVersion(cuCtxGetCurrent)");
        if (q != cudaDriverEntryPointSuccess || !fn) {
            set_error("tf_solve_bsr_static: the driver offers no cuCtxGetCurrent");
            return TF_CUDA_ERROR;
        }
        g_ctx_get = reinterpret_cast<CtxGetCurrentFn>(fn);
    }
    *ctx = nullptr;
    if (g_ctx_get(ctx) != CUDA_SUCCESS || !*ctx) {
        set_error("tf_solve_bsr_static: no current CUDA context");
        return TF_CUDA_ERROR;
    }
    return TF_OK;
}

// Device address of g_static_scratch for `device`, looked up once per device
// and context with that device current.
tf_status scratch_address(int device, double** out) {
    if (device < 0 || device >= 64) {
        set_error("device ordinal out of range for the static solve");
        return TF_BAD_INPUT;
    }
    std::lock_guard<std::mutex> lock(g_addr_mutex);
    CUcontext ctx = nullptr;
    tf_status s = current_context(&ctx);
    if (s != TF_OK) return s;
    if (!g_addr[device].ptr || g_addr[device].ctx != ctx) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_static_scratch)");
        g_addr[device].ptr = static_cast<double*>(p);
        g_addr[device].ctx = ctx;
    }
    *out = g_addr[device].ptr;
    return TF_OK;
}

}  // namespace
}  // namespace tf

using namespace tf;

// With up to max_blocks thread blocks, which wait for `absent` more at their meetings
// (tests; tf_solve_bsr_static asks for one per SM, max_blocks = 0, and none absent).
extern "C" TF_API tf_status tf_static_solve_blocks(int32_t max_blocks, int32_t absent, int32_t n_block_rows, const int32_t* rowptr,
                                                   const int32_t* colidx, const double* val, const double* b,
                                                   double* x, double rtol, int32_t max_iter, void* stream,
                                                   int32_t* iters, double* relres) {
    if (n_block_rows <= 0 || !rowptr || !colidx || !val || !b || !x || !(rtol > 0.0) || max_iter <= 0 ||
        max_blocks < 0 || absent < 0) {
        set_error("tf_solve_bsr_static: bad arguments");
        return TF_BAD_INPUT;
    }
    if (n_block_rows > kStaticMaxNodes) {
        set_error("tf_solve_bsr_static: " + std::to_string(n_block_rows) + " block rows exceed the static limit of " +
                  std::to_string(kStaticMaxNodes));
        return TF_BAD_INPUT;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    TF_CUDA(cudaStreamIsCapturing(st, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
        set_error("tf_solve_bsr_static: the stream is being captured; this call synchronises and reads back, "
                  "so it cannot run inside a capture");
        return TF_BAD_INPUT;
    }
    int device = 0;
    TF_CUDA(cudaGetDevice(&device));
    double* base = nullptr;
    tf_status s = scratch_address(device, &base);
    if (s != TF_OK) return s;
    int sms = max_blocks;
    if (max_blocks == 0) TF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    SCtx c{n_block_rows, 0, 0, max_iter, rtol * rtol, rowptr, colidx, val, base};
    // the count to kCountStart; the scalars are the kernel's to write
    TF_CUDA(cudaMemsetAsync(base + kOffScal, 0xff, sizeof(double) * (kNumScal + 2), st));
    TF_CUDA(cudaFuncSetAttribute(ks_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kStaticSmem));
    // One block per SM.  Where not all of them can be resident together (a stream
    // that owns a part of the SMs only), half as many until they can: one always fits.
    int blocks = std::min(sms, cdiv(n_block_rows, 32));
    while (true) {
        c.rows = cdiv(n_block_rows, blocks);
        blocks = cdiv(n_block_rows, c.rows);
        c.meet = blocks + absent;
        const cudaError_t e =
            launch_cooperative(ks_solve, blocks, kStaticThreads, kStaticSmem, st, c, b, x);
        if (e == cudaSuccess) break;
        (void)cudaGetLastError();
        if (e != cudaErrorCooperativeLaunchTooLarge || blocks == 1) return cuda_fail(e, "tf_solve_bsr_static");
        blocks /= 2;
    }
    double q[kNumScal];
    TF_CUDA(cudaMemcpyAsync(q, base + kOffScal, sizeof(q), cudaMemcpyDeviceToHost, st));
    TF_CUDA(cudaStreamSynchronize(st));
    const bool stuck = !(q[Q_FLAG] < QF_STUCK);  // or not written: an overlapping call's memset
    if (iters) *iters = stuck ? 0 : static_cast<int32_t>(q[Q_ITER]);
    if (relres) *relres = !stuck && q[Q_BB] > 0.0 ? sqrt(q[Q_RR] / q[Q_BB]) : 0.0;
    if (q[Q_FLAG] == QF_CONVERGED) return TF_OK;
    if (stuck) {
        set_error("tf_solve_bsr_static: the thread blocks lost each other (overlapping calls?)");
        return TF_CUDA_ERROR;
    }
    if (q[Q_FLAG] == QF_NAN) {
        set_error("tf_solve_bsr_static: non-finite value");
        return TF_NAN_DETECTED;
    }
    if (q[Q_FLAG] == QF_BREAKDOWN) {
        set_error("tf_solve_bsr_static: BiCGStab breakdown");
        return TF_KRYLOV_BREAKDOWN;
    }
    set_error("tf_solve_bsr_static: iteration cap reached");
    return TF_KRYLOV_NOT_CONVERGED;
}

extern "C" TF_API tf_status tf_solve_bsr_static(int32_t n_block_rows, const int32_t* rowptr, const int32_t* colidx,
                                                const double* val, const double* b, double* x, double rtol,
                                                int32_t max_iter, void* stream, int32_t* iters, double* relres) {
    return tf_static_solve_blocks(0, 0, n_block_rows, rowptr, colidx, val, b, x, rtol, max_iter, stream, iters,
                                  relres);
}
