// What the node-parallel kernels of the linear solve share: their operands,
// the node of a thread, and the per-instance reductions (also fused into the
// multigrid's last kernel).
#pragma once

#include "tf_internal.cuh"

namespace tf {

constexpr int kThreads = kNodeThreads;

enum Flag { F_RUNNING = 0, F_CONVERGED = 1, F_BREAKDOWN = 2, F_NAN = 3 };
// Cause of a breakdown (S_WHY): which denominator vanished.
enum Why { W_NONE = 0, W_CG_PAP = 1, W_CG_RZ = 2, W_BI_RV = 3, W_BI_OMEGA = 4, W_BI_RHO = 5 };
static const char* const kWhy[] = {"", "(p, Ap) <= 0", "(r, M^-1 r) <= 0", "(rhat, A phat) = 0", "omega = 0",
                            "(rhat, r) = 0"};

struct Ctx {
    const int* __restrict__ wslot0;
    const int* __restrict__ scol;
    const double* __restrict__ val;
    const double* __restrict__ dinv;
    double* scal;               // [nseg][S_COUNT]
    double* part;               // [3][ncta]
    unsigned* tickets;          // [nseg]
    int ncta;
    const int* __restrict__ cta_seg;
    const int* __restrict__ cta_node0;
    const int* __restrict__ cta_node1;
    const int* __restrict__ seg_cta0;
    const int* __restrict__ seg_solve;
    const int* __restrict__ xrow;     // extra blocks (tf_add_K_triplets), null: none
    const int* __restrict__ xcol;
    const double* __restrict__ xval;
    int nn;
    int* check;                       // checked build: failed index checks
};

struct Where {
    int node;    // node of this thread
    bool valid;  // node inside this CTA's range
    int seg;     // instance of this CTA
    double* s;   // its scalars
};

__device__ __forceinline__ Where where(const Ctx& c) {
    Where w;
    w.seg = c.cta_seg[blockIdx.x];
    w.node = c.cta_node0[blockIdx.x] + threadIdx.x;
    w.valid = w.node < c.cta_node1[blockIdx.x];
    w.s = c.scal + (size_t)w.seg * S_COUNT;
    return w;
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sm)[kThreads / 32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) sm[k][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double x = lane < kThreads / 32 ? sm[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
            v[k] = x;  // valid in thread 0
        }
    }
    __syncthreads();
}

// Writes this CTA's partial sums; returns true in the CTA of the instance
// that arrives last, whose thread 0 then holds the fixed-order totals.
template <int NV>
__device__ __forceinline__ bool reduce_seg(const Ctx& c, int seg, double (&v)[NV], double (&tot)[NV]) {
    __shared__ double sm[NV][kThreads / 32];
    __shared__ bool last;
    block_sum<NV>(v, sm);
    const int b0 = c.seg_cta0[seg], b1 = c.seg_cta0[seg + 1];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) c.part[(size_t)k * c.ncta + blockIdx.x] = v[k];
        __threadfence();
        const unsigned ticket = atomicAdd(&c.tickets[seg], 1u);
        last = (ticket == (unsigned)(b1 - b0 - 1));
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        acc[k] = 0.0;
        for (int b = b0 + threadIdx.x; b < b1; b += kThreads) acc[k] += __ldcg(&c.part[(size_t)k * c.ncta + b]);
    }
    block_sum<NV>(acc, sm);
#pragma unroll
    for (int k = 0; k < NV; ++k) tot[k] = acc[k];
    if (threadIdx.x == 0) c.tickets[seg] = 0u;
    return true;
}

__device__ __forceinline__ bool stopped(const Where& w) { return __ldcg(&w.s[S_FLAG]) != 0.0; }

// rz = (r, M^-1 r) of CG: beta = rz / rz_old (not at the start of a solve)
__device__ __forceinline__ void cg_rz(double* s, double rz, bool start) {
    if (!start) s[S_BETA] = rz / s[S_RZ];
    s[S_RZ] = rz;
    if (!isfinite(rz)) {
        s[S_FLAG] = F_NAN;
    } else if (!(rz > 0.0)) {
        s[S_FLAG] = F_BREAKDOWN;
        s[S_WHY] = W_CG_RZ;
    }
}

inline Ctx make_ctx(tf_handle* h) {
    Device& d = h->d;
    Ctx c;
    c.wslot0 = d.wslot0;
    c.scol = d.scol;
    c.val = d.val;
    c.dinv = d.dinv;
    c.scal = d.scal;
    c.part = d.part;
    c.tickets = d.tickets;
    c.ncta = d.ncta;
    c.cta_seg = d.cta_seg;
    c.cta_node0 = d.cta_node0;
    c.cta_node1 = d.cta_node1;
    c.seg_cta0 = d.seg_cta0;
    c.seg_solve = d.seg_solve;
    c.xrow = d.nxb > 0 ? d.xrow : nullptr;
    c.xcol = d.xcol;
    c.xval = d.xval;
    c.nn = d.nn;
    c.check = d.check;
    return c;
}

}  // namespace tf
