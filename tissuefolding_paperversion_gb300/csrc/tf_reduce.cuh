// What the node-parallel kernels of the linear solve share: their operands,
// the node of a thread, and the per-instance reductions (also fused into the
// multigrid's last kernel).
#pragma once

#include "tf_internal.cuh"
#include "tf_stream.h"

namespace tf {

constexpr int kThreads = kNodeThreads;

enum Flag { F_RUNNING = 0, F_CONVERGED = 1, F_BREAKDOWN = 2, F_NAN = 3, F_DRIFT = 4 };
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
    int single, split, cta_nodes;     // one instance; see Device::split
    int stream;                       // the matrix is read past L2 (stream_matrix)
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
    int node;     // node of this thread
    bool valid;   // node inside this CTA's range
    int seg;      // instance of this CTA
    double* s;    // its scalars
    double flag;  // its stop flag
    int n1;       // end of this CTA's nodes
};

// With one instance nothing is looked up: the operands' loads need not wait for
// the tables', and the kernels below issue them before they test the flag (a
// batch tests first: its stopped instances would only cost bandwidth).
__device__ __forceinline__ Where where(const Ctx& c) {
    Where w;
    if (c.single) {
        w.seg = 0;
        w.node = blockIdx.x * c.cta_nodes + threadIdx.x;
        w.n1 = min((int)(blockIdx.x + 1) * c.cta_nodes, c.nn);
    } else {
        w.seg = c.cta_seg[blockIdx.x];
        w.node = c.cta_node0[blockIdx.x] + threadIdx.x;
        w.n1 = c.cta_node1[blockIdx.x];
    }
    w.valid = w.node < w.n1;
    w.s = c.scal + (size_t)w.seg * S_COUNT;
    w.flag = __ldcg(&w.s[S_FLAG]);
    return w;
}
__device__ __forceinline__ bool stopped(const Where& w) { return w.flag != 0.0; }
// The operands of this thread are to be loaded before the flag is tested.
__device__ __forceinline__ bool load_now(const Ctx& c, const Where& w) { return w.valid && (c.single || !stopped(w)); }

template <int NV>
__device__ __forceinline__ void warp_sum(double (&v)[NV]) {  // the sums are lane 0's
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
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
// that arrives last, whose thread 0 then holds the fixed-order totals.  In split
// CTAs the values are warp 0's, and it works alone: no barrier.  (MODE kSplit or
// kWhole: the kernel is compiled for one of the two.)
enum { kWhole = 0, kSplit = 1, kEither = 2 };
template <int NV, int MODE = kEither>
__device__ __forceinline__ bool reduce_seg(const Ctx& c, int seg, double (&v)[NV], double (&tot)[NV]) {
    __shared__ double sm[NV][kThreads / 32];
    __shared__ bool last;
    const int b0 = c.single ? 0 : c.seg_cta0[seg], b1 = c.single ? c.ncta : c.seg_cta0[seg + 1];
    if (MODE == kSplit || (MODE == kEither && c.split)) {
        if (threadIdx.x >= 32) return false;
        warp_sum<NV>(v);
        unsigned ticket = 0;
        if (threadIdx.x == 0) {
#pragma unroll
            for (int k = 0; k < NV; ++k) c.part[(size_t)k * c.ncta + blockIdx.x] = v[k];
            __threadfence();
            ticket = atomicAdd(&c.tickets[seg], 1u);
        }
        if (__shfl_sync(0xffffffffu, ticket, 0) != (unsigned)(b1 - b0 - 1)) return false;
        __threadfence();
#pragma unroll
        for (int k = 0; k < NV; ++k) tot[k] = 0.0;
#pragma unroll 8
        for (int b = b0 + (int)threadIdx.x; b < b1; b += 32)
#pragma unroll
            for (int k = 0; k < NV; ++k) tot[k] += __ldcg(&c.part[(size_t)k * c.ncta + b]);
        warp_sum<NV>(tot);
        if (threadIdx.x == 0) c.tickets[seg] = 0u;
        return true;
    }
    block_sum<NV>(v, sm);
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
    c.single = d.nseg == 1;
    c.split = d.split;
    c.stream = !d.split && stream_matrix(d.matrix_bytes, use_multigrid(h), d.l2_bytes);
    c.cta_nodes = d.cta_nodes;
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
