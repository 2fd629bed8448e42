// Smoothed-aggregation algebraic multigrid: the preconditioner of the
// Krylov solve of A du = g (A = K^T) on large meshes, in place of the
// block-Jacobi one.  No counterpart in the reference, which factorises the
// system with Pardiso (NewtonRaphsonSolver.cpp:418-683); the solution it
// converges to is the same (the Krylov tolerance is unchanged).
//
// Set-up, once per handle, on the host from the block pattern and the
// reference node positions:
//   * greedy aggregation of the node graph: a node whose neighbours are all
//     free becomes an aggregate with them; left-over nodes join the
//     neighbouring aggregate they touch most.  Aggregates never cross
//     instances (the graph of a batch is disconnected);
//   * near-null space: the six rigid-body modes at level 0 (translations and
//     rotations about the aggregate centroid), zero on fixed DOFs; at coarser
//     levels the R factors of the level below;
//   * tentative prolongator per aggregate from a modified Gram-Schmidt QR of
//     its near-null-space rows (6 coarse DOFs per aggregate; a dependent
//     column is dropped and its coarse DOF gets a unit diagonal);
//   * block patterns of the smoothed prolongator P = (I - omega D^-1 A) P_t
//     (node i couples to the aggregates of its neighbours), of T = A P and of
//     the coarse matrix P^T T, with per output block the ordered list of the
//     products that make it (no atomics, reproducible).
//   Plain aggregation (tf_options.precond 3) keeps P = P_t.
// Numeric phase, once per time step (all on the device), level by level:
//   lambda_max of D^-1 A by power iteration (smoother weights and prolongator
//   smoothing weight omega = 4 / (3.15 lambda)); P; T = A P; A_{l+1} = P^T T;
//   6x6 block inverses; Gauss-Jordan inverse of the coarsest level per
//   instance (<= 16 nodes); the explicit dense operator of the levels whose
//   matrices are small enough (k_dense_build).
// Application (one V-cycle per preconditioner call, all kernels, capturable
// in a CUDA graph): block-Jacobi pre- and post-smoothing (one damped sweep each
// way at level 0, kCoarseSweeps with Chebyshev weights on the coarser levels),
// residual,
// restriction, coarse correction.  Kernels of an instance whose Krylov
// solve has stopped return at once.
// Precision: the preconditioner is any fixed linear operator as far as the
// Krylov method is concerned, so the whole V-cycle -- its matrices (an FP32
// copy of the level-0 values and block inverses, the coarse operators and
// prolongators) and its vectors -- is FP32: half the bytes of its
// bandwidth-bound sweeps, and no FP32/FP64 conversions on the FP64 pipe.  The
// level-0 smoother reads S = D^-1 A in FP16 (entries of order one), a quarter
// of the FP64 bytes.
// The Krylov recurrences, their SpMVs with A and the convergence test are
// untouched FP64.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include <cuda_fp16.h>

#include "tf_reduce.cuh"

namespace tf {

namespace {

constexpr int kT = 256;
constexpr int kRestrictThreads = 128;  // per coarse node in the level-0 restriction
constexpr int kCoarseNodes = 16;  // nodes per instance at the coarsest level (96 DOFs)
constexpr int kCoarseDofs = 6 * kCoarseNodes;
constexpr int kInvThreads = 512;  // of the coarsest level's inverse
constexpr int kSmemOptIn = 227 * 1024;  // the most a CTA may ask for: no handle lowers another's limit
constexpr int kPowerIters = 16;
// The first level whose dense operators (one m x m FP32 matrix per instance,
// m = 6 nodes) fit these bytes, and every level below it, is applied as one
// matrix-vector product: reading 64 MB takes ~10 us at the HBM rate, where a
// level run kernel by kernel takes eight launches (~40 us on the 391-node
// level of the 320,000-prism sheet) and the levels below another ~20 us.
constexpr int64_t kDenseBytes = 64 << 20;
constexpr int kDenseThreads = 512;
constexpr int kDenseCols = 16;    // columns of the dense operator built together by one CTA
constexpr int kDenseQuads = kDenseCols / 4;  // lanes per row, four columns each
constexpr int kDenseRows = 3600;  // rows of an instance: its vectors have to fit shared memory, 64 bytes a row
// V-cycles the dense operator stands for.  Three instead of one cost nothing per
// application and leave the coarse levels nearly solved: 95 -> 70 CG iterations per
// 1.0M-prism wing step, 42 -> 39 BiCGStab iterations on the 320,000-prism sheet (two
// cycles: 78 and 41).
constexpr int kDenseCycles = 3;
constexpr int kDenseSweeps = 3;  // their sweeps each way
// damped block-Jacobi sweeps before and after the coarse correction on the
// levels >= 1 (level 0 sweeps once each way): more sweeps on the small,
// launch-bound coarse levels cut the Krylov iterations (320,000-prism sheet:
// 88 / 64 / 58 per step with 1 / 2 / 3 sweeps, 80 / 68.7 / 68.4 ms; 1M-prism
// wing: 201 / 150 / 128, 177 / 153 / 144 ms) while extra level-0 sweeps,
// which cost a full-size SpMV each, barely do
constexpr int kCoarseSweeps = 3;
// The sweeps of a level >= 1 are those of a Chebyshev polynomial of D^-1 A over
// [lambda / kChebRatio, lambda]: sweep k takes sweep_weight(k) times the level's
// weight, the post-sweeps in the reverse order (the cycle stays symmetric).  The
// same kernels reach further down the spectrum than with equal weights: Krylov
// iterations per step 38 -> 31 on the 320,000-prism sheet (23.7 -> 20.3 ms), 70 ->
// 57 on the 1M-prism wing (53.0 -> 46.1 ms), 106 -> 85 for 32 tissues (33.2 -> 28.2
// ms), 63 -> 50 at 46,208 prisms (7.0 -> 6.0 ms), kLevel0Weight included.  Ratios
// 4 / 8 / 15: 66 / 65 / 65, 97 / 92 / 84 and 56 / 53 / 50 iterations (wing, tissues,
// 46,208); the polynomial exceeds one beyond lambda (1 + 1 / ratio), and the power
// iteration's lambda is some 9 % low on the wing: 25 diverges there.
constexpr double kChebRatio = 8.0;
// Level 0 sweeps once each way, with this times its weight: 0.85 / 1 / 1.15 / 1.3
// give 43 / 41 / 38 / 36 iterations at 1,600 prisms, 25 / 24 / 21 / 20 at 9,728
// viscous ones, 63 / 62 / 61 / 60 at 46,208.  It converges for eigenvalues up to
// 1.3 times the estimate.
constexpr double kLevel0Weight = 1.2;

// ---- host set-up -----------------------------------------------------------------

// 1 / root k of the Chebyshev polynomial of degree n, over the weight 4 / (3 lambda)
static float sweep_weight(int k, int n) {
    const double lo = 1.0 / kChebRatio;
    const double root = 0.5 * (1.0 + lo) + 0.5 * (1.0 - lo) * std::cos(M_PI * (2 * k + 1) / (2.0 * n));
    return static_cast<float>(0.75 / root);
}

struct HostLevel {
    int n = 0, bs = 3;
    std::vector<int> rowptr, colidx;   // block pattern of this level
    std::vector<int> seg0;             // [nseg+1] node offsets per instance
    std::vector<double> B;             // [n * bs * 6] near-null space rows
};

// Greedy aggregation; returns the aggregate of each node and their count.
int aggregate(const std::vector<int>& rowptr, const std::vector<int>& colidx, int n, std::vector<int>& agg) {
    agg.assign(n, -1);
    int na = 0;
    for (int i = 0; i < n; ++i) {
        if (agg[i] >= 0) continue;
        bool free = true;
        for (int p = rowptr[i]; p < rowptr[i + 1] && free; ++p) free = agg[colidx[p]] < 0;
        if (!free) continue;
        for (int p = rowptr[i]; p < rowptr[i + 1]; ++p) agg[colidx[p]] = na;
        agg[i] = na++;
    }
    std::vector<int> cnt;
    for (int i = 0; i < n; ++i) {
        if (agg[i] >= 0) continue;
        // join the neighbouring aggregate with most connections (smallest id on ties)
        int best = -1, bestc = 0;
        for (int p = rowptr[i]; p < rowptr[i + 1]; ++p) {
            const int a = agg[colidx[p]];
            if (a < 0) continue;
            int c = 0;
            for (int q = rowptr[i]; q < rowptr[i + 1]; ++q) c += agg[colidx[q]] == a;
            if (c > bestc || (c == bestc && a < best)) {
                best = a;
                bestc = c;
            }
        }
        agg[i] = best >= 0 ? best : na++;
    }
    return na;
}

// Modified Gram-Schmidt of the m x 6 matrix M (row-major) in place: Q in M,
// R (6 x 6, row-major).  Returns the mask of dropped (dependent) columns.
int mgs(std::vector<double>& M, int m, double* R) {
    int dead = 0;
    std::fill(R, R + 36, 0.0);
    double ref[6];
    for (int c = 0; c < 6; ++c) {
        double s = 0.0;
        for (int r = 0; r < m; ++r) s += M[6 * r + c] * M[6 * r + c];
        ref[c] = std::sqrt(s);
    }
    for (int c = 0; c < 6; ++c) {
        for (int q = 0; q < c; ++q) {
            if (dead & (1 << q)) continue;
            double s = 0.0;
            for (int r = 0; r < m; ++r) s += M[6 * r + q] * M[6 * r + c];
            R[6 * q + c] = s;
            for (int r = 0; r < m; ++r) M[6 * r + c] -= s * M[6 * r + q];
        }
        double s = 0.0;
        for (int r = 0; r < m; ++r) s += M[6 * r + c] * M[6 * r + c];
        const double nv = std::sqrt(s);
        if (!(nv > 1e-10 * ref[c]) || !(ref[c] > 0.0)) {
            dead |= 1 << c;
            for (int r = 0; r < m; ++r) M[6 * r + c] = 0.0;
            for (int q = 0; q < 6; ++q) R[6 * q + c] = 0.0;
            continue;
        }
        R[6 * c + c] = nv;
        for (int r = 0; r < m; ++r) M[6 * r + c] /= nv;
    }
    return dead;
}

template <class T>
tf_status up(T** dst, const std::vector<T>& v) {
    const size_t n = std::max<size_t>(v.size(), 1);
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(dst), n * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("device allocation failed in the multigrid set-up");
        return TF_OUT_OF_MEMORY;
    }
    if (!v.empty()) TF_CUDA(cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return TF_OK;
}

template <class T>
tf_status zeros(T** dst, size_t n) {
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(dst), std::max<size_t>(n, 1) * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("device allocation failed in the multigrid set-up");
        return TF_OUT_OF_MEMORY;
    }
    TF_CUDA(cudaMemset(*dst, 0, std::max<size_t>(n, 1) * sizeof(T)));
    return TF_OK;
}

#define AMG_TRY(expr)               \
    do {                            \
        tf_status _s = (expr);      \
        if (_s != TF_OK) return _s; \
    } while (0)


struct DenseBuild;
__global__ void k_dense_build(DenseBuild B);

}  // namespace

// Device view of one level: what the V-cycle reads and writes, all FP32
// (see the precision note above); the smoother weights are FP64 scalars.
struct AmgLevel {
    int n = 0, bs = 3;
    // matrix of levels >= 1: CSR of 6x6 row-major blocks
    int* rowptr = nullptr;
    int* colidx = nullptr;
    int* rowof = nullptr;
    int* diag = nullptr;  // block index of (i, i)
    float* val = nullptr;
    int64_t nnzb = 0;
    float* dinv = nullptr;   // [n][36] block inverses (levels >= 1)
    int* seg = nullptr;      // [n] instance of each node (levels >= 1)
    int* seg0 = nullptr;     // [nseg+1] node offsets per instance (levels >= 1)
    // prolongator to level + 1 (absent at the coarsest level): bs x 6
    // row-major blocks, once by fine row and once by coarse column
    int* prow = nullptr;     // [n+1] blocks of each fine node
    int* pcol = nullptr;     // [npb] coarse node of each block
    float* Pv = nullptr;     // [npb][bs*6]
    int* pcptr = nullptr;    // [n_{l+1}+1] blocks of each coarse node (column order)
    int* pcrow = nullptr;    // [npb] fine node of each block, column order
    float* Pc = nullptr;     // [npb][bs*6] the blocks in column order
    __half* Pvh = nullptr;   // level 0: FP16 copies of Pv and Pc for the V-cycle's transfers
    __half* Pch = nullptr;
    __half* valh = nullptr;  // levels >= 1: S = D^-1 A in FP16 [nnzb][36] for the V-cycle's sweeps
    int64_t npb = 0;
    uint8_t* dead = nullptr; // [n * bs] (levels >= 1) DOFs with a zero prolongator column
    // coarse image of the extra blocks outside the element pattern (levels >=
    // 1): X_l = P^T X_{l-1} P, CSR of 6x6 blocks (null: none)
    int* xrow = nullptr;
    int* xcol = nullptr;
    float* xval = nullptr;
    int64_t nx = 0;
    // vectors (levels >= 1: r input, e output; all levels: x, t work)
    float *r = nullptr, *x = nullptr, *t = nullptr, *e = nullptr;
    int ncoarse = 0;         // nodes of level + 1
    int single = 0;          // one instance
    int* check = nullptr;    // checked build: failed index checks
};

// The level-0 transfer of the V-cycle with the smoothing folded in,
// Q = (I - omega S) P (pattern of T = A P, 3x6 blocks, FP16 like P's own copy
// for the transfers): by row in the 32-row slices of the node-parallel kernels
// (entries 0-15 of a lane's block as two 16-byte packs, 16-17 as one word), and
// by coarse column.
struct AmgQ {
    int* slot0 = nullptr;    // [ncta * kWarps + 1] first slot of each warp's rows
    int* col = nullptr;      // [nslots * 32] coarse node of each slot and lane
    uint4* v16 = nullptr;    // [nslots * 2 * 32]
    uint32_t* v2 = nullptr;  // [nslots * 32]
    int* cptr = nullptr;     // [n_1 + 1] blocks of each coarse node
    int* crow = nullptr;     // [nT] fine node of each
    uint32_t* cval = nullptr;  // [nT][9]
    // set-up: per T block its P block (-1: none), slice position and column position
    int* tp = nullptr;
    int* pos = nullptr;
    int* cpos = nullptr;
};

// Lists of the numeric set-up of the transfer from level l to l + 1
// (device arrays, built once on the host from the block patterns).
struct AmgSetup {
    float* Pt = nullptr;     // [n][bs*6] tentative prolongator (one block per fine node)
    int* agg = nullptr;      // [n] aggregate of each fine node
    int* pbrow = nullptr;    // [npb] fine node of each prolongator block
    int* sptr = nullptr;     // [npb+1] fine-matrix blocks (i, j), agg(j) = column, per block (i, .)
    int* slist = nullptr;
    int* cperm = nullptr;    // [npb] row-order block at each column-order position
    int64_t nT = 0;          // blocks of T = A P (bs x 6)
    int* trow = nullptr;     // [nT] fine node of each T block
    int* tptr = nullptr;     // [nT+1] pairs (fine-matrix block, prolongator block) per T block
    int* ta = nullptr;
    int* tb = nullptr;
    float* T = nullptr;      // [nT][bs*6]
    int* gptr = nullptr;     // [nnzb_{l+1}+1] pairs (prolongator block, T block) per coarse block
    int* gp = nullptr;
    int* gt = nullptr;
    int* xptr = nullptr;     // [nx_{l+1}+1] triples (extra block (J, I), P block (J, K), P block (I, M))
    int* xtrip = nullptr;    // per coarse extra block (K, M)
};

struct Amg {
    int nlev = 0;
    bool smooth = true;        // smoothed (true) or plain (false) aggregation
    AmgLevel L[kAmgMaxLevels];
    AmgSetup S[kAmgMaxLevels];
    AmgQ Q;
    double* omega = nullptr;   // [nlev] smoother weights 4 / (3 lambda)
    double* omega0 = nullptr;  // level 0's in the V-cycle (omega[0] smooths the prolongator)
    double* pscal = nullptr;   // [nlev][2] power-iteration scalars (scale, lambda)
    float* x1 = nullptr;       // [3 n] the smoothed part of a V-cycle's result (k_q_smooth)
    float* pv = nullptr;       // power-iteration vectors (max n*bs each)
    float* pw = nullptr;
    double* part = nullptr;    // per-CTA partial sums
    unsigned* ticket = nullptr;
    float* val32 = nullptr;    // FP32 copy of the level-0 values (sliced layout)
    // the smoother's level-0 operator S = D^-1 A in FP16, slot by slot in the
    // sliced order: entries 0-7 of a row's block as one 16-byte pack
    // ([slot][lane][8]), then entry 8 of every block ([slot][lane]) -- two
    // loads per block instead of nine
    __half* valh = nullptr;
    float* dinv32 = nullptr;   // FP32 copy of the level-0 block inverses
    float* diag32 = nullptr;   // FP32 copy of the level-0 diagonal blocks, [9 n] row-major
    int nseg = 1;
    int* cnode0 = nullptr;     // [nseg+1] coarsest-level node offsets per instance
    int* cinv0 = nullptr;      // [nseg+1] offsets of the dense inverses
    float* cinv = nullptr;     // coarsest inverses, m_g x m_g row-major
    bool coarse_exact = true;
    int max_cm = 0;
    int v0_smem = 0;           // shared memory of the level-0 prolongation (3 floats per block of a CTA)
    // levels dense..nlev-1 are applied as one dense operator per instance
    // (0: none, the coarsest level has too many DOFs for an exact inverse)
    int dense = 0;
    float* dmat = nullptr;     // the operators, m_g x m_g row-major (cinv when dense is the coarsest level)
    int* doff = nullptr;       // [nseg+1] their offsets
    int2* dgroup = nullptr;    // column groups (instance, first column) of their construction
    int ndgroup = 0;
    float* dwork = nullptr;    // work vectors of the construction, per CTA
    int dgrid = 0;             // its CTAs
    int dlvl[kAmgMaxLevels] = {};  // offset of each level's vectors within a CTA's work
    int64_t dstride = 0;
    int dsmem = 0;             // its shared memory
    int smooth_unroll = 4;     // slots in flight per lane in the level-0 smoother's row product (2, 4, 8)
    std::vector<int> h_n;      // nodes per level (host)
    std::vector<int> h_prow[kAmgMaxLevels], h_pcol[kAmgMaxLevels];  // prolongator patterns (host)
    int64_t x_version = -1;    // extra-block layout the coarse extra blocks were built for
    // what the next solve has to redo: 0 nothing, 1 the FP32 copies of the
    // level-0 matrix (new assembly, same time step), 2 the whole hierarchy
    int stale = 2;
    bool reused = false;       // the last numeric phase kept the coarse levels
    long rebuilds = 0;         // full numeric rebuilds so far
};

void amg_free(Amg* a) {
    if (!a) return;
    for (int l = 0; l < kAmgMaxLevels; ++l) {  // nlev is not known yet where a set-up ran out of memory
        AmgLevel& L = a->L[l];
        void* ptrs[] = {L.rowptr, L.colidx, L.rowof, L.diag, L.val, L.seg, L.seg0, L.prow, L.pcol, L.Pv,
                        L.pcptr, L.pcrow, L.Pc, L.dead, L.r, L.x, L.t, L.e, L.Pvh, L.Pch, L.valh};
        for (void* p : ptrs)
            if (p) cudaFree(p);
        if (l > 0 && L.dinv) cudaFree(L.dinv);
        AmgSetup& S = a->S[l];
        void* sptrs[] = {S.Pt, S.agg, S.pbrow, S.sptr, S.slist, S.cperm, S.trow, S.tptr, S.ta, S.tb, S.T,
                         S.gptr, S.gp, S.gt, S.xptr, S.xtrip, L.xrow, L.xcol, L.xval};
        for (void* p : sptrs)
            if (p) cudaFree(p);
    }
    if (a->dmat != a->cinv && a->dmat) cudaFree(a->dmat);
    if (a->doff != a->cinv0 && a->doff) cudaFree(a->doff);
    void* ptrs[] = {a->omega, a->omega0, a->pscal, a->pv, a->pw, a->part, a->ticket, a->cnode0, a->cinv0, a->cinv,
                    a->val32, a->dinv32, a->valh, a->diag32, a->dgroup, a->dwork,
                    a->Q.slot0, a->Q.col, a->Q.v16, a->Q.v2, a->Q.cptr, a->Q.crow, a->Q.cval, a->Q.tp, a->Q.pos,
                    a->Q.cpos, a->x1};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete a;
}

// Layouts of Q (see AmgQ) from the pattern of T = A P.
static tf_status build_q(const Device& d, AmgQ* q, const std::vector<int>& trowptr, const std::vector<int>& tcol,
                         const std::vector<int>& prow, const std::vector<int>& pcol, int nc) {
    const int n = d.nn;
    const int64_t nT = (int64_t)tcol.size();
    std::vector<int> c0(d.ncta), c1(d.ncta);
    TF_CUDA(cudaMemcpy(c0.data(), d.cta_node0, sizeof(int) * (size_t)d.ncta, cudaMemcpyDeviceToHost));
    TF_CUDA(cudaMemcpy(c1.data(), d.cta_node1, sizeof(int) * (size_t)d.ncta, cudaMemcpyDeviceToHost));
    std::vector<int> slot0((size_t)d.ncta * kWarps + 1, 0), tp(nT, -1), pos(nT), cpos(nT), cptr(nc + 1, 0), crow(nT);
    int ns = 0;
    for (int c = 0; c < d.ncta; ++c)
        for (int w = 0; w < (d.split ? 1 : kWarps); ++w) {
            const int r0 = c0[c] + 32 * w, r1 = std::min(r0 + 32, c1[c]);
            int most = 0;
            for (int i = r0; i < r1; ++i) {
                most = std::max(most, trowptr[i + 1] - trowptr[i]);
                for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) pos[t] = (ns + t - trowptr[i]) * 32 + (i - r0);
            }
            for (int v = w; v < (d.split ? kWarps : w + 1); ++v)  // split: the warps share the slice's slots
                slot0[(size_t)c * kWarps + v] = ns + (d.split ? most * v / kWarps : 0);
            ns += most;
        }
    slot0[(size_t)d.ncta * kWarps] = ns;
    std::vector<int> col((size_t)ns * 32, 0);
    for (int64_t t = 0; t < nT; ++t) {
        col[pos[t]] = tcol[t];
        cptr[tcol[t] + 1]++;
    }
    for (int J = 0; J < nc; ++J) cptr[J + 1] += cptr[J];
    {
        std::vector<int> fill(cptr.begin(), cptr.end() - 1);
        for (int i = 0; i < n; ++i) {
            int b = prow[i];
            for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) {
                cpos[t] = fill[tcol[t]]++;
                crow[cpos[t]] = i;
                while (b < prow[i + 1] && pcol[b] < tcol[t]) ++b;  // both sorted by column
                if (b < prow[i + 1] && pcol[b] == tcol[t]) tp[t] = b;
            }
        }
    }
    AMG_TRY(up(&q->slot0, slot0));
    AMG_TRY(up(&q->col, col));
    AMG_TRY(zeros(&q->v16, (size_t)ns * 64));
    AMG_TRY(zeros(&q->v2, (size_t)ns * 32));
    AMG_TRY(up(&q->cptr, cptr));
    AMG_TRY(up(&q->crow, crow));
    AMG_TRY(zeros(&q->cval, (size_t)nT * 9));
    AMG_TRY(up(&q->tp, tp));
    AMG_TRY(up(&q->pos, pos));
    AMG_TRY(up(&q->cpos, cpos));
    return TF_OK;
}

namespace {
__global__ void k_coarse_invert(AmgLevel L, const int* __restrict__ cnode0, const int* __restrict__ cinv0,
                                float* __restrict__ cinv);
}

// Symbolic set-up from the level-0 pattern, the reference positions and the
// fixed DOFs.  Level 0 uses the handle's own matrix, block inverses and
// sliced storage.
tf_status amg_build(tf_handle* h, const double* pos) {
    Device& d = h->d;
    Amg* a = new Amg;
    h->amg = a;
    a->nseg = d.nseg;
    a->smooth = h->opt.precond != 3;
    std::vector<HostLevel> H(1);
    H[0].n = d.nn;
    H[0].bs = 3;
    H[0].rowptr = h->h_rowptr;
    H[0].colidx = h->h_colidx;
    H[0].seg0 = h->h_seg_node0;
    int lev = 0;
    while (true) {
        HostLevel& F = H[lev];
        int maxn = 0;
        for (int g = 0; g < d.nseg; ++g) maxn = std::max(maxn, F.seg0[g + 1] - F.seg0[g]);
        if (maxn <= kCoarseNodes || lev + 1 >= kAmgMaxLevels) break;
        std::vector<int> agg;
        const int na = aggregate(F.rowptr, F.colidx, F.n, agg);
        if (na >= F.n) break;  // no coarsening possible
        // members per aggregate (node order)
        std::vector<int> mptr(na + 1, 0), mlist(F.n);
        for (int i = 0; i < F.n; ++i) mptr[agg[i] + 1]++;
        for (int c = 0; c < na; ++c) mptr[c + 1] += mptr[c];
        {
            std::vector<int> fill(mptr.begin(), mptr.end() - 1);
            for (int i = 0; i < F.n; ++i) mlist[fill[agg[i]]++] = i;
        }
        // tentative prolongator and the next near-null space
        const int bs = F.bs;
        std::vector<double> P((size_t)F.n * bs * 6, 0.0), Bc((size_t)na * 36, 0.0);
        std::vector<uint8_t> dead((size_t)na * 6, 0);
        std::vector<double> M;
        for (int c = 0; c < na; ++c) {
            const int m0 = mptr[c], m1 = mptr[c + 1];
            const int rows = (m1 - m0) * bs;
            M.assign((size_t)rows * 6, 0.0);
            if (lev == 0) {
                double cen[3] = {0, 0, 0};
                for (int q = m0; q < m1; ++q)
                    for (int k = 0; k < 3; ++k) cen[k] += pos[3 * (size_t)mlist[q] + k];
                for (int k = 0; k < 3; ++k) cen[k] /= (m1 - m0);
                for (int q = m0; q < m1; ++q) {
                    const int i = mlist[q];
                    const double rx = pos[3 * (size_t)i] - cen[0], ry = pos[3 * (size_t)i + 1] - cen[1],
                                 rz = pos[3 * (size_t)i + 2] - cen[2];
                    // rows x, y, z of [I | e_x x r, e_y x r, e_z x r]
                    const double rowsv[3][6] = {{1, 0, 0, 0, rz, -ry}, {0, 1, 0, -rz, 0, rx}, {0, 0, 1, ry, -rx, 0}};
                    for (int k = 0; k < 3; ++k) {
                        const bool fx = h->h_fixed[3 * (size_t)i + k] != 0;
                        for (int col = 0; col < 6; ++col)
                            M[(size_t)(bs * (q - m0) + k) * 6 + col] = fx ? 0.0 : rowsv[k][col];
                    }
                }
            } else {
                for (int q = m0; q < m1; ++q) {
                    const int i = mlist[q];
                    for (int k = 0; k < 6; ++k)
                        for (int col = 0; col < 6; ++col)
                            M[(size_t)(6 * (q - m0) + k) * 6 + col] = F.B[(size_t)i * 36 + 6 * k + col];
                }
            }
            double R[36];
            const int dm = mgs(M, rows, R);
            for (int k = 0; k < 6; ++k) dead[(size_t)c * 6 + k] = (dm >> k) & 1;
            std::copy(R, R + 36, Bc.begin() + (size_t)c * 36);
            for (int q = m0; q < m1; ++q) {
                const int i = mlist[q];
                for (int k = 0; k < bs; ++k)
                    for (int col = 0; col < 6; ++col)
                        P[((size_t)i * bs + k) * 6 + col] = M[(size_t)(bs * (q - m0) + k) * 6 + col];
            }
        }
        // prolongator pattern: block (i, J) for the aggregates J of node i's
        // neighbours (smoothed: P = (I - omega D^-1 A) P_tentative) or for
        // node i's own aggregate only (plain: P = P_tentative)
        std::vector<int> prow(F.n + 1, 0), pcol, mark(na, -1), cols;
        for (int i = 0; i < F.n; ++i) {
            cols.assign(1, agg[i]);
            mark[agg[i]] = i;
            if (a->smooth)
                for (int p = F.rowptr[i]; p < F.rowptr[i + 1]; ++p) {
                    const int J = agg[F.colidx[p]];
                    if (mark[J] != i) {
                        mark[J] = i;
                        cols.push_back(J);
                    }
                }
            std::sort(cols.begin(), cols.end());
            pcol.insert(pcol.end(), cols.begin(), cols.end());
            prow[i + 1] = static_cast<int>(pcol.size());
        }
        const int npb = static_cast<int>(pcol.size());
        std::vector<int> pbrow(npb);
        for (int i = 0; i < F.n; ++i)
            for (int b = prow[i]; b < prow[i + 1]; ++b) pbrow[b] = i;
        // smoothing lists: fine block (i, j) adds to prolongator block (i, agg(j))
        std::vector<int> sptr(npb + 1, 0), slist;
        if (a->smooth) {
            const int fnnzb = F.rowptr[F.n];
            std::vector<int> sb(fnnzb);
            for (int i = 0; i < F.n; ++i)
                for (int p = F.rowptr[i]; p < F.rowptr[i + 1]; ++p) {
                    const int J = agg[F.colidx[p]];
                    sb[p] = static_cast<int>(std::lower_bound(pcol.begin() + prow[i], pcol.begin() + prow[i + 1], J) -
                                             pcol.begin());
                    sptr[sb[p] + 1]++;
                }
            for (int b = 0; b < npb; ++b) sptr[b + 1] += sptr[b];
            slist.resize(fnnzb);
            std::vector<int> fill(sptr.begin(), sptr.end() - 1);
            for (int p = 0; p < fnnzb; ++p) slist[fill[sb[p]]++] = p;
        }
        // the same blocks by coarse column (fine nodes ascending within a column)
        std::vector<int> pcptr(na + 1, 0), cperm(npb), pcrow(npb);
        for (int b = 0; b < npb; ++b) pcptr[pcol[b] + 1]++;
        for (int c = 0; c < na; ++c) pcptr[c + 1] += pcptr[c];
        {
            std::vector<int> fill(pcptr.begin(), pcptr.end() - 1);
            for (int b = 0; b < npb; ++b) {
                const int q = fill[pcol[b]]++;
                cperm[q] = b;
                pcrow[q] = pbrow[b];
            }
        }
        // T = A P: pattern per fine row and, per T block, its pairs
        // (fine-matrix block (i, j), prolongator block (j, J))
        std::vector<int> trowptr(F.n + 1, 0), tcol;
        std::fill(mark.begin(), mark.end(), -1);
        for (int i = 0; i < F.n; ++i) {
            cols.clear();
            for (int p = F.rowptr[i]; p < F.rowptr[i + 1]; ++p) {
                const int j = F.colidx[p];
                for (int b = prow[j]; b < prow[j + 1]; ++b)
                    if (mark[pcol[b]] != i) {
                        mark[pcol[b]] = i;
                        cols.push_back(pcol[b]);
                    }
            }
            std::sort(cols.begin(), cols.end());
            tcol.insert(tcol.end(), cols.begin(), cols.end());
            trowptr[i + 1] = static_cast<int>(tcol.size());
        }
        const int64_t nT = (int64_t)tcol.size();
        std::vector<int> trow(nT), tptr(nT + 1, 0), posJ(na, -1);
        for (int i = 0; i < F.n; ++i) {
            for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) {
                trow[t] = i;
                posJ[tcol[t]] = t;
            }
            for (int p = F.rowptr[i]; p < F.rowptr[i + 1]; ++p) {
                const int j = F.colidx[p];
                for (int b = prow[j]; b < prow[j + 1]; ++b) tptr[posJ[pcol[b]] + 1]++;
            }
        }
        for (int64_t t = 0; t < nT; ++t) tptr[t + 1] += tptr[t];
        std::vector<int> ta(tptr[nT]), tb(tptr[nT]);
        {
            std::vector<int> fill(tptr.begin(), tptr.end() - 1);
            for (int i = 0; i < F.n; ++i) {
                for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) posJ[tcol[t]] = t;
                for (int p = F.rowptr[i]; p < F.rowptr[i + 1]; ++p) {
                    const int j = F.colidx[p];
                    for (int b = prow[j]; b < prow[j + 1]; ++b) {
                        const int k = fill[posJ[pcol[b]]]++;
                        ta[k] = p;
                        tb[k] = b;
                    }
                }
            }
        }
        if (lev == 0) AMG_TRY(build_q(d, &a->Q, trowptr, tcol, prow, pcol, na));
        // coarse pattern: row I joins the T rows of the fine nodes with a
        // block in column I
        HostLevel C;
        C.n = na;
        C.bs = 6;
        C.B = std::move(Bc);
        C.seg0.assign(d.nseg + 1, 0);
        // aggregates of an instance are contiguous and its first node is a
        // root: roots are created in node order, left-over nodes only join
        // aggregates of their own instance
        for (int g = 0; g <= d.nseg; ++g) C.seg0[g] = g < d.nseg ? (F.seg0[g] < F.n ? agg[F.seg0[g]] : na) : na;
        C.rowptr.assign(na + 1, 0);
        std::fill(mark.begin(), mark.end(), -1);
        for (int c = 0; c < na; ++c) {
            cols.clear();
            for (int q = pcptr[c]; q < pcptr[c + 1]; ++q) {
                const int i = pcrow[q];
                for (int t = trowptr[i]; t < trowptr[i + 1]; ++t)
                    if (mark[tcol[t]] != c) {
                        mark[tcol[t]] = c;
                        cols.push_back(tcol[t]);
                    }
            }
            std::sort(cols.begin(), cols.end());
            C.colidx.insert(C.colidx.end(), cols.begin(), cols.end());
            C.rowptr[c + 1] = static_cast<int>(C.colidx.size());
        }
        const int64_t cnnzb = (int64_t)C.colidx.size();
        // Galerkin pairs (prolongator block (i, I), T block (i, J)) per coarse block (I, J)
        std::vector<int> gptr(cnnzb + 1, 0);
        for (int c = 0; c < na; ++c) {
            for (int p = C.rowptr[c]; p < C.rowptr[c + 1]; ++p) posJ[C.colidx[p]] = p;
            for (int q = pcptr[c]; q < pcptr[c + 1]; ++q) {
                const int i = pcrow[q];
                for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) gptr[posJ[tcol[t]] + 1]++;
            }
        }
        for (int64_t c = 0; c < cnnzb; ++c) gptr[c + 1] += gptr[c];
        std::vector<int> gp(gptr[cnnzb]), gt(gptr[cnnzb]);
        {
            std::vector<int> fill(gptr.begin(), gptr.end() - 1);
            for (int c = 0; c < na; ++c) {
                for (int p = C.rowptr[c]; p < C.rowptr[c + 1]; ++p) posJ[C.colidx[p]] = p;
                for (int q = pcptr[c]; q < pcptr[c + 1]; ++q) {
                    const int i = pcrow[q];
                    for (int t = trowptr[i]; t < trowptr[i + 1]; ++t) {
                        const int k = fill[posJ[tcol[t]]]++;
                        gp[k] = cperm[q];
                        gt[k] = t;
                    }
                }
            }
        }
        // device arrays of the fine level's transfer
        AmgLevel& DL = a->L[lev];
        DL.npb = npb;
        a->h_prow[lev] = prow;
        a->h_pcol[lev] = pcol;
        AMG_TRY(up(&DL.prow, prow));
        AMG_TRY(up(&DL.pcol, pcol));
        AMG_TRY(zeros(&DL.Pv, (size_t)npb * bs * 6));
        AMG_TRY(up(&DL.pcptr, pcptr));
        AMG_TRY(up(&DL.pcrow, pcrow));
        AMG_TRY(zeros(&DL.Pc, (size_t)npb * bs * 6));
        if (lev == 0) {
            AMG_TRY(zeros(&DL.Pvh, (size_t)npb * bs * 6));
            AMG_TRY(zeros(&DL.Pch, (size_t)npb * bs * 6));
        }
        AmgSetup& DS = a->S[lev];
        DS.nT = nT;
        AMG_TRY(up(&DS.Pt, std::vector<float>(P.begin(), P.end())));
        AMG_TRY(up(&DS.agg, agg));
        AMG_TRY(up(&DS.pbrow, pbrow));
        AMG_TRY(up(&DS.sptr, sptr));
        AMG_TRY(up(&DS.slist, slist));
        AMG_TRY(up(&DS.cperm, cperm));
        AMG_TRY(up(&DS.trow, trow));
        AMG_TRY(up(&DS.tptr, tptr));
        AMG_TRY(up(&DS.ta, ta));
        AMG_TRY(up(&DS.tb, tb));
        AMG_TRY(zeros(&DS.T, (size_t)nT * bs * 6));
        AMG_TRY(up(&DS.gptr, gptr));
        AMG_TRY(up(&DS.gp, gp));
        AMG_TRY(up(&DS.gt, gt));
        // the coarse level's own arrays
        AmgLevel& CL = a->L[lev + 1];
        CL.n = na;
        CL.bs = 6;
        CL.nnzb = cnnzb;
        std::vector<int> rowof(cnnzb), diag(na);
        std::vector<int> seg(na);
        for (int c = 0; c < na; ++c) {
            for (int p = C.rowptr[c]; p < C.rowptr[c + 1]; ++p) {
                rowof[p] = c;
                if (C.colidx[p] == c) diag[c] = p;
            }
        }
        for (int g = 0; g < d.nseg; ++g)
            for (int c = C.seg0[g]; c < C.seg0[g + 1]; ++c) seg[c] = g;
        AMG_TRY(up(&CL.rowptr, C.rowptr));
        AMG_TRY(up(&CL.colidx, C.colidx));
        AMG_TRY(up(&CL.rowof, rowof));
        AMG_TRY(up(&CL.diag, diag));
        AMG_TRY(up(&CL.seg, seg));
        AMG_TRY(up(&CL.seg0, C.seg0));
        AMG_TRY(up(&CL.dead, dead));
        AMG_TRY(zeros(&CL.val, (size_t)cnnzb * 36));  // float
        AMG_TRY(zeros(&CL.valh, (size_t)cnnzb * 36));
        AMG_TRY(zeros(&CL.dinv, (size_t)na * 36));
        H.push_back(std::move(C));
        ++lev;
    }
    a->nlev = lev + 1;
    if (a->nlev < 2) {  // nothing to coarsen: block-Jacobi is used instead
        amg_free(a);
        h->amg = nullptr;
        return TF_OK;
    }
    // level 0 device view: the handle's own arrays
    AmgLevel& L0 = a->L[0];
    L0.n = d.nn;
    L0.bs = 3;
    L0.nnzb = d.nnzb;
    {
        // blocks of the prolongator rows of each node-parallel CTA
        std::vector<int> c0(d.ncta), c1(d.ncta), prow0(d.nn + 1);
        TF_CUDA(cudaMemcpy(c0.data(), d.cta_node0, sizeof(int) * (size_t)d.ncta, cudaMemcpyDeviceToHost));
        TF_CUDA(cudaMemcpy(c1.data(), d.cta_node1, sizeof(int) * (size_t)d.ncta, cudaMemcpyDeviceToHost));
        TF_CUDA(cudaMemcpy(prow0.data(), L0.prow, sizeof(int) * (size_t)(d.nn + 1), cudaMemcpyDeviceToHost));
        int maxb = 1;
        for (int c = 0; c < d.ncta; ++c) maxb = std::max(maxb, prow0[c1[c]] - prow0[c0[c]]);
        a->v0_smem = static_cast<int>(3 * sizeof(float) * (size_t)maxb);
    }
    size_t maxv = 0;
    for (int l = 0; l < a->nlev; ++l) {
        AmgLevel& L = a->L[l];
        const size_t nv = (size_t)L.n * L.bs;
        maxv = std::max(maxv, nv);
        AMG_TRY(zeros(&L.x, nv));
        AMG_TRY(zeros(&L.t, nv));
        if (l > 0) {
            AMG_TRY(zeros(&L.r, nv));
            AMG_TRY(zeros(&L.e, nv));
        }
        a->h_n.push_back(L.n);
    }
    for (int l = 0; l < a->nlev; ++l) {
        a->L[l].ncoarse = l + 1 < a->nlev ? a->L[l + 1].n : 0;
        a->L[l].check = d.check;
        a->L[l].single = d.nseg == 1;
    }
    AMG_TRY(zeros(&a->omega, (size_t)a->nlev));
    AMG_TRY(zeros(&a->omega0, 1));
    AMG_TRY(zeros(&a->val32, (size_t)d.nval));
    AMG_TRY(zeros(&a->valh, (size_t)d.nval));
    AMG_TRY(zeros(&a->dinv32, 9 * (size_t)d.nn));
    AMG_TRY(zeros(&a->diag32, 9 * (size_t)d.nn));
    AMG_TRY(zeros(&a->x1, 3 * (size_t)d.nn));
    AMG_TRY(zeros(&a->pscal, 2 * (size_t)a->nlev));
    if (!h->side_stream) {
        TF_CUDA(cudaStreamCreateWithFlags(&h->side_stream, cudaStreamNonBlocking));
        TF_CUDA(cudaStreamCreateWithFlags(&h->cap_side, cudaStreamNonBlocking));
        TF_CUDA(cudaEventCreateWithFlags(&h->fork_ev, cudaEventDisableTiming));
        TF_CUDA(cudaEventCreateWithFlags(&h->join_ev, cudaEventDisableTiming));
    }
    AMG_TRY(zeros(&a->pv, maxv));
    AMG_TRY(zeros(&a->pw, maxv));
    int64_t maxc = 0;  // CTAs of the warp-per-row power iteration on the coarse levels
    for (int l = 1; l < a->nlev; ++l) maxc = std::max<int64_t>(maxc, cdiv(32 * (int64_t)a->L[l].n, kT));
    AMG_TRY(zeros(&a->part, (size_t)std::max<int64_t>({(int64_t)cdiv((int64_t)maxv, kT), (int64_t)d.ncta, maxc}) + 1));
    AMG_TRY(zeros(&a->ticket, 1));
    // coarsest level: dense inverse per instance
    const HostLevel& CH = H.back();
    std::vector<int> cinv0(d.nseg + 1, 0);
    a->max_cm = 0;
    for (int g = 0; g < d.nseg; ++g) {
        const int m = CH.bs * (CH.seg0[g + 1] - CH.seg0[g]);
        a->max_cm = std::max(a->max_cm, m);
        cinv0[g + 1] = cinv0[g] + m * m;
    }
    a->coarse_exact = a->max_cm <= kCoarseDofs;
    AMG_TRY(up(&a->cnode0, CH.seg0));
    AMG_TRY(up(&a->cinv0, cinv0));
    AMG_TRY(zeros(&a->cinv, (size_t)std::max(cinv0[d.nseg], 1)));
    if (!a->coarse_exact) return TF_OK;
    TF_CUDA(cudaFuncSetAttribute(k_coarse_invert, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * kCoarseDofs * kCoarseDofs)));
    // the dense operator: from the finest level that fits down (the coarsest
    // level's inverse exists anyway)
    a->dense = a->nlev - 1;
    std::vector<int> doff = cinv0;
    for (int l = a->nlev - 2; l >= 1; --l) {
        std::vector<int> off(d.nseg + 1, 0);
        int64_t total = 0;
        bool fits = true;
        for (int g = 0; g < d.nseg; ++g) {
            const int64_t m = 6 * (int64_t)(H[l].seg0[g + 1] - H[l].seg0[g]);
            total += m * m;
            fits = fits && total * (int64_t)sizeof(float) <= kDenseBytes && m <= kDenseRows;
            if (!fits) break;
            off[g + 1] = static_cast<int>(total);
        }
        if (!fits) break;
        a->dense = l;
        doff = off;
    }
    if (a->dense == a->nlev - 1) {
        a->dmat = a->cinv;
        a->doff = a->cinv0;
        return TF_OK;
    }
    std::vector<int2> group;
    std::vector<int> maxn(a->nlev, 0);
    for (int l = a->dense; l < a->nlev; ++l)
        for (int g = 0; g < d.nseg; ++g) maxn[l] = std::max(maxn[l], H[l].seg0[g + 1] - H[l].seg0[g]);
    for (int g = 0; g < d.nseg; ++g) {
        const int m = 6 * (H[a->dense].seg0[g + 1] - H[a->dense].seg0[g]);
        for (int c = 0; c < m; c += kDenseCols) group.push_back(make_int2(g, c));
    }
    a->dsmem = static_cast<int>(sizeof(float) * 6 * (size_t)maxn[a->dense] * kDenseCols);
    TF_CUDA(cudaFuncSetAttribute(k_dense_build, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(float) * kDenseRows * kDenseCols)));
    for (int l = a->dense; l < a->nlev; ++l) {  // r, x, t, e per level, the result too at the first
        a->dlvl[l] = static_cast<int>(a->dstride);
        a->dstride += (int64_t)(l == a->dense ? 5 : 4) * 6 * maxn[l] * kDenseCols;
    }
    a->ndgroup = static_cast<int>(group.size());
    a->dgrid = std::min(a->ndgroup, 152);
    AMG_TRY(up(&a->dgroup, group));
    AMG_TRY(up(&a->doff, doff));
    AMG_TRY(zeros(&a->dmat, (size_t)doff[d.nseg]));
    AMG_TRY(zeros(&a->dwork, (size_t)a->dgrid * (size_t)a->dstride));
    return TF_OK;
}

// The hierarchy of a handle that could do without: its size is several times the
// handle's own on small meshes (11,163 nodes: 200 MB beside 56), so where it does not
// fit the handle keeps block-Jacobi instead of being refused.
tf_status amg_build_trial(tf_handle* h, const double* pos) {
    const tf_status s = amg_build(h, pos);
    if (s != TF_OUT_OF_MEMORY) return s;
    amg_free(h->amg);
    h->amg = nullptr;
    h->amg_trial = false;
    return TF_OK;
}

// Patterns of the coarse images X_{l+1} = P_l^T X_l P_l of the extra blocks
// (packing couples, tf_add_K_triplets, DOF-binding merges), rebuilt on the
// host whenever the extra-block layout changes: per coarse extra block the
// list of triples (X_l block (J, I), P_l block (J, K), P_l block (I, M))
// whose products it sums.  The coarse operators then see the couplings the
// element graph does not have (e.g. between two surfaces pressed together).
tf_status amg_extra_symbolic(tf_handle* h) {
    Amg* a = h->amg;
    for (int l = 0; l < a->nlev; ++l) {
        AmgLevel& L = a->L[l];
        AmgSetup& S = a->S[l];
        void* ptrs[] = {S.xptr, S.xtrip, l > 0 ? L.xrow : nullptr, l > 0 ? L.xcol : nullptr,
                        l > 0 ? L.xval : nullptr};
        for (void* q : ptrs)
            if (q) cudaFree(q);
        S.xptr = S.xtrip = nullptr;
        if (l > 0) {
            L.xrow = L.xcol = nullptr;
            L.xval = nullptr;
            L.nx = 0;
        }
    }
    a->x_version = h->extra_version;
    if (h->d.nxb == 0 || h->h_xcols.empty()) return TF_OK;
    // level 0: (column, block index) per row, in the device layout
    std::vector<std::vector<std::pair<int, int>>> X(h->d.nn);
    for (int J = 0; J < h->d.nn; ++J)
        for (size_t q = 0; q < h->h_xcols[J].size(); ++q)
            X[J].emplace_back(h->h_xcols[J][q], h->h_xrow[J] + static_cast<int>(q));
    for (int l = 0; l + 1 < a->nlev; ++l) {
        const std::vector<int>& prow = a->h_prow[l];
        const std::vector<int>& pcol = a->h_pcol[l];
        const int nc = a->h_n[l + 1];
        struct Trip {
            int K, M, q, b1, b2;
        };
        std::vector<Trip> trips;
        for (size_t J = 0; J < X.size(); ++J)
            for (const auto& e : X[J])
                for (int b1 = prow[J]; b1 < prow[J + 1]; ++b1)
                    for (int b2 = prow[e.first]; b2 < prow[e.first + 1]; ++b2)
                        trips.push_back({pcol[b1], pcol[b2], e.second, b1, b2});
        if (trips.empty()) break;
        std::sort(trips.begin(), trips.end(), [](const Trip& u, const Trip& v) {
            return u.K != v.K ? u.K < v.K : (u.M != v.M ? u.M < v.M : u.q < v.q);
        });
        std::vector<int> xrow(nc + 1, 0), xcol, xptr(1, 0), xtrip;
        std::vector<std::vector<std::pair<int, int>>> Xn(nc);
        for (size_t t = 0; t < trips.size(); ++t) {
            const Trip& u = trips[t];
            if (t == 0 || u.K != trips[t - 1].K || u.M != trips[t - 1].M) {
                if (t > 0) xptr.push_back(static_cast<int>(xtrip.size() / 3));
                Xn[u.K].emplace_back(u.M, static_cast<int>(xcol.size()));
                xcol.push_back(u.M);
                xrow[u.K + 1]++;
            }
            xtrip.insert(xtrip.end(), {u.q, u.b1, u.b2});
        }
        xptr.push_back(static_cast<int>(xtrip.size() / 3));
        for (int K = 0; K < nc; ++K) xrow[K + 1] += xrow[K];
        AmgLevel& C = a->L[l + 1];
        AmgSetup& S = a->S[l];
        C.nx = static_cast<int64_t>(xcol.size());
        AMG_TRY(up(&C.xrow, xrow));
        AMG_TRY(up(&C.xcol, xcol));
        AMG_TRY(zeros(&C.xval, 36 * (size_t)C.nx));
        AMG_TRY(up(&S.xptr, xptr));
        AMG_TRY(up(&S.xtrip, xtrip));
        X.swap(Xn);
    }
    return TF_OK;
}

namespace {

__device__ __forceinline__ bool seg_stopped(const double* scal, int seg) {
    return __ldcg(&scal[(size_t)seg * S_COUNT + S_FLAG]) != 0.0;
}

// ... and of the instance of node i of a coarse level (one instance: no look-up)
__device__ __forceinline__ bool level_stopped(const AmgLevel& L, const double* scal, int i) {
    return seg_stopped(scal, L.single ? 0 : L.seg[i]);
}

// Sum of one value over the grid: partials per CTA, the last CTA to arrive
// folds them in a fixed order, all its threads at once (no waiting).  True in
// thread 0 of that CTA.
__device__ bool grid_sum(double v, double* part, unsigned* ticket, double* total) {
    __shared__ double sm[1][kT / 32 + 1];
    __shared__ bool last;
    double x[1] = {v};
    cta_sum<kT, 1>(x, sm);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = x[0];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double t[1] = {0.0};
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) t[0] += __ldcg(&part[b]);
    cta_sum<kT, 1>(t, sm);
    if (threadIdx.x != 0) return false;
    *total = t[0];
    *ticket = 0u;
    return true;
}

// Level-0 node of this thread (CTA tables of the node-parallel kernels).
struct Node0 {
    int i, seg;
    bool valid;
    int row;  // row of this thread's share of a row product (split CTAs: the lane's, whatever the warp)
};
__device__ __forceinline__ Node0 node0(const Device& d) {
    Node0 q;
    int n0, n1;
    if (d.nseg == 1) {
        q.seg = 0;
        n0 = blockIdx.x * d.cta_nodes;
        n1 = min(n0 + d.cta_nodes, d.nn);
    } else {
        q.seg = d.cta_seg[blockIdx.x];
        n0 = d.cta_node0[blockIdx.x];
        n1 = d.cta_node1[blockIdx.x];
    }
    q.i = n0 + threadIdx.x;
    q.valid = q.i < n1;
    q.row = d.split ? min(n0 + (int)(threadIdx.x & 31), n1 - 1) : q.i;
    return q;
}

__device__ __forceinline__ void mul3(const float* __restrict__ D, const float r[3], float z[3]) {
    z[0] = fmaf(D[0], r[0], fmaf(D[1], r[1], D[2] * r[2]));
    z[1] = fmaf(D[3], r[0], fmaf(D[4], r[1], D[5] * r[2]));
    z[2] = fmaf(D[6], r[0], fmaf(D[7], r[1], D[8] * r[2]));
}

// Row of S = D^-1 A (FP16, sliced) times x, FP32 sums: this thread's share of it
// (split CTAs), from the warp's slots s0 .. s1.
template <int U = 4>
__device__ __forceinline__ void row0_part(const Device& d, int s0, int s1, const __half* __restrict__ valh,
                                          const float* __restrict__ x, float (&y)[3], const Ahead& p = Ahead{}) {
    const int lane = threadIdx.x & 31;
    float y0 = 0.f, y1 = 0.f, y2 = 0.f;
    const int* __restrict__ col = d.scol + lane;
    const uint4* __restrict__ p8 = reinterpret_cast<const uint4*>(valh) + lane;
    const __half* __restrict__ p1 = valh + (size_t)(d.nval / kSlotDoubles) * (kSlice * 8) + lane;
    auto slot = [&](int s, int j) {
        if (!TF_IN(d.check, j, d.nn, CK_V0_COL)) return;
        const uint4 pk = __ldg(&p8[(size_t)s * kSlice]);
        const float a8 = __half2float(p1[(size_t)s * kSlice]);
        // the low half of each word is the even entry
        const float2 a01 = make_float2(__half2float(__ushort_as_half((unsigned short)(pk.x & 0xffffu))),
                                       __half2float(__ushort_as_half((unsigned short)(pk.x >> 16))));
        const float2 a23 = make_float2(__half2float(__ushort_as_half((unsigned short)(pk.y & 0xffffu))),
                                       __half2float(__ushort_as_half((unsigned short)(pk.y >> 16))));
        const float2 a45 = make_float2(__half2float(__ushort_as_half((unsigned short)(pk.z & 0xffffu))),
                                       __half2float(__ushort_as_half((unsigned short)(pk.z >> 16))));
        const float2 a67 = make_float2(__half2float(__ushort_as_half((unsigned short)(pk.w & 0xffffu))),
                                       __half2float(__ushort_as_half((unsigned short)(pk.w >> 16))));
        const float x0 = x[3 * j], x1 = x[3 * j + 1], x2 = x[3 * j + 2];
        y0 = fmaf(a01.x, x0, fmaf(a01.y, x1, fmaf(a23.x, x2, y0)));
        y1 = fmaf(a23.y, x0, fmaf(a45.x, x1, fmaf(a45.y, x2, y1)));
        y2 = fmaf(a67.x, x0, fmaf(a67.y, x1, fmaf(a8, x2, y2)));
    };
    if constexpr (U == 0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (p.j[u] >= 0) slot(s0 + u, p.j[u]);
    }
#pragma unroll (U == 0 ? 1 : U)
    for (int s = U == 0 ? s0 + kAhead : s0; s < s1; ++s) slot(s, __ldg(&col[(size_t)s * kSlice]));
    y[0] = y0;
    y[1] = y1;
    y[2] = y2;
}

// The whole row on its node's thread, the extra blocks X (FP64) entering as
// D^-1 (X x).  Every thread of the CTA calls it.
template <int U = 4>
__device__ __forceinline__ void row0s(const Device& d, const __half* __restrict__ valh,
                                      const float* __restrict__ dinv32, const float* __restrict__ x, const Node0& q0,
                                      float (&y)[3]) {
    const int wg = blockIdx.x * kWarps + (threadIdx.x >> 5), i = q0.i;
    const int s0 = __ldg(&d.wslot0[wg]), s1 = __ldg(&d.wslot0[wg + 1]);
    Ahead p;
    if constexpr (U == 0) p = load_ahead(d.scol, s0, s1);
    row0_part<U>(d, s0, s1, valh, x, y, p);
    if (d.split) split_sum(y);
    if (!d.xrow) return;
    if (d.split) {  // the warps share the rows' extra blocks as well, if the CTA has any
        const int n0 = i - (int)threadIdx.x;
        if (d.xrow[n0] == d.xrow[min(n0 + 32, d.nn)]) return;
    } else if (!q0.valid || d.xrow[i] == d.xrow[i + 1]) {
        return;
    }
    float e[3] = {0.f, 0.f, 0.f}, z[3];
    const int step = d.split ? kWarps : 1, x1 = d.xrow[q0.row + 1];
    for (int q = d.xrow[q0.row] + (d.split ? (int)(threadIdx.x >> 5) : 0); q < x1; q += step) {
        const int j = d.xcol[q];
        if (!TF_IN(d.check, j, d.nn, CK_EXTRA_COL)) continue;
        const double* __restrict__ v = d.xval + 9 * (size_t)q;
#pragma unroll
        for (int r = 0; r < 3; ++r)
            e[r] = fmaf((float)v[3 * r], x[3 * j],
                        fmaf((float)v[3 * r + 1], x[3 * j + 1], fmaf((float)v[3 * r + 2], x[3 * j + 2], e[r])));
    }
    if (d.split) {
        __syncthreads();  // split_sum's shared memory again
        split_sum(e);
        if (!q0.valid) return;
    }
    mul3(dinv32 + 9 * (size_t)i, e, z);
#pragma unroll
    for (int r = 0; r < 3; ++r) y[r] += z[r];
}

// Warp-cooperative product of row i of a 6x6-block CSR matrix with x.
// Lane 6 k + a (< 30) takes row a of blocks k, k + 5, k + 10, ... of the
// row: six FMAs per block row, every value used once (lane groups read
// 5 consecutive blocks); the five partial sums of each row a are then
// gathered by shuffles.  Every lane returns y.
__device__ __forceinline__ void row6_warp(const AmgLevel& L, int i, const float* __restrict__ x, float y[6]) {
    const int lane = threadIdx.x & 31;
    const int kb = lane / 6, a = lane - 6 * kb;
    float acc = 0.f;
    const int p0 = L.rowptr[i], p1 = L.rowptr[i + 1];
    if (lane < 30) {
#pragma unroll 2
        for (int p = p0 + kb; p < p1; p += 5) {
            const int j = __ldg(&L.colidx[p]);
            const float* __restrict__ v = L.val + 36 * (size_t)p + 6 * a;
            const float* __restrict__ xj = x + 6 * (size_t)j;
#pragma unroll
            for (int b2 = 0; b2 < 6; ++b2) acc = fmaf(__ldg(&v[b2]), xj[b2], acc);
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        float s2 = 0.f;
#pragma unroll
        for (int g = 0; g < 5; ++g) s2 += __shfl_sync(0xffffffffu, acc, 6 * g + k);
        y[k] = s2;
    }
    if (L.xrow)  // coarse image of the extra blocks (few; every lane adds them)
        for (int q = L.xrow[i]; q < L.xrow[i + 1]; ++q) {
            const float* __restrict__ v = L.xval + 36 * (size_t)q;
            const float* __restrict__ xj = x + 6 * (size_t)L.xcol[q];
#pragma unroll
            for (int k = 0; k < 6; ++k)
#pragma unroll
                for (int m = 0; m < 6; ++m) y[k] = fmaf(v[6 * k + m], xj[m], y[k]);
        }
}

// y_a = (S x)_a on lane a < 6 for a row of a 6-DOF level (blocks p0 .. p1), S =
// D^-1 A stored in FP16 (the element blocks only; extra6 adds the coarse image of
// the extra blocks).  Lane 6 k + a (< 30) takes row a of blocks k, k + 5, ...; the
// columns of up to 30 blocks are loaded before the first is used, so a row costs
// three dependent loads (range, columns, values) however long it is (two blocks
// per lane at a time: 7.5 against 6.6 us per sweep of the 8,978-node level); they
// precede the wait for the kernel before (row6_load), which leaves x's.
struct Row6 {  // what of a row does not change during a solve, loaded ahead
    int p0, p1, j[6];
    __half2 v[6][3];
};
__device__ __forceinline__ Row6 row6_load(const AmgLevel& L, int i) {
    Row6 R;
    const int lane = threadIdx.x & 31;
    const int kb = lane / 6, a = lane - 6 * kb;
    R.p0 = __ldg(&L.rowptr[i]);
    R.p1 = __ldg(&L.rowptr[i + 1]);
#pragma unroll
    for (int u = 0; u < 6; ++u) {
        const int p = R.p0 + kb + 5 * u;
        R.j[u] = -1;
        if (lane >= 30 || p >= R.p1) continue;
        R.j[u] = __ldg(&L.colidx[p]);
        const __half2* __restrict__ v = reinterpret_cast<const __half2*>(L.valh + 36 * (size_t)p + 6 * a);
#pragma unroll
        for (int b = 0; b < 3; ++b) R.v[u][b] = __ldg(&v[b]);
    }
    return R;
}
__device__ __forceinline__ float row6_warp_h(const AmgLevel& L, const Row6& R, const float* __restrict__ x) {
    const int lane = threadIdx.x & 31;
    const int kb = lane / 6, a = lane - 6 * kb;
    float acc = 0.f;
#pragma unroll
    for (int u = 0; u < 6; ++u) {
        if (R.j[u] < 0) continue;
        const float2* __restrict__ xj = reinterpret_cast<const float2*>(x + 6 * (size_t)R.j[u]);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const float2 f = __half22float2(R.v[u][b]), w = xj[b];
            acc = fmaf(f.x, w.x, fmaf(f.y, w.y, acc));
        }
    }
    if (lane < 30)
        for (int p = R.p0 + kb + 30; p < R.p1; p += 5) {
            const float2* __restrict__ xj = reinterpret_cast<const float2*>(x + 6 * (size_t)__ldg(&L.colidx[p]));
            const __half2* __restrict__ v = reinterpret_cast<const __half2*>(L.valh + 36 * (size_t)p + 6 * a);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const float2 f = __half22float2(__ldg(&v[b])), w = xj[b];
                acc = fmaf(f.x, w.x, fmaf(f.y, w.y, acc));
            }
        }
    float y = acc;
#pragma unroll
    for (int g = 1; g < 5; ++g) y += __shfl_down_sync(0xffffffffu, acc, 6 * g);
    return y;
}

// e = X x for row i, the coarse image of the extra blocks, on every lane: five
// blocks at a time, lane 6 k + a row a of block k (every lane all of a block: 9.4
// against 4.7 us per sweep of 722 nodes in contact)
__device__ __forceinline__ void extra6(const AmgLevel& L, int i, const float* __restrict__ x, float e[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) e[k] = 0.f;
    if (!L.xrow) return;
    const int q0 = L.xrow[i], q1 = L.xrow[i + 1];
    if (q0 == q1) return;
    const int lane = threadIdx.x & 31;
    const int kb = lane / 6, a = lane - 6 * kb;
    float acc = 0.f;
    if (lane < 30)
#pragma unroll 2
        for (int q = q0 + kb; q < q1; q += 5) {
            const float2* __restrict__ v = reinterpret_cast<const float2*>(L.xval + 36 * (size_t)q + 6 * a);
            const float2* __restrict__ xj = reinterpret_cast<const float2*>(x + 6 * (size_t)L.xcol[q]);
#pragma unroll
            for (int b = 0; b < 3; ++b) acc = fmaf(v[b].x, xj[b].x, fmaf(v[b].y, xj[b].y, acc));
        }
    float s = acc;
#pragma unroll
    for (int g = 1; g < 5; ++g) s += __shfl_down_sync(0xffffffffu, acc, 6 * g);
#pragma unroll
    for (int k = 0; k < 6; ++k) e[k] = __shfl_sync(0xffffffffu, s, k);
}

// r[a] without dynamic register indexing (which would go to local memory).
__device__ __forceinline__ float pick6(const float r[6], int a) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) v = (k == a) ? r[k] : v;
    return v;
}

// Lane a < 6 of the warp: (D r)_a for the 6x6 block D (r known to all lanes).
__device__ __forceinline__ float lane_mul6(const float* __restrict__ D, const float r[6], int a) {
    float s = 0.f;
#pragma unroll
    for (int b = 0; b < 6; ++b) s = fmaf(__ldg(&D[6 * a + b]), r[b], s);
    return s;
}

// ---- numeric phase -----------------------------------------------------------

__global__ void k_to_f32(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        b[k] = (float)a[k];
}

__global__ void k_f32_to_h(int64_t n, const float* __restrict__ a, __half* __restrict__ b) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
        b[k] = __float2half_rn(a[k]);
}

// S = D^-1 A of a 6-DOF level in FP16, one thread per block row
__global__ void k_to_h6(AmgLevel L) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= L.nnzb * 6) return;
    const int64_t p = gid / 6;
    const int k = (int)(gid - 6 * p);
    const float* __restrict__ Di = L.dinv + 36 * (size_t)L.rowof[p] + 6 * k;
    const float* __restrict__ A = L.val + 36 * (size_t)p;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        float v = 0.f;
#pragma unroll
        for (int m = 0; m < 6; ++m) v = fmaf(Di[m], A[6 * m + c], v);
        L.valh[36 * (size_t)p + 6 * k + c] = __float2half_rn(v);
    }
}

// S = D^-1 A for the smoother, block by block in the sliced layout, FP16
// (its entries are O(1): the FP16 range and 11-bit mantissa suffice for a
// preconditioner; the Krylov operator itself stays FP64).
__global__ void k_to_h(Device d, const float* __restrict__ val32, const float* __restrict__ dinv32,
                       __half* __restrict__ valh, float* __restrict__ diag32) {
    const Node0 q = node0(d);
    const int lane = threadIdx.x & 31;
    const int wg = blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int s0 = d.wslot0[wg], s1 = d.wslot0[wg + 1];
    float D[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) D[k] = (d.split || q.valid) ? dinv32[9 * (size_t)q.row + k] : 0.f;
    if (q.valid) {
        const float* __restrict__ Dg = val32 + d.diag[q.i];
#pragma unroll
        for (int k = 0; k < 9; ++k) diag32[9 * (size_t)q.i + k] = Dg[kSlice * k];
    }
    uint4* __restrict__ p8 = reinterpret_cast<uint4*>(valh) + lane;
    __half* __restrict__ p1 = valh + (size_t)(d.nval / kSlotDoubles) * (kSlice * 8) + lane;
    for (int s = s0; s < s1; ++s) {
        const size_t base = (size_t)s * kSlotDoubles + lane;
        float A[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) A[k] = val32[base + 32 * k];
        __half h[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                h[3 * r + c] =
                    __float2half_rn(fmaf(D[3 * r], A[c], fmaf(D[3 * r + 1], A[3 + c], D[3 * r + 2] * A[6 + c])));
        uint4 pk;
        pk.x = (uint32_t)__half_as_ushort(h[0]) | ((uint32_t)__half_as_ushort(h[1]) << 16);
        pk.y = (uint32_t)__half_as_ushort(h[2]) | ((uint32_t)__half_as_ushort(h[3]) << 16);
        pk.z = (uint32_t)__half_as_ushort(h[4]) | ((uint32_t)__half_as_ushort(h[5]) << 16);
        pk.w = (uint32_t)__half_as_ushort(h[6]) | ((uint32_t)__half_as_ushort(h[7]) << 16);
        p8[(size_t)s * kSlice] = pk;
        p1[(size_t)s * kSlice] = h[8];
    }
}

// Element (r, c) of fine-matrix block b: level 0 reads the FP32 copy of the
// sliced storage, coarser levels their 6x6 CSR blocks.
template <int BS, bool L0>
__device__ __forceinline__ const float* fine_block(const AmgLevel& F, const int* __restrict__ bofs0,
                                                   const float* __restrict__ val0, int b) {
    return L0 ? val0 + __ldg(&bofs0[b]) : F.val + 36 * (size_t)b;
}
template <int BS, bool L0>
__device__ __forceinline__ float fine_at(const float* blk, int r, int c) {
    return L0 ? __ldg(&blk[kSlice * (3 * r + c)]) : __ldg(&blk[6 * r + c]);
}

// Prolongator block b = (i, J): P_t(i) [agg(i) = J] - omega D_i^-1 sum over
// the fine blocks (i, j) with agg(j) = J of A_ij P_t(j).  One thread per
// block; plain aggregation has empty lists and omega 0 (a copy of P_t).
template <int BS, bool L0>
__global__ void k_smooth_p(AmgLevel F, AmgSetup S, const double* __restrict__ omega, int smooth,
                           const int* __restrict__ colidx0, const int* __restrict__ bofs0,
                           const float* __restrict__ val0, const float* __restrict__ dinv0) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= F.npb) return;
    const int i = S.pbrow[b], J = F.pcol[b];
    float W[BS][6];
#pragma unroll
    for (int r = 0; r < BS; ++r)
#pragma unroll
        for (int c = 0; c < 6; ++c) W[r][c] = 0.f;
    for (int q = S.sptr[b]; q < S.sptr[b + 1]; ++q) {
        const int ab = __ldg(&S.slist[q]);
        const int j = L0 ? __ldg(&colidx0[ab]) : __ldg(&F.colidx[ab]);
        const float* blk = fine_block<BS, L0>(F, bofs0, val0, ab);
        const float* __restrict__ Pj = S.Pt + (size_t)j * BS * 6;
#pragma unroll
        for (int m = 0; m < BS; ++m) {
            float pm[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) pm[c] = __ldg(&Pj[6 * m + c]);
#pragma unroll
            for (int r = 0; r < BS; ++r) {
                const float av = fine_at<BS, L0>(blk, r, m);
#pragma unroll
                for (int c = 0; c < 6; ++c) W[r][c] = fmaf(av, pm[c], W[r][c]);
            }
        }
    }
    const float om = smooth ? (float)__ldg(omega) : 0.f;
    const bool own = __ldg(&S.agg[i]) == J;
    const float* __restrict__ Di = L0 ? dinv0 + 9 * (size_t)i : F.dinv + 36 * (size_t)i;
    const float* __restrict__ Pi = S.Pt + (size_t)i * BS * 6;
    float* __restrict__ out = F.Pv + (size_t)b * BS * 6;
#pragma unroll
    for (int r = 0; r < BS; ++r)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            float s = 0.f;
#pragma unroll
            for (int m = 0; m < BS; ++m) s = fmaf(__ldg(&Di[BS * r + m]), W[m][c], s);
            out[6 * r + c] = fmaf(-om, s, own ? __ldg(&Pi[6 * r + c]) : 0.f);
        }
}

// The prolongator blocks in coarse-column order (for the restriction).
__global__ void k_p_columns(AmgLevel F, AmgSetup S, int bsz) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= F.npb * bsz) return;
    const int64_t q = k / bsz;
    F.Pc[k] = F.Pv[(size_t)__ldg(&S.cperm[q]) * bsz + (k - q * bsz)];
}

// T = A P, row r of T block t = (i, J): sum over its pairs (A_ij, P_jJ).
template <int BS, bool L0>
__global__ void k_ap(AmgLevel F, AmgSetup S, const int* __restrict__ bofs0, const float* __restrict__ val0) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= S.nT * BS) return;
    const int64_t t = gid / BS;
    const int r = static_cast<int>(gid - BS * t);
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int q = S.tptr[t]; q < S.tptr[t + 1]; ++q) {
        const float* blk = fine_block<BS, L0>(F, bofs0, val0, __ldg(&S.ta[q]));
        const float* __restrict__ Pb = F.Pv + (size_t)__ldg(&S.tb[q]) * BS * 6;
#pragma unroll
        for (int m = 0; m < BS; ++m) {
            const float av = fine_at<BS, L0>(blk, r, m);
#pragma unroll
            for (int c = 0; c < 6; ++c) acc[c] = fmaf(av, __ldg(&Pb[6 * m + c]), acc[c]);
        }
    }
    float* out = S.T + (size_t)t * BS * 6 + 6 * r;
#pragma unroll
    for (int c = 0; c < 6; ++c) out[c] = acc[c];
}

// Q = (I - omega S) P in its two layouts, one thread per block (i, J):
// P_iJ - omega D_i^-1 T_iJ.
__global__ void k_make_q(AmgQ Q, AmgSetup S, const float* __restrict__ Pv, const float* __restrict__ dinv,
                         const double* __restrict__ omega) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S.nT) return;
    const int i = S.trow[t], b = Q.tp[t];
    const float om = (float)__ldg(omega);
    const float* __restrict__ T = S.T + 18 * (size_t)t;
    const float* __restrict__ D = dinv + 9 * (size_t)i;
    float v[18];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const float s = fmaf(__ldg(&D[3 * r]), __ldg(&T[c]),
                                 fmaf(__ldg(&D[3 * r + 1]), __ldg(&T[6 + c]), __ldg(&D[3 * r + 2]) * __ldg(&T[12 + c])));
            v[6 * r + c] = fmaf(-om, s, b >= 0 ? __ldg(&Pv[18 * (size_t)b + 6 * r + c]) : 0.f);
        }
    uint32_t w[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
        w[k] = (uint32_t)__half_as_ushort(__float2half_rn(v[2 * k])) |
               ((uint32_t)__half_as_ushort(__float2half_rn(v[2 * k + 1])) << 16);
    const int p = Q.pos[t], lane = p & 31;
    const size_t s = (size_t)(p >> 5);
    Q.v16[64 * s + lane] = make_uint4(w[0], w[1], w[2], w[3]);
    Q.v16[64 * s + 32 + lane] = make_uint4(w[4], w[5], w[6], w[7]);
    Q.v2[32 * s + lane] = w[8];
    uint32_t* __restrict__ o = Q.cval + 9 * (size_t)Q.cpos[t];
#pragma unroll
    for (int k = 0; k < 9; ++k) o[k] = w[k];
}

// Coarse block c = (I, J), row p: sum over its pairs (P_iI, T_iJ) of
// (P_iI^T T_iJ)(p, :).
template <int BS>
__global__ void k_ptap(AmgLevel F, AmgSetup S, AmgLevel C) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= C.nnzb * 6) return;
    const int64_t c = gid / 6;
    const int p = static_cast<int>(gid - 6 * c);
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int q = S.gptr[c]; q < S.gptr[c + 1]; ++q) {
        const float* __restrict__ Pb = F.Pv + (size_t)__ldg(&S.gp[q]) * BS * 6;
        const float* __restrict__ Tb = S.T + (size_t)__ldg(&S.gt[q]) * BS * 6;
#pragma unroll
        for (int k = 0; k < BS; ++k) {
            const float pk = __ldg(&Pb[6 * k + p]);
#pragma unroll
            for (int c2 = 0; c2 < 6; ++c2) acc[c2] = fmaf(pk, __ldg(&Tb[6 * k + c2]), acc[c2]);
        }
    }
    const int I = C.rowof[c];
    if (C.colidx[c] == I && C.dead[6 * I + p]) acc[p] = 1.f;  // dropped coarse DOF: unit diagonal
    float* out = C.val + 36 * (size_t)c + 6 * p;
#pragma unroll
    for (int q2 = 0; q2 < 6; ++q2) out[q2] = acc[q2];
}

// Coarse extra block c = (K, M), row p: sum over its triples (X_JI, P_JK,
// P_IM) of (P_JK^T X_JI P_IM)(p, :).  Level 0's extra blocks are the FP64
// 3x3 blocks of the Krylov operator.
template <int BS, bool L0>
__global__ void k_xgal(AmgLevel F, AmgSetup S, AmgLevel C, const double* __restrict__ x0) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= C.nx * 6) return;
    const int64_t c = gid / 6;
    const int p = static_cast<int>(gid - 6 * c);
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int t = S.xptr[c]; t < S.xptr[c + 1]; ++t) {
        const int q = __ldg(&S.xtrip[3 * t]);
        const float* __restrict__ P1 = F.Pv + (size_t)__ldg(&S.xtrip[3 * t + 1]) * BS * 6;
        const float* __restrict__ P2 = F.Pv + (size_t)__ldg(&S.xtrip[3 * t + 2]) * BS * 6;
#pragma unroll
        for (int r = 0; r < BS; ++r) {
            const float pr = __ldg(&P1[6 * r + p]);
#pragma unroll
            for (int s2 = 0; s2 < BS; ++s2) {
                const float xv = L0 ? (float)__ldg(&x0[9 * (size_t)q + 3 * r + s2])
                                    : __ldg(&F.xval[36 * (size_t)q + 6 * r + s2]);
                const float px = pr * xv;
#pragma unroll
                for (int m = 0; m < 6; ++m) acc[m] = fmaf(px, __ldg(&P2[6 * s2 + m]), acc[m]);
            }
        }
    }
    float* out = C.xval + 36 * (size_t)c + 6 * p;
#pragma unroll
    for (int m = 0; m < 6; ++m) out[m] = acc[m];
}

// Inverse of a 6x6 block by Gauss-Jordan with partial pivoting (FP64 work).
__device__ void inv6(const float* __restrict__ A, float* __restrict__ out) {
    double M[6][12];
#pragma unroll
    for (int a = 0; a < 6; ++a)
#pragma unroll
        for (int b = 0; b < 6; ++b) {
            M[a][b] = A[6 * a + b];
            M[a][6 + b] = a == b ? 1.0 : 0.0;
        }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        int piv = k;
        double best = fabs(M[k][k]);
#pragma unroll
        for (int r = k + 1; r < 6; ++r)
            if (fabs(M[r][k]) > best) {
                best = fabs(M[r][k]);
                piv = r;
            }
        if (piv != k)
#pragma unroll
            for (int c = 0; c < 12; ++c) {
                const double tmp = M[k][c];
                M[k][c] = M[piv][c];
                M[piv][c] = tmp;
            }
        const double dk = M[k][k];
        const double rinv = dk != 0.0 ? 1.0 / dk : 1.0;
#pragma unroll
        for (int c = 0; c < 12; ++c) M[k][c] *= rinv;
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            if (r == k) continue;
            const double f = M[r][k];
#pragma unroll
            for (int c = 0; c < 12; ++c) M[r][c] = fma(-f, M[k][c], M[r][c]);
        }
    }
#pragma unroll
    for (int a = 0; a < 6; ++a)
#pragma unroll
        for (int b = 0; b < 6; ++b) out[6 * a + b] = (float)M[a][6 + b];
}

__global__ void k_inv6(AmgLevel L) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L.n) return;
    inv6(L.val + 36 * (size_t)L.diag[i], L.dinv + 36 * (size_t)i);
}

// power iteration for lambda_max(D^-1 A): v0 deterministic, scale = 1/|v0|
__global__ void k_pw_init(int64_t m, float* __restrict__ v, double* part, unsigned* ticket, double* scal) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    if (k < m) {
        unsigned h = static_cast<unsigned>(k) * 2654435761u + 12345u;
        h ^= h >> 13;
        h *= 0x5bd1e995u;
        h ^= h >> 15;
        // zero-mean pseudo-random values: every mode, the rough ones included,
        // is present from the start (a positive vector barely excites the
        // largest eigenvalues, which would be underestimated)
        const float x = (h & 0xffffu) / 65536.0f - 0.5f;
        v[k] = x;
        s = (double)x * x;
    }
    double tot;
    if (grid_sum(s, part, ticket, &tot)) scal[0] = 1.0 / sqrt(tot);
}

__device__ __forceinline__ void pw_finish(double tot, double* scal, double* omega, double* level0 = nullptr) {
    const double lam = sqrt(tot);
    scal[0] = lam > 0.0 ? 1.0 / lam : 1.0;
    scal[1] = lam;
    // 5 % margin: the power iteration approaches lambda_max from below
    *omega = lam > 0.0 ? (4.0 / 3.0) / (1.05 * lam) : 1.0;
    if (level0) *level0 = kLevel0Weight * *omega;
}

__global__ void k_pw_step0(Device d, const __half* __restrict__ valh, const float* __restrict__ dinv32,
                           const float* __restrict__ v, float* __restrict__ w, double* part, unsigned* ticket,
                           double* scal, double* omega, double* level0) {
    const Node0 q = node0(d);
    double s = 0.0;
    float y[3] = {0.f, 0.f, 0.f};
    row0s(d, valh, dinv32, v, q, y);  // D^-1 A v = S v, the smoother's operator
    if (q.valid) {
        const float sc = (float)__ldcg(&scal[0]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float z = sc * y[k];
            w[3 * q.i + k] = z;
            s += (double)z * z;
        }
    }
    double tot;
    if (grid_sum(s, part, ticket, &tot)) pw_finish(tot, scal, omega, level0);
}

__global__ void k_pw_step6(AmgLevel L, const float* __restrict__ v, float* __restrict__ w, double* part,
                           unsigned* ticket, double* scal, double* omega) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // one warp per row
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    if (i < L.n) {
        float y[6];
        row6_warp(L, i, v, y);
        const float sc = (float)__ldcg(&scal[0]);
#pragma unroll
        for (int k = 0; k < 6; ++k) y[k] *= sc;
        if (lane < 6) {
            const float z = lane_mul6(L.dinv + 36 * (size_t)i, y, lane);
            w[6 * i + lane] = z;
            s = (double)z * z;
        }
    }
    double tot;
    if (grid_sum(s, part, ticket, &tot)) pw_finish(tot, scal, omega);
}

// Gauss-Jordan inverse of the coarsest matrix of each instance, in place
// (one CTA each, FP64 work, FP32 result).  Bound by the m^2 FP64 updates of
// each of the m steps on one SM (m <= 96: 0.2 ms); the pivot is found by one
// warp.  1.26 -> 0.3 ms at m = 90 against an m x 2m form with a serial pivot
// search.
__global__ void __launch_bounds__(kInvThreads) k_coarse_invert(AmgLevel L, const int* __restrict__ cnode0,
                                                               const int* __restrict__ cinv0,
                                                               float* __restrict__ cinv) {
    extern __shared__ double M[];  // m x m
    __shared__ double f[kCoarseDofs], prow[kCoarseDofs];
    __shared__ int swapped[kCoarseDofs];  // row exchanged with row k at step k
    __shared__ int piv;
    __shared__ double tiny, pval;
    const int g = blockIdx.x;
    const int n0 = cnode0[g], n1 = cnode0[g + 1];
    const int m = 6 * (n1 - n0);
    if (m == 0) return;
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < m * m; k += blockDim.x) M[k] = 0.0;
    __syncthreads();
    for (int I = n0 + threadIdx.x; I < n1; I += blockDim.x) {
        for (int p = L.rowptr[I]; p < L.rowptr[I + 1]; ++p) {
            const int J = L.colidx[p] - n0;
            const float* v = L.val + 36 * (size_t)p;
            for (int a = 0; a < 6; ++a)
                for (int b = 0; b < 6; ++b) M[(6 * (I - n0) + a) * m + 6 * J + b] = (double)v[6 * a + b];
        }
        if (L.xrow)
            for (int q = L.xrow[I]; q < L.xrow[I + 1]; ++q) {
                const int J = L.xcol[q] - n0;
                if (J < 0 || J >= n1 - n0) continue;  // couples another instance: outside this inverse
                const float* v = L.xval + 36 * (size_t)q;
                for (int a = 0; a < 6; ++a)
                    for (int b = 0; b < 6; ++b) M[(6 * (I - n0) + a) * m + 6 * J + b] += (double)v[6 * a + b];
            }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        double dmax = 0.0;
        for (int r = lane; r < m; r += 32) dmax = fmax(dmax, fabs(M[r * m + r]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        if (lane == 0) tiny = 1e-12 * dmax;
    }
    __syncthreads();
    for (int k = 0; k < m; ++k) {
        if (threadIdx.x < 32) {  // the largest entry of column k from row k down, the first of equal ones
            double bv = -1.0;
            int best = m;
            for (int r = k + lane; r < m; r += 32) {
                const double v = fabs(M[r * m + k]);
                if (v > bv) {
                    bv = v;
                    best = r;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int ob = __shfl_xor_sync(0xffffffffu, best, o);
                if (ov > bv || (ov == bv && ob < best)) {
                    bv = ov;
                    best = ob;
                }
            }
            if (lane == 0) {
                piv = bv > tiny ? best : -1;
                swapped[k] = bv > tiny ? best : k;
                pval = bv > tiny ? M[best * m + k] : 0.0;
            }
        }
        __syncthreads();
        const int pr = piv;
        if (pr < 0) {
            // (numerically) singular direction, e.g. a free rigid mode of an
            // unconstrained sheet: no coarse correction along it
            for (int c = threadIdx.x; c < m; c += blockDim.x) M[k * m + c] = M[c * m + k] = 0.0;
            __syncthreads();
            continue;
        }
        // the pivot row scaled (unit column in place of column k), the rest of
        // column k as the multipliers
        const double rinv = 1.0 / pval;
        for (int c = threadIdx.x; c < m; c += blockDim.x) {
            const double v = M[pr * m + c];
            if (pr != k) M[pr * m + c] = M[k * m + c];
            prow[c] = (c == k ? 1.0 : v) * rinv;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < m; r += blockDim.x) {
            f[r] = r == k ? 0.0 : M[r * m + k];
            if (r != k) M[r * m + k] = 0.0;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < m * m; q += blockDim.x) {
            const int r = q / m, c = q - r * m;
            M[q] = r == k ? prow[c] : fma(-f[r], prow[c], M[q]);
        }
        __syncthreads();
    }
    // the row exchanges of A are column exchanges of its inverse, last first
    for (int k = m - 1; k >= 0; --k) {
        const int pr = swapped[k];
        if (pr == k) continue;
        for (int r = threadIdx.x; r < m; r += blockDim.x) {
            const double tmp = M[r * m + k];
            M[r * m + k] = M[r * m + pr];
            M[r * m + pr] = tmp;
        }
        __syncthreads();
    }
    float* out = cinv + cinv0[g];
    for (int q = threadIdx.x; q < m * m; q += blockDim.x) out[q] = (float)M[q];
}

// ---- V-cycle (FP32) -------------------------------------------------------------

struct V0 {  // level-0 operands
    Device d;
    const double* omega;
    const float* dinv32;  // FP32 copy of the block inverses
    const __half* valh;   // S = D^-1 A, FP16
    const float* diag32;  // diagonal blocks D, FP32 [9 n]
};

// The level-0 part of a V-cycle: pre-sweep from zero x = omega D^-1 r, residual
// t = r - A x, coarse correction x += P e, post-sweep x += omega D^-1 (r - A x).
// With S = D^-1 A and z = omega D^-1 r the result is
//     (2 z - omega S z) + Q e,   Q = (I - omega S) P,
// and the restricted residual P^T (r - A z) is Q^T r for a symmetric A (the
// viscous tangent's asymmetry, of the order of eta |grad v| / E, only changes
// the preconditioner).  So the smoother's matrix is read once instead of twice,
// and that product does not wait for the coarse levels: k_restrict with Q (Q^T r),
// the coarse levels, k_q_post; k_q_smooth runs beside the coarse levels where
// those are a chain of launches, and is part of k_q_post where they are one
// dense product.  Bound by reading S (66 MB at 320,000 prisms) and Q twice (52 MB
// each): 77 us of kernels before (pre, residual, restriction, prolongation,
// post), 19 + 14 us now with 16 us beside the coarse levels; 32.3 -> 30.3 ms per
// 320,000-prism step, 46.6 -> 38.2 ms per step of 32 batched tissues.  Systems
// with extra blocks (packing couples, added entries) keep the kernels that apply
// the current matrix: k_v0_resid .. k_v0_post below.

// r_C(I) = sum over the blocks (i, I) of P_iI^T t_i (of Q for the folded level-0
// transfer) and, with presmooth (the sweep's weight), the coarse level's first sweep
// x_C = presmooth omega_C D_C^-1 r_C.  One CTA of kRestrictThreads per coarse node, its threads striding over the
// (block, row) pairs of the column, stored contiguously (one warp per node: 7.5
// against 6.0 us from 8,978 to 391 nodes).  V: __half or float values, 6 per pair.
template <int BS, class V>
__global__ void __launch_bounds__(kRestrictThreads) k_restrict(const int* __restrict__ cptr,
                                                               const int* __restrict__ crow,
                                                               const V* __restrict__ val, AmgLevel C, int nf, int* check,
                                                               const float* __restrict__ t,
                                                               const double* __restrict__ scal,
                                                               const double* __restrict__ omegaC, float presmooth) {
    __shared__ float sm[kRestrictThreads / 32][6];
    const int I = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q0 = __ldg(&cptr[I]), np = BS * (__ldg(&cptr[I + 1]) - q0);
    pdl_enter();
    pdl_next();
    if (level_stopped(C, scal, I)) return;
    float rc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int q = threadIdx.x; q < np; q += kRestrictThreads) {
        const int m = q / BS, k = q - BS * m;
        const int i = __ldg(&crow[q0 + m]);
        if (!TF_IN(check, i, nf, CK_RESTRICT_ROW)) continue;
        const float tk = t[BS * (size_t)i + k];
        const V* __restrict__ P = val + 6 * ((size_t)BS * q0 + q);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            float2 f;
            if constexpr (sizeof(V) == 2) f = __half22float2(__ldg(reinterpret_cast<const __half2*>(P) + b));
            else f = __ldg(reinterpret_cast<const float2*>(P) + b);
            rc[2 * b] = fmaf(f.x, tk, rc[2 * b]);
            rc[2 * b + 1] = fmaf(f.y, tk, rc[2 * b + 1]);
        }
    }
#pragma unroll
    for (int b = 0; b < 6; ++b)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rc[b] += __shfl_xor_sync(0xffffffffu, rc[b], o);
    if (lane < 6) sm[warp][lane] = pick6(rc, lane);
    __syncthreads();
    if (warp > 0) return;
#pragma unroll
    for (int b = 0; b < 6; ++b) {
        rc[b] = 0.f;
#pragma unroll
        for (int w = 0; w < kRestrictThreads / 32; ++w) rc[b] += sm[w][b];
    }
    if (lane < 6) {
        C.r[6 * I + lane] = pick6(rc, lane);
        if (presmooth != 0.f)
            C.x[6 * I + lane] = presmooth * (float)__ldg(omegaC) * lane_mul6(C.dinv + 36 * (size_t)I, rc, lane);
    }
}

// x = 2 z - omega S z
template <int U>
__global__ void k_q_smooth(V0 a, const float* __restrict__ z, float* __restrict__ x) {
    pdl_enter();
    const Node0 q = node0(a.d);
    if (seg_stopped(a.d.scal, q.seg)) return;
    float y[3];
    row0s<U>(a.d, a.valh, a.dinv32, z, q, y);
    if (!q.valid) return;
    const float om = (float)__ldg(a.omega);
#pragma unroll
    for (int k = 0; k < 3; ++k) x[3 * q.i + k] = fmaf(-om, y[k], 2.f * z[3 * q.i + k]);
}

// (Q e)_i added to x: the warp's slots s0 .. s1
__device__ __forceinline__ void row_q(const AmgQ& Q, int s0, int s1, const float* __restrict__ e, int nc, int* check,
                                      float (&x)[3], const Ahead* p) {
    const int lane = threadIdx.x & 31;
    auto slot = [&](int s, int J) {
        if (!TF_IN(check, J, nc, CK_PROLONG_COL)) return;
        const uint4 a = __ldg(&Q.v16[64 * (size_t)s + lane]), b = __ldg(&Q.v16[64 * (size_t)s + 32 + lane]);
        const uint32_t c = __ldg(&Q.v2[32 * (size_t)s + lane]);
        const float2* __restrict__ ej = reinterpret_cast<const float2*>(e + 6 * (size_t)J);
        const float2 e0 = ej[0], e1 = ej[1], e2 = ej[2];
        const uint32_t w[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&w[3 * k]));
            const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&w[3 * k + 1]));
            const float2 f2 = __half22float2(*reinterpret_cast<const __half2*>(&w[3 * k + 2]));
            x[k] = fmaf(f0.x, e0.x, fmaf(f0.y, e0.y, fmaf(f1.x, e1.x, fmaf(f1.y, e1.y,
                   fmaf(f2.x, e2.x, fmaf(f2.y, e2.y, x[k]))))));
        }
    };
    if (p)
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (p->j[u] >= 0) slot(s0 + u, p->j[u]);
#pragma unroll 4
    for (int s = p ? s0 + kAhead : s0; s < s1; ++s) slot(s, __ldg(&Q.col[32 * (size_t)s + lane]));
}

// out = x + Q e, x = 2 z - omega S z read from k_q_smooth (SMOOTH: formed here
// from z), as the FP64 preconditioned vector.  DOT: with (r, out) and CG's beta
// (start: the first of a solve, which also sets p = out).
template <int U, bool SMOOTH, bool DOT>
__global__ void k_q_post(V0 a, Ctx c, AmgQ Q, int nc, const float* __restrict__ zx, const float* __restrict__ e,
                         double* __restrict__ out, const double* __restrict__ r, double* __restrict__ p, int start) {
    // before the wait: what does not change during a solve
    const Node0 q = node0(a.d);
    const int wg = blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int q0 = __ldg(&Q.slot0[wg]), q1 = __ldg(&Q.slot0[wg + 1]);
    const float om = SMOOTH ? (float)__ldg(a.omega) : 0.f;
    int s0 = 0, s1 = 0;
    Ahead ps, pq;
    if constexpr (SMOOTH) {
        s0 = __ldg(&a.d.wslot0[wg]);
        s1 = __ldg(&a.d.wslot0[wg + 1]);
        if constexpr (U == 0) ps = load_ahead(a.d.scol, s0, s1);
    }
    if constexpr (U == 0) pq = load_ahead(Q.col, q0, q1);
    pdl_enter();
    if (__ldcg(&a.d.scal[(size_t)q.seg * S_COUNT + S_FLAG]) != 0.0) return;
    float x[3] = {0.f, 0.f, 0.f}, own[3];
    double ri[3];
    if constexpr (SMOOTH) {
        row0_part<U>(a.d, s0, s1, a.valh, zx, x, ps);
#pragma unroll
        for (int k = 0; k < 3; ++k) x[k] *= -om;
    }
    row_q(Q, q0, q1, e, nc, a.d.check, x, U == 0 ? &pq : nullptr);
    if (q.valid)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            own[k] = (SMOOTH ? 2.f : 1.f) * zx[3 * q.i + k];
            if constexpr (DOT) ri[k] = r[3 * q.i + k];
        }
    if (a.d.split) split_sum(x);
    double v[1] = {0.0};
    if (q.valid) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double o = (double)(own[k] + x[k]);
            out[3 * q.i + k] = o;
            if constexpr (DOT) {
                if (start) p[3 * q.i + k] = o;
                v[0] = fma(ri[k], o, v[0]);
            }
        }
    }
    if constexpr (DOT) {
        double tot[1];
        if (reduce_seg<1>(c, q.seg, v, tot) && threadIdx.x == 0)
            cg_rz(a.d.scal + (size_t)q.seg * S_COUNT, tot[0], start != 0);
    }
}

// t = r - A x
template <int U>
__global__ void k_v0_resid(V0 a, const double* __restrict__ r, const float* __restrict__ x, float* __restrict__ t) {
    pdl_enter();
    const Node0 q = node0(a.d);
    if (seg_stopped(a.d.scal, q.seg)) return;
    float y[3];
    row0s<U>(a.d, a.valh, a.dinv32, x, q, y);
    if (!q.valid) return;
    // A x = D (S x), D the diagonal block
    const float* __restrict__ Dg = a.diag32 + 9 * (size_t)q.i;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        t[3 * q.i + k] = (float)r[3 * q.i + k] - fmaf(__ldg(&Dg[3 * k]), y[0],
                                                      fmaf(__ldg(&Dg[3 * k + 1]), y[1], __ldg(&Dg[3 * k + 2]) * y[2]));
}

// out = x + omega D^-1 (r - A x), written back as the FP64 preconditioned vector
template <int U>
__global__ void k_v0_post(V0 a, const double* __restrict__ r, const float* __restrict__ x, double* __restrict__ out) {
    pdl_enter();
    const Node0 q = node0(a.d);
    if (seg_stopped(a.d.scal, q.seg)) return;
    float y[3];
    row0s<U>(a.d, a.valh, a.dinv32, x, q, y);
    if (!q.valid) return;
    // x + omega D^-1 (r - A x) = x + omega (D^-1 r - S x)
    const float om = (float)__ldg(a.omega);
    float rr[3] = {(float)r[3 * q.i], (float)r[3 * q.i + 1], (float)r[3 * q.i + 2]}, z[3];
    mul3(a.dinv32 + 9 * (size_t)q.i, rr, z);
#pragma unroll
    for (int k = 0; k < 3; ++k) out[3 * q.i + k] = (double)fmaf(om, z[k] - y[k], x[3 * q.i + k]);
}

// x_i += sum over the prolongator blocks (i, J) of P_iJ e_J.  The CTA's
// nodes own a contiguous range of blocks: consecutive threads take
// consecutive (block, row) pairs -- coalesced reads of the prolongator --
// into shared memory, then each node adds its blocks' rows in block order.
__global__ void k_v0_prolong(V0 a, AmgLevel F, const float* __restrict__ e, float* __restrict__ x) {
    extern __shared__ float part[];  // [3 * blocks of the CTA's nodes]
    pdl_enter();
    if (seg_stopped(a.d.scal, a.d.cta_seg[blockIdx.x])) return;
    const int n0 = a.d.cta_node0[blockIdx.x], n1 = a.d.cta_node1[blockIdx.x];
    const int b0 = __ldg(&F.prow[n0]);
    const int nitem = 3 * (__ldg(&F.prow[n1]) - b0);
    for (int q = threadIdx.x; q < nitem; q += blockDim.x) {
        const int bq = q / 3, k = q - 3 * bq;
        const int J = __ldg(&F.pcol[b0 + bq]);
        float s = 0.f;
        if (!TF_IN(F.check, J, F.ncoarse, CK_PROLONG_COL)) {
            part[q] = 0.f;
            continue;
        }
        const __half2* __restrict__ P2 = reinterpret_cast<const __half2*>(F.Pvh + 18 * (size_t)(b0 + bq) + 6 * k);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 f = __half22float2(__ldg(&P2[c]));
            s = fmaf(f.x, e[6 * J + 2 * c], fmaf(f.y, e[6 * J + 2 * c + 1], s));
        }
        part[q] = s;
    }
    __syncthreads();
    const int i = n0 + threadIdx.x;
    if (i >= n1) return;
    const int p0 = __ldg(&F.prow[i]) - b0, p1 = __ldg(&F.prow[i + 1]) - b0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float s = x[3 * i + k];
        for (int b = p0; b < p1; ++b) s += part[3 * b + k];
        x[3 * i + k] = s;
    }
}

// t = r - A x with A x = D (S x) + X x  (one warp per row, lane k < 6 writing component k)
__global__ void k_v6_resid(AmgLevel L, const double* __restrict__ scal, const float* __restrict__ x) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    Row6 R;
    float D[6];
    if (i < L.n) {
        R = row6_load(L, i);
        const float* __restrict__ Dg = L.val + 36 * (size_t)__ldg(&L.diag[i]) + 6 * min(lane, 5);
#pragma unroll
        for (int k = 0; k < 6; ++k) D[k] = __ldg(&Dg[k]);
    }
    pdl_enter();
    pdl_next();
    if (i >= L.n || level_stopped(L, scal, i)) return;
    const float s = row6_warp_h(L, R, x);
    float y[6], e[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) y[k] = __shfl_sync(0xffffffffu, s, k);
    extra6(L, i, x, e);
    if (lane >= 6) return;
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) t = fmaf(D[k], y[k], t);
    L.t[6 * i + lane] = L.r[6 * i + lane] - t - pick6(e, lane);
}

// out = x + weight omega D^-1 (r - A x) = x + weight omega (D^-1 (r - X x) - S x),
// S = D^-1 A in FP16, X the extra blocks  (one warp per row)
__global__ void k_v6_post(AmgLevel L, const double* __restrict__ scal, const double* __restrict__ omega, float weight,
                          const float* __restrict__ x, float* __restrict__ out) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    Row6 R;
    float D[6], om = 0.f;
    if (i < L.n) {
        R = row6_load(L, i);
        const float* __restrict__ Dg = L.dinv + 36 * (size_t)i + 6 * min(lane, 5);
#pragma unroll
        for (int k = 0; k < 6; ++k) D[k] = __ldg(&Dg[k]);
        om = weight * (float)__ldg(omega);
    }
    pdl_enter();
    pdl_next();
    if (i >= L.n) return;
    float rr[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) rr[k] = L.r[6 * i + k];
    if (level_stopped(L, scal, i)) return;
    const float y = row6_warp_h(L, R, x);
    if (L.xrow) {
        float e[6];
        extra6(L, i, x, e);
#pragma unroll
        for (int k = 0; k < 6; ++k) rr[k] -= e[k];
    }
    if (lane >= 6) return;
    float z = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) z = fmaf(D[k], rr[k], z);
    out[6 * i + lane] = fmaf(om, z - y, x[6 * i + lane]);
}

// x_i += sum over the prolongator blocks (i, J) of P_iJ e_J (6-DOF fine level),
// one thread per DOF (one per node: 7.8 against 5.5 us to 8,978 nodes)
__global__ void k_v6_prolong(AmgLevel F, const double* __restrict__ scal, const float* __restrict__ e, float* x) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x, i = q / 6, k = q - 6 * i;
    const int b0 = i < F.n ? __ldg(&F.prow[i]) : 0, b1 = i < F.n ? __ldg(&F.prow[i + 1]) : 0;
    pdl_enter();
    pdl_next();
    if (i >= F.n || level_stopped(F, scal, i)) return;
    float s = x[q];
#pragma unroll 4
    for (int b = b0; b < b1; ++b) {
        const int J = __ldg(&F.pcol[b]);
        if (!TF_IN(F.check, J, F.ncoarse, CK_PROLONG_COL)) continue;
        const float2* __restrict__ P = reinterpret_cast<const float2*>(F.Pv + 36 * (size_t)b + 6 * k);
        const float2* __restrict__ ej = reinterpret_cast<const float2*>(e + 6 * (size_t)J);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 p = __ldg(&P[c]), v = ej[c];
            s = fmaf(p.x, v.x, fmaf(p.y, v.y, s));
        }
    }
    x[q] = s;
}

// Buffers of the damped-Jacobi sweeps of a coarse level (a sweep reads one
// vector and writes another): the pre-sweeps after the first (fused into the
// restriction, into x) alternate x and e; the post-sweeps alternate x and t
// and the last writes e, the level's output.
__host__ __device__ __forceinline__ float* pre_sweep_out(const AmgLevel& L, const float* cur) {
    return cur == L.x ? L.e : L.x;
}
__host__ __device__ __forceinline__ float* post_sweep_out(const AmgLevel& L, const float* cur, int s, int sweeps) {
    if (s == sweeps) return L.e;
    return cur == L.x ? L.t : L.x;
}

// e = M r on level `dense`, M the explicit operator of the V-cycles from that
// level down (k_dense_build), one warp per row.  Bound by reading M (22 MB at
// the 391-node level of the 320,000-prism sheet); it replaces the three sweeps
// each way, residual, restriction and prolongation of that level and the
// levels below.
__global__ void k_dense(AmgLevel L, const double* __restrict__ scal, const int* __restrict__ doff,
                        const float* __restrict__ mat) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // row over all instances
    const int g = L.single || k >= 6 * L.n ? 0 : L.seg[k / 6];
    const int lane = threadIdx.x & 31;
    const int k0 = L.single ? 0 : 6 * L.seg0[g];
    const int m2 = L.single ? 3 * L.n : 3 * (L.seg0[g + 1] - L.seg0[g]);  // pairs of a row (m is even)
    const float2* __restrict__ M =
        reinterpret_cast<const float2*>(mat + (L.single ? 0 : doff[g]) + (size_t)(k - k0) * (2 * m2));
    float2 a[8];  // before the wait: the operator's first entries
#pragma unroll
    for (int u = 0; u < 8; ++u)
        a[u] = k < 6 * L.n && lane + 32 * u < m2 ? __ldg(&M[lane + 32 * u]) : make_float2(0.f, 0.f);
    pdl_enter();
    pdl_next();
    if (k >= 6 * L.n || seg_stopped(scal, g)) return;
    const float2* __restrict__ r = reinterpret_cast<const float2*>(L.r + k0);
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < 8; ++u)
        if (lane + 32 * u < m2) {
            const float2 b = r[lane + 32 * u];
            s = fmaf(a[u].x, b.x, fmaf(a[u].y, b.y, s));
        }
#pragma unroll 8
    for (int q = lane + 256; q < m2; q += 32) {
        const float2 f = __ldg(&M[q]), b = r[q];
        s = fmaf(f.x, b.x, fmaf(f.y, b.y, s));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) L.e[k] = s;
}

// The dense operator column by column: kDenseCycles V-cycles (each on the
// residual the one before left) of the levels first..last applied to the unit
// vectors, in FP32 with the FP32 operators.  A CTA builds kDenseCols columns
// at once, four lanes per row with four columns each, so a lane uses every
// matrix value it loads four times (one column per lane, sixteen lanes per
// row, spent its time handing the same values to every lane: 1.83 against
// 1.10 ms at 286 nodes, three cycles).  Its vectors live in its own slice of `work`,
// [component][column]; the one the row products read is staged in shared
// memory.  Run when the coarse levels are rebuilt.
struct DenseBuild {
    AmgLevel L[kAmgMaxLevels];
    const double* omega;
    const int* cinv0;
    const float* cinv;
    int first, last;
    float weight[kDenseSweeps];
    const int2* group;
    int ngroup;
    float* work;
    int64_t stride;
    int off[kAmgMaxLevels];
    float* mat;
    const int* doff;
};

__device__ __forceinline__ float4 fma4(float a, float4 x, float4 y) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

// y += s M x for a 6x6 block M (row-major) and this lane's columns
__device__ __forceinline__ void block6(const float* __restrict__ M, float s, const float4* x, float4 (&y)[6]) {
    const float4* __restrict__ v = reinterpret_cast<const float4*>(M);
    float4 xv[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const float4 f = x[k * kDenseQuads];
        xv[k] = make_float4(s * f.x, s * f.y, s * f.z, s * f.w);
    }
#pragma unroll
    for (int u = 0; u < 9; ++u) {
        const float4 f = __ldg(&v[u]);
        y[(4 * u) / 6] = fma4(f.x, xv[(4 * u) % 6], y[(4 * u) / 6]);
        y[(4 * u + 1) / 6] = fma4(f.y, xv[(4 * u + 1) % 6], y[(4 * u + 1) / 6]);
        y[(4 * u + 2) / 6] = fma4(f.z, xv[(4 * u + 2) % 6], y[(4 * u + 2) / 6]);
        y[(4 * u + 3) / 6] = fma4(f.w, xv[(4 * u + 3) % 6], y[(4 * u + 3) / 6]);
    }
}
__device__ __forceinline__ void load6(const float4* x, float4 (&y)[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) y[k] = x[k * kDenseQuads];
}
__device__ __forceinline__ void store6(float4* x, const float4 (&y)[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) x[k * kDenseQuads] = y[k];
}

// acc -= (A x)_i; x: the vector of the instance (first node n0) in shared memory
__device__ __forceinline__ void dense_row(const AmgLevel& L, int i, int n0, int n1, const float4* x, int c,
                                          float4 (&acc)[6]) {
    const int p1 = __ldg(&L.rowptr[i + 1]);
    for (int p = __ldg(&L.rowptr[i]); p < p1; ++p)
        block6(L.val + 36 * (size_t)p, -1.f, x + 6 * (__ldg(&L.colidx[p]) - n0) * kDenseQuads + c, acc);
    if (!L.xrow) return;
    for (int q = L.xrow[i]; q < L.xrow[i + 1]; ++q) {
        const int j = L.xcol[q] - n0;
        if (j < 0 || j >= n1 - n0) continue;  // couples another instance: outside this operator
        block6(L.xval + 36 * (size_t)q, -1.f, x + 6 * j * kDenseQuads + c, acc);
    }
}

// out_i = (x_i or 0) + omega D_i^-1 acc
__device__ __forceinline__ void dense_smooth(const AmgLevel& L, int i, float om, const float4 (&acc)[6],
                                             const float4* x, float4* out) {
    const float* __restrict__ Di = L.dinv + 36 * (size_t)i;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int m = 0; m < 6; ++m) s = fma4(__ldg(&Di[6 * k + m]), acc[m], s);
        out[k * kDenseQuads] = fma4(om, s, x ? x[k * kDenseQuads] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
}

// The vector a pass of row products reads, brought into shared memory.
__device__ __forceinline__ void dense_stage(const float4* x, float4* xs, int n) {
    for (int q = threadIdx.x; q < n * kDenseQuads; q += kDenseThreads) xs[q] = x[q];
    __syncthreads();
}

__global__ void __launch_bounds__(kDenseThreads) k_dense_build(DenseBuild B) {
    extern __shared__ __align__(16) float4 xs[];  // [6 nodes][kDenseCols] of the largest instance
    const int c = threadIdx.x % kDenseQuads, h = threadIdx.x / kDenseQuads;
    constexpr int nh = kDenseThreads / kDenseQuads;  // rows in flight
    float4* work = reinterpret_cast<float4*>(B.work + (int64_t)blockIdx.x * B.stride);
    for (int gi = blockIdx.x; gi < B.ngroup; gi += gridDim.x) {
        const int g = B.group[gi].x, col0 = B.group[gi].y;
        float4 *r[kAmgMaxLevels], *x[kAmgMaxLevels], *t[kAmgMaxLevels], *e[kAmgMaxLevels];
        for (int l = B.first; l <= B.last; ++l) {
            const size_t n = (size_t)6 * (B.L[l].seg0[g + 1] - B.L[l].seg0[g]) * kDenseQuads;
            r[l] = work + B.off[l] / 4;
            x[l] = r[l] + n;
            t[l] = x[l] + n;
            e[l] = t[l] + n;
        }
        const AmgLevel& L1 = B.L[B.first];
        const int m = 6 * (L1.seg0[g + 1] - L1.seg0[g]);
        float4* y = e[B.first] + (size_t)m * kDenseQuads;
        for (int k = h; k < m; k += nh) {
            const int u = k - col0 - 4 * c;  // the unit column of this row among the lane's four
            r[B.first][k * kDenseQuads + c] = make_float4(u == 0, u == 1, u == 2, u == 3);
            y[k * kDenseQuads + c] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        for (int cyc = 0; cyc < kDenseCycles; ++cyc) {
            for (int l = B.first; l < B.last; ++l) {  // down
                const AmgLevel& F = B.L[l];
                const AmgLevel& C = B.L[l + 1];
                const int f0 = F.seg0[g], f1 = F.seg0[g + 1], c0 = C.seg0[g], c1 = C.seg0[g + 1];
                const float om = (float)__ldg(B.omega + l);
                for (int i = f0 + h; i < f1; i += nh) {
                    const size_t q = (size_t)6 * (i - f0) * kDenseQuads + c;
                    float4 acc[6];
                    load6(r[l] + q, acc);
                    dense_smooth(F, i, om * B.weight[0], acc, nullptr, x[l] + q);
                }
                __syncthreads();
                float4 *cur = x[l], *oth = e[l];
                for (int s = 2; s <= kDenseSweeps + 1; ++s) {  // the last pass leaves the residual in t
                    dense_stage(cur, xs, 6 * (f1 - f0));
                    for (int i = f0 + h; i < f1; i += nh) {
                        const size_t q = (size_t)6 * (i - f0) * kDenseQuads + c;
                        float4 acc[6];
                        load6(r[l] + q, acc);
                        dense_row(F, i, f0, f1, xs, c, acc);
                        if (s <= kDenseSweeps) dense_smooth(F, i, om * B.weight[s - 1], acc, cur + q, oth + q);
                        else store6(t[l] + q, acc);
                    }
                    __syncthreads();
                    if (s <= kDenseSweeps) {
                        float4* sw = cur;
                        cur = oth;
                        oth = sw;
                    }
                }
                x[l] = cur;
                e[l] = oth;
                for (int I = c0 + h; I < c1; I += nh) {
                    float4 acc[6];
#pragma unroll
                    for (int b = 0; b < 6; ++b) acc[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int p = __ldg(&F.pcptr[I]); p < __ldg(&F.pcptr[I + 1]); ++p) {
                        const float* __restrict__ P = F.Pc + 36 * (size_t)p;
                        const float4* ti = t[l] + (size_t)6 * (__ldg(&F.pcrow[p]) - f0) * kDenseQuads + c;
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            const float4 tk = ti[k * kDenseQuads];
#pragma unroll
                            for (int b = 0; b < 6; ++b) acc[b] = fma4(__ldg(&P[6 * k + b]), tk, acc[b]);
                        }
                    }
                    store6(r[l + 1] + (size_t)6 * (I - c0) * kDenseQuads + c, acc);
                }
                __syncthreads();
            }
            {  // coarsest level
                const AmgLevel& C = B.L[B.last];
                const int mc = 6 * (C.seg0[g + 1] - C.seg0[g]);
                const float* __restrict__ Mi = B.cinv + B.cinv0[g];
                for (int k = h; k < mc; k += nh) {
                    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int j = 0; j < mc; ++j)
                        s = fma4(__ldg(&Mi[(size_t)k * mc + j]), r[B.last][j * kDenseQuads + c], s);
                    e[B.last][k * kDenseQuads + c] = s;
                }
                __syncthreads();
            }
            for (int l = B.last - 1; l >= B.first; --l) {  // up
                const AmgLevel& F = B.L[l];
                const int f0 = F.seg0[g], f1 = F.seg0[g + 1], c0 = B.L[l + 1].seg0[g];
                const float om = (float)__ldg(B.omega + l);
                for (int i = f0 + h; i < f1; i += nh) {
                    float4* xi = x[l] + (size_t)6 * (i - f0) * kDenseQuads + c;
                    float4 s[6];
                    load6(xi, s);
                    for (int b = __ldg(&F.prow[i]); b < __ldg(&F.prow[i + 1]); ++b)
                        block6(F.Pv + 36 * (size_t)b, 1.f,
                               e[l + 1] + (size_t)6 * (__ldg(&F.pcol[b]) - c0) * kDenseQuads + c, s);
                    store6(xi, s);
                }
                __syncthreads();
                float4 *cur = x[l], *oth = e[l];
                for (int s = 1; s <= kDenseSweeps; ++s) {
                    dense_stage(cur, xs, 6 * (f1 - f0));
                    for (int i = f0 + h; i < f1; i += nh) {
                        const size_t q = (size_t)6 * (i - f0) * kDenseQuads + c;
                        float4 acc[6];
                        load6(r[l] + q, acc);
                        dense_row(F, i, f0, f1, xs, c, acc);
                        dense_smooth(F, i, om * B.weight[kDenseSweeps - s], acc, cur + q, oth + q);
                    }
                    __syncthreads();
                    float4* sw = cur;
                    cur = oth;
                    oth = sw;
                }
                x[l] = oth;
                e[l] = cur;  // the level's correction
            }
            for (int k = h; k < m; k += nh) {
                const size_t q = (size_t)k * kDenseQuads + c;
                y[q] = fma4(1.f, e[B.first][q], y[q]);
            }
            if (cyc + 1 == kDenseCycles) break;
            const int f0 = L1.seg0[g], f1 = L1.seg0[g + 1];
            dense_stage(e[B.first], xs, m);
            for (int i = f0 + h; i < f1; i += nh) {  // r -= A e
                const size_t q = (size_t)6 * (i - f0) * kDenseQuads + c;
                float4 acc[6];
                load6(r[B.first] + q, acc);
                dense_row(L1, i, f0, f1, xs, c, acc);
                store6(r[B.first] + q, acc);
            }
            __syncthreads();
        }
        for (int k = h; k < m; k += nh) {
            const float4 v = y[(size_t)k * kDenseQuads + c];
            const float o[4] = {v.x, v.y, v.z, v.w};
            float* out = B.mat + B.doff[g] + (size_t)k * m + col0 + 4 * c;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (col0 + 4 * c + u < m) out[u] = o[u];
        }
        __syncthreads();
    }
}

}  // namespace

void amg_mark_stale(tf_handle* h, int level) {
    if (h->amg) h->amg->stale = std::max(h->amg->stale, level);
}

bool amg_reused(const tf_handle* h) { return h->amg && h->amg->reused; }

long amg_rebuilds(const tf_handle* h) { return h->amg ? h->amg->rebuilds : 0; }

bool use_multigrid(const tf_handle* h) { return h->amg != nullptr && !h->amg_off; }

// Numeric phase for the current matrix.  Within a time step the matrix of
// a later Newton iteration differs little from the first one's, so a new
// assembly only refreshes the FP32 copies the level-0 smoother reads; the
// coarse operators, block inverses and smoother weights are rebuilt at the
// first solve of each time step (and whenever a solve with reused coarse
// levels fails, see krylov_solve).
// The level-0 copies the smoother reads, from the current assembly: FP32
// values and block inverses, the FP16 operator S = D^-1 A and the diagonal
// blocks (kernels only: also captured into the device Newton loop).
void amg_refresh(tf_handle* h) {
    Amg* a = h->amg;
    Device& d = h->d;
    cudaStream_t st = h->stream;
    k_to_f32<<<4 * 152, kT, 0, st>>>(d.nval, d.val, a->val32);
    h->launches++;
    k_to_f32<<<4 * 152, kT, 0, st>>>(9 * (int64_t)d.nn, d.dinv, a->dinv32);
    h->launches++;
    k_to_h<<<d.ncta, kNodeThreads, 0, st>>>(d, a->val32, a->dinv32, a->valh, a->diag32);
    h->launches++;
}

// The refresh above has run for the current assembly (inside the device
// Newton loop): nothing is stale, the coarse levels are the reused ones.
void amg_refreshed(tf_handle* h) {
    if (!h->amg) return;
    h->amg->stale = 0;
    h->amg->reused = true;
}

tf_status amg_numeric(tf_handle* h) {
    NvtxRange nvtx_range("tf multigrid numeric");
    Amg* a = h->amg;
    if (a->stale == 0) return TF_OK;
    if (a->v0_smem > 48 * 1024)  // outside any stream capture: the V-cycles launched later need it
        TF_CUDA(cudaFuncSetAttribute(k_v0_prolong, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemOptIn));
    Device& d = h->d;
    cudaStream_t st = h->stream;
    amg_refresh(h);
    a->reused = a->stale == 1;
    if (a->reused) {
        a->stale = 0;
        return TF_OK;
    }
    ++a->rebuilds;
    if (a->x_version != h->extra_version) AMG_TRY(amg_extra_symbolic(h));
    // level by level: smoother weight from lambda_max(D^-1 A) (the
    // prolongator smoothing uses it too), prolongator, Galerkin product
    // A_{l+1} = P^T (A P) and the next level's block inverses
    const int last = a->coarse_exact ? a->nlev - 1 : a->nlev;  // levels with a smoother
    for (int l = 0; l < a->nlev; ++l) {
        AmgLevel& L = a->L[l];
        if (l < last) {
            const int64_t m = (int64_t)L.n * L.bs;
            double* scal = a->pscal + 2 * l;
            float *v = a->pv, *w = a->pw;
            k_pw_init<<<cdiv(m, kT), kT, 0, st>>>(m, v, a->part, a->ticket, scal);
            TF_LAUNCH_CHECK(h);
            for (int it = 0; it < kPowerIters; ++it) {
                if (l == 0)
                    k_pw_step0<<<d.ncta, kNodeThreads, split_bytes<float>(d), st>>>(d, a->valh, a->dinv32, v, w, a->part, a->ticket,
                                                                scal, a->omega, a->omega0);
                else
                    k_pw_step6<<<cdiv(32 * (int64_t)L.n, kT), kT, 0, st>>>(L, v, w, a->part, a->ticket, scal,
                                                                            a->omega + l);
                TF_LAUNCH_CHECK(h);
                std::swap(v, w);
            }
        }
        if (l + 1 == a->nlev) break;
        AmgSetup& S = a->S[l];
        AmgLevel& C = a->L[l + 1];
        const int sm = a->smooth ? 1 : 0;
        if (l == 0) {
            k_smooth_p<3, true><<<cdiv(L.npb, kT), kT, 0, st>>>(L, S, a->omega, sm, d.colidx, d.bofs, a->val32,
                                                                a->dinv32);
            TF_LAUNCH_CHECK(h);
            k_ap<3, true><<<cdiv(S.nT * 3, kT), kT, 0, st>>>(L, S, d.bofs, a->val32);
        } else {
            k_smooth_p<6, false><<<cdiv(L.npb, kT), kT, 0, st>>>(L, S, a->omega + l, sm, nullptr, nullptr,
                                                                 nullptr, nullptr);
            TF_LAUNCH_CHECK(h);
            k_ap<6, false><<<cdiv(S.nT * 6, kT), kT, 0, st>>>(L, S, nullptr, nullptr);
        }
        TF_LAUNCH_CHECK(h);
        k_p_columns<<<cdiv(L.npb * L.bs * 6, kT), kT, 0, st>>>(L, S, L.bs * 6);
        TF_LAUNCH_CHECK(h);
        if (l == 0) {
            k_f32_to_h<<<4 * 152, kT, 0, st>>>(L.npb * L.bs * 6, L.Pv, L.Pvh);
            TF_LAUNCH_CHECK(h);
            k_f32_to_h<<<4 * 152, kT, 0, st>>>(L.npb * L.bs * 6, L.Pc, L.Pch);
            TF_LAUNCH_CHECK(h);
        }
        if (l == 0 && d.nxb == 0) {  // a new extra-block layout rebuilds everything
            k_make_q<<<cdiv(S.nT, kT), kT, 0, st>>>(a->Q, S, L.Pv, a->dinv32, a->omega0);
            TF_LAUNCH_CHECK(h);
        }
        if (l == 0) k_ptap<3><<<cdiv(C.nnzb * 6, kT), kT, 0, st>>>(L, S, C);
        else k_ptap<6><<<cdiv(C.nnzb * 6, kT), kT, 0, st>>>(L, S, C);
        TF_LAUNCH_CHECK(h);
        if (C.nx > 0) {
            if (l == 0) k_xgal<3, true><<<cdiv(C.nx * 6, kT), kT, 0, st>>>(L, S, C, d.xval);
            else k_xgal<6, false><<<cdiv(C.nx * 6, kT), kT, 0, st>>>(L, S, C, nullptr);
            TF_LAUNCH_CHECK(h);
        }
        k_inv6<<<cdiv(C.n, kT), kT, 0, st>>>(C);
        TF_LAUNCH_CHECK(h);
        k_to_h6<<<cdiv(C.nnzb * 6, kT), kT, 0, st>>>(C);
        TF_LAUNCH_CHECK(h);
    }
    if (a->coarse_exact) {
        AmgLevel& L = a->L[a->nlev - 1];
        const size_t smem = sizeof(double) * (size_t)a->max_cm * a->max_cm;
        k_coarse_invert<<<a->nseg, kInvThreads, smem, st>>>(L, a->cnode0, a->cinv0, a->cinv);
        TF_LAUNCH_CHECK(h);
        if (a->dense < a->nlev - 1) {
            DenseBuild B;
            for (int l = 0; l < a->nlev; ++l) B.L[l] = a->L[l];
            B.omega = a->omega;
            B.cinv0 = a->cinv0;
            B.cinv = a->cinv;
            B.first = a->dense;
            B.last = a->nlev - 1;
            for (int s = 0; s < kDenseSweeps; ++s) B.weight[s] = sweep_weight(s, kDenseSweeps);
            B.group = a->dgroup;
            B.ngroup = a->ndgroup;
            B.work = a->dwork;
            B.stride = a->dstride;
            for (int l = 0; l < a->nlev; ++l) B.off[l] = a->dlvl[l];
            B.mat = a->dmat;
            B.doff = a->doff;
            k_dense_build<<<a->dgrid, kDenseThreads, a->dsmem, st>>>(B);
            TF_LAUNCH_CHECK(h);
        }
    }
    a->stale = 0;
    return TF_OK;
}

// The level-0 smoother's row product with 2, 4 or 8 slots in flight per
// lane, timed on the handle's own matrix (k_v0_resid: one residual of the
// current smoother operator into the level's work vector); called once per
// handle by the solve autotuner.
tf_status amg_autotune(tf_handle* h) {
    Amg* a = h->amg;
    Device& d = h->d;
    cudaStream_t st = h->stream;
    AmgLevel& L0 = a->L[0];
    V0 v0{d, a->omega0, a->dinv32, a->valh, a->diag32};
    float best = 1e30f;
    for (int u : {2, 4, 8}) {
        for (int r = 0; r < 4; ++r) {  // one warm-up, three timed
            if (r == 1) TF_CUDA(cudaEventRecord(h->ev[4], st));
            if (u == 2) k_v0_resid<2><<<d.ncta, kNodeThreads, split_bytes<float>(d), st>>>(v0, d.g, L0.x, L0.t);
            else if (u == 4) k_v0_resid<4><<<d.ncta, kNodeThreads, split_bytes<float>(d), st>>>(v0, d.g, L0.x, L0.t);
            else k_v0_resid<8><<<d.ncta, kNodeThreads, split_bytes<float>(d), st>>>(v0, d.g, L0.x, L0.t);
            TF_LAUNCH_CHECK(h);
        }
        TF_CUDA(cudaEventRecord(h->ev[5], st));
        TF_CUDA(cudaEventSynchronize(h->ev[5]));
        float ms = 0.f;
        TF_CUDA(cudaEventElapsedTime(&ms, h->ev[4], h->ev[5]));
        if (ms < best) {
            best = ms;
            a->smooth_unroll = u;
        }
    }
    return TF_OK;
}

int amg_smoother_unroll(const tf_handle* h) { return use_multigrid(h) ? h->amg->smooth_unroll : 0; }

// Level 0 through Q (k_restrict<3> on Q by column, k_q_smooth, k_q_post): every system
// without extra blocks.
static bool uses_q(const tf_handle* h) { return h->d.nxb == 0; }

// k_q_smooth beside the coarse levels: where those are a chain of launches
// (level 1 kernel by kernel) there is time to hide it in.
static bool forks(const Amg* a) { return a->dense != 1; }

bool amg_fuses_dot(const tf_handle* h) { return use_multigrid(h) && uses_q(h); }

AmgPre amg_pre(const tf_handle* h) {
    if (!use_multigrid(h)) return AmgPre{nullptr, nullptr, nullptr, nullptr};
    const Amg* a = h->amg;
    return AmgPre{a->dinv32, a->omega0, a->L[0].x, a->L[0].t};
}

int amg_vcycle_kernels(const tf_handle* h) {
    const Amg* a = h->amg;
    const int per = 2 * kCoarseSweeps + 2;  // kernels of a coarse level run kernel by kernel
    const int fine = uses_q(h) ? (forks(a) ? 3 : 2) : 4;
    if (a->dense > 0) return fine + per * (a->dense - 1) + 1;
    return fine + per * (a->nlev - 2) + 2 * kCoarseSweeps - 1;
}

template <int U>
static void launch_q_smooth(tf_handle* h, cudaStream_t st, const V0& v0, const float* z, float* x) {
    k_q_smooth<U><<<h->d.ncta, kNodeThreads, split_bytes<float>(h->d), st>>>(v0, z, x);
}

// The last kernel of a V-cycle through Q.  After k_q_smooth on the side
// stream it has two predecessors, so it is an ordinary launch there.
template <int U, bool SMOOTH>
static void launch_q_post(tf_handle* h, const V0& v0, const float* zx, double* out, const double* r, double* p,
                          int dot) {
    Amg* a = h->amg;
    const Ctx c = make_ctx(h);
    const int nb = h->d.ncta, nc = a->L[1].n;
    const float* e = a->L[1].e;
    const size_t sb = split_bytes<float>(h->d);
    const int start = dot == kVcycleStart ? 1 : 0;
    if constexpr (SMOOTH) {
        if (dot) launch_pdl_smem(k_q_post<U, true, true>, nb, kNodeThreads, sb, h->stream, v0, c, a->Q, nc, zx, e, out,
                                 r, p, start);
        else launch_pdl_smem(k_q_post<U, true, false>, nb, kNodeThreads, sb, h->stream, v0, c, a->Q, nc, zx, e, out, r,
                             p, 0);
    } else {
        if (dot) k_q_post<U, false, true><<<nb, kNodeThreads, sb, h->stream>>>(v0, c, a->Q, nc, zx, e, out, r, p,
                                                                             start);
        else k_q_post<U, false, false><<<nb, kNodeThreads, sb, h->stream>>>(v0, c, a->Q, nc, zx, e, out, r, p, 0);
    }
}

// out = M^-1 r: one V-cycle (all launches on h->stream and, joined to it, the
// side stream; no host work).  The input's FP32 copy and first sweep are in
// place (AmgPre).  Levels above `dense` run kernel by kernel over all
// instances; `dense` and the levels below it are one product with their dense
// operator.
void amg_vcycle(tf_handle* h, const double* r, double* out, int dot, double* p) {
    Amg* a = h->amg;
    Device& d = h->d;
    cudaStream_t st = h->stream;
    const int nl = a->nlev;
    const int stop = a->dense > 0 ? a->dense : nl - 1;  // first level not handled kernel by kernel
    V0 v0{d, a->omega0, a->dinv32, a->valh, a->diag32};
    AmgLevel& L0 = a->L[0];
    float weight[kCoarseSweeps];
    for (int s = 0; s < kCoarseSweeps; ++s) weight[s] = sweep_weight(s, kCoarseSweeps);
    auto presmooth = [&](int l) { return l == a->dense ? 0.f : weight[0]; };
    const bool q = uses_q(h), fork = q && forks(a);
    if (q) {
        if (fork) {
            cudaEventRecord(h->fork_ev, st);
            cudaStreamWaitEvent(h->side_stream, h->fork_ev, 0);
            switch (d.split ? 0 : a->smooth_unroll) {
                case 0: launch_q_smooth<0>(h, h->side_stream, v0, L0.x, a->x1); break;
                case 2: launch_q_smooth<2>(h, h->side_stream, v0, L0.x, a->x1); break;
                case 8: launch_q_smooth<8>(h, h->side_stream, v0, L0.x, a->x1); break;
                default: launch_q_smooth<4>(h, h->side_stream, v0, L0.x, a->x1); break;
            }
            cudaEventRecord(h->join_ev, h->side_stream);
        }
        launch_pdl(k_restrict<3, __half>, a->L[1].n, kRestrictThreads, st, (const int*)a->Q.cptr, (const int*)a->Q.crow,
                   reinterpret_cast<const __half*>(a->Q.cval), a->L[1], L0.n, L0.check, (const float*)L0.t,
                   (const double*)d.scal, (const double*)(a->omega + 1), presmooth(1));
    } else {
        switch (a->smooth_unroll) {
            case 2: launch_pdl_smem(k_v0_resid<2>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, L0.t); break;
            case 8: launch_pdl_smem(k_v0_resid<8>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, L0.t); break;
            default: launch_pdl_smem(k_v0_resid<4>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, L0.t); break;
        }
        launch_pdl(k_restrict<3, __half>, a->L[1].n, kRestrictThreads, st, (const int*)L0.pcptr, (const int*)L0.pcrow,
                   (const __half*)L0.Pch, a->L[1], L0.n, L0.check, (const float*)L0.t, (const double*)d.scal,
                   (const double*)(a->omega + 1), presmooth(1));
    }
    float* cur[kAmgMaxLevels] = {};
    for (int l = 1; l < stop; ++l) {
        AmgLevel& L = a->L[l];
        const int nb = cdiv(32 * (int64_t)L.n, kT);
        float* x = L.x;  // first pre-sweep: fused into the restriction
        for (int s = 2; s <= kCoarseSweeps; ++s) {
            float* o = pre_sweep_out(L, x);
            launch_pdl(k_v6_post, nb, kT, st, L, (const double*)d.scal, (const double*)(a->omega + l), weight[s - 1],
                       (const float*)x, o);
            x = o;
        }
        cur[l] = x;
        launch_pdl(k_v6_resid, nb, kT, st, L, (const double*)d.scal, (const float*)x);
        launch_pdl(k_restrict<6, float>, a->L[l + 1].n, kRestrictThreads, st, (const int*)L.pcptr, (const int*)L.pcrow,
                   (const float*)L.Pc, a->L[l + 1], L.n, L.check, (const float*)L.t, (const double*)d.scal,
                   (const double*)(a->omega + l + 1), presmooth(l + 1));
    }
    if (a->dense > 0) {
        AmgLevel& LD = a->L[stop];
        launch_pdl(k_dense, cdiv(32 * 6 * (int64_t)LD.n, kT), kT, st, LD, (const double*)d.scal, (const int*)a->doff,
                   (const float*)a->dmat);
    } else {
        // x from the restriction's pre-smoothing; two sweeps more, and three the other way, into e
        AmgLevel& LC = a->L[nl - 1];
        const int nbc = cdiv(32 * (int64_t)LC.n, kT);
        float* x = LC.x;
        for (int s = 2; s <= 2 * kCoarseSweeps; ++s) {
            float* o = s % 2 == 0 ? LC.e : LC.t;
            launch_pdl(k_v6_post, nbc, kT, st, LC, (const double*)d.scal, (const double*)(a->omega + nl - 1),
                       weight[s <= kCoarseSweeps ? s - 1 : 2 * kCoarseSweeps - s], (const float*)x, o);
            x = o;
        }
    }
    for (int l = stop - 1; l >= 1; --l) {
        AmgLevel& L = a->L[l];
        float* x = cur[l];
        launch_pdl(k_v6_prolong, cdiv(6 * (int64_t)L.n, kT), kT, st, L, d.scal, (const float*)a->L[l + 1].e, x);
        for (int s = 1; s <= kCoarseSweeps; ++s) {
            float* o = post_sweep_out(L, x, s, kCoarseSweeps);
            launch_pdl(k_v6_post, cdiv(32 * (int64_t)L.n, kT), kT, st, L, (const double*)d.scal,
                       (const double*)(a->omega + l), weight[kCoarseSweeps - s], (const float*)x, o);
            x = o;
        }
    }
    if (q) {
        if (fork) {
            cudaStreamWaitEvent(st, h->join_ev, 0);
            if (d.split) launch_q_post<0, false>(h, v0, a->x1, out, r, p, dot);
            else launch_q_post<4, false>(h, v0, a->x1, out, r, p, dot);
        } else {
            switch (d.split ? 0 : a->smooth_unroll) {
                case 0: launch_q_post<0, true>(h, v0, L0.x, out, r, p, dot); break;
                case 2: launch_q_post<2, true>(h, v0, L0.x, out, r, p, dot); break;
                case 8: launch_q_post<8, true>(h, v0, L0.x, out, r, p, dot); break;
                default: launch_q_post<4, true>(h, v0, L0.x, out, r, p, dot); break;
            }
        }
        return;
    }
    launch_pdl_smem(k_v0_prolong, d.ncta, kNodeThreads, (size_t)a->v0_smem, st, v0, L0, (const float*)a->L[1].e,
                    L0.x);
    switch (a->smooth_unroll) {
        case 2: launch_pdl_smem(k_v0_post<2>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, out); break;
        case 8: launch_pdl_smem(k_v0_post<8>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, out); break;
        default: launch_pdl_smem(k_v0_post<4>, d.ncta, kNodeThreads, split_bytes<float>(d), st, v0, r, L0.x, out); break;
    }
}

}  // namespace tf

extern "C" TF_API tf_status tf_multigrid_blocks(tf_handle* h, int64_t* blocks, int64_t* prolongator_blocks) {
    if (!h || !blocks || !prolongator_blocks) {
        tf::set_error("tf_multigrid_blocks: bad arguments");
        return TF_BAD_INPUT;
    }
    tf::Amg* a = tf::use_multigrid(h) ? h->amg : nullptr;
    for (int l = 0; l < (a ? a->nlev : 0); ++l) {
        blocks[l] = a->L[l].nnzb;
        prolongator_blocks[l] = a->L[l].npb;
    }
    return TF_OK;
}

extern "C" TF_API tf_status tf_multigrid_info(tf_handle* h, int32_t* levels, int32_t* nodes, double* weights) {
    if (!h || !levels) {
        tf::set_error("tf_multigrid_info: bad arguments");
        return TF_BAD_INPUT;
    }
    tf::Amg* a = tf::use_multigrid(h) ? h->amg : nullptr;
    *levels = a ? a->nlev : 0;
    if (!a) return TF_OK;
    if (nodes)
        for (int l = 0; l < a->nlev; ++l) nodes[l] = a->h_n[l];
    if (weights) {
        TF_CUDA(cudaSetDevice(h->device));
        TF_CUDA(cudaStreamSynchronize(h->stream));
        TF_CUDA(cudaMemcpy(weights, a->omega, sizeof(double) * a->nlev, cudaMemcpyDeviceToHost));
    }
    return TF_OK;
}
