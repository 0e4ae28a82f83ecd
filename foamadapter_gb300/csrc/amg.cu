// Multigrid-preconditioned CG (FP64) for a single scalar system, and the
// multigrid solver on its own.
//
// The reference selects the first through a Ginkgo configuration: solver::Cg
// whose preconditioner is solver::Multigrid with multigrid::Pgm levels
// (tutorials/cylinder2D/system/gko/config.mg.json).  GAMG in an fvSolution
// maps to Ginkgo's solver::Multigrid as the solver
// (src/compatibility/fvSolution.cpp:27): cfg->method = FVGB_SOLVER_MULTIGRID
// iterates x += V(b - A x) with the same hierarchy and V-cycle.  Ginkgo is not
// part of the reference checkout; this is this library's own aggregation AMG
// built on the published parallel-graph-match (PGM) idea:
//
// Setup, symbolic (host, once per system, from the first matrix solved):
//  * PGM aggregation (pgm_aggregate): strength |a_ij| between rows; in up to
//    15 rounds every unaggregated row picks its strongest unaggregated
//    neighbour (ties: the lower index) and mutual picks become pairs; the
//    rounds stop when at most 5% of the rows are left or no pair forms.  A row
//    left over joins the aggregate of its strongest aggregated neighbour, or
//    stays alone.  Aggregates are numbered by their lowest row.  Each level
//    applies it twice (double pairwise aggregation, as in Notay's AGMG): the
//    pairs are matched again on their Galerkin matrix, so a level keeps about
//    a quarter of the rows and the hierarchy has half as many levels.
//  * Galerkin coarse matrix A_c = P^T A P for the piecewise-constant P: its
//    pattern and, for each coarse entry, the fine entries it sums (fine rows
//    ascending, entries in row order).  Levels are added until at most
//    kCoarseRows rows remain, the aggregation stops shrinking the system
//    (more than 90% of the rows left), or kMaxLevels is reached.
// Setup, numeric (device, whenever the matrix values changed): the coarse
// values by those fixed sums, the Jacobi diagonals, and the inverse of the
// coarsest matrix by Gauss-Jordan elimination in one cluster, its rows dealt over the
// blocks, or in one block where they do not fit their shared memory (no pivoting: the
// matrix is symmetric positive definite).
// V-cycle z = M r: per level one damped-Jacobi sweep from zero (weight 0.9),
// the residual, restriction by aggregate sums, the coarser level, then the
// coarse correction and one more damped-Jacobi sweep; the coarsest level is
// solved exactly with the dense inverse.  Pre- and post-smoothing are the same
// symmetric sweep, so M is symmetric positive definite and CG applies.
// Kernels: the first sweep of level 0 is formed by the CG kernels that produce
// r (k_init, k_update), a coarse level's by the restriction that produces its
// right-hand side; residual and restriction are one kernel over whole aggregates
// (k_resid_restrict), or two where an aggregate exceeds a block (k_resid, k_restrict); level
// 0 adds the coarse correction before its second sweep (k_prolong, k_post), inside it up to
// kFusedPostRows rows in the CG, where that sweep also forms beta (k_post_rz); coarser
// levels form it inside the sweep (k_post_fused); the small levels and the
// coarsest one's dense solve run in one cluster (k_tail).  Coarse levels are sliced
// ELL like the system matrix.
//
// A solve is one CUDA graph (init, a device-side while loop over the CG
// iteration with the V-cycle inside, or over the multigrid iteration, bounded
// by max_iter).  Its stopping test and statistics are those of the Jacobi-PCG
// (Ginkgo criteria: ||r|| below max(rel_tol ||r_0||, abs_tol), or
// max(rel_tol ||b||, abs_tol) with FVGB_SOLVE_RHS_BASELINE).  Every reduction
// has a fixed order, so a solve is deterministic; its iterates are not those
// of the Jacobi-PCG.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <thread>
#include <type_traits>
#include <vector>

#include "internal.cuh"

namespace {

constexpr int kT = 256;
constexpr int kCoarseRows = 256;
constexpr int kMaxLevels = 25;
constexpr double kOmega = 0.9;
constexpr int kPgmRounds = 15;
constexpr double kPgmLeftRatio = 0.05;
constexpr int kTailThreads = 1024;
constexpr int kFusedPostRows = 1 << 19;  // level 0's coarse correction inside its last sweep up to here
constexpr int kTailSmem = 200 * 1024;  // the levels whose parts fit this together run in the tail

struct HostCsr {
    int n = 0;
    std::vector<int> rp, ci;
    std::vector<double> v;
};

// ------------------------------------------------------------ host threads
// f(begin, end, chunk) over [0, n) in contiguous chunks on up to 16 threads
// (one when n is small).  Every use below writes only its own rows, or
// per-chunk results that are joined in chunk order: the results are those of
// the sequential loop.
template <class F>
int parallel_chunks(int n, int min_per_chunk, F f) {
    const int hw = (int)std::thread::hardware_concurrency();
    const int nt = std::max(1, std::min({16, hw > 0 ? hw : 1, n / std::max(1, min_per_chunk)}));
    if (nt == 1) {
        f(0, n, 0);
        return 1;
    }
    std::vector<std::thread> th;
    th.reserve((size_t)nt);
    for (int t = 0; t < nt; ++t)
        th.emplace_back(f, (int)((int64_t)n * t / nt), (int)((int64_t)n * (t + 1) / nt), t);
    for (std::thread& x : th) x.join();
    return nt;
}

// Ids next, next+1, ... for the rows with flag set, in row order (a prefix
// sum over chunks); returns how many.
int number_flagged(int n, const std::vector<char>& flag, std::vector<int>& id, int next) {
    std::vector<int> cnt(16, 0), base(17, 0);
    const int nt = parallel_chunks(n, 1 << 15, [&](int b, int e, int t) {
        int c = 0;
        for (int i = b; i < e; ++i) c += flag[i] ? 1 : 0;
        cnt[t] = c;
    });
    for (int t = 0; t < nt; ++t) base[t + 1] = base[t] + cnt[t];
    parallel_chunks(n, 1 << 15, [&](int b, int e, int t) {
        int k = next + base[t];
        for (int i = b; i < e; ++i)
            if (flag[i]) id[i] = k++;
    });
    return base[nt];
}

// ------------------------------------------------------------ PGM (host)
int pgm_aggregate(int n, const int* rp, const int* ci, const double* v, std::vector<int>& agg) {
    agg.assign(n, -1);
    std::vector<int> pick(n, -1);
    std::vector<int> tmp(n, -1);  // provisional aggregate id of each row
    std::vector<int> id(n, -1);
    std::vector<char> flag(n, 0);
    int next = 0, left = n;
    for (int round = 0; round < kPgmRounds; ++round) {
        parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
            for (int i = b; i < e; ++i) {
                pick[i] = -1;
                if (tmp[i] >= 0) continue;
                double best = 0.0;
                for (int k = rp[i]; k < rp[i + 1]; ++k) {
                    const int j = ci[k];
                    if (j == i || tmp[j] >= 0) continue;
                    const double w = std::fabs(v[k]);
                    if (w > best || (w == best && w > 0.0 && (pick[i] < 0 || j < pick[i]))) {
                        best = w;
                        pick[i] = j;
                    }
                }
            }
        });
        // mutual picks pair up (pairs are disjoint); the lower row numbers the
        // pair, pairs numbered in the order of their lower rows
        parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
            for (int i = b; i < e; ++i) {
                const int j = pick[i];
                flag[i] = (tmp[i] < 0 && j > i && pick[j] == i) ? 1 : 0;
            }
        });
        const int formed = number_flagged(n, flag, id, next);
        parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
            for (int i = b; i < e; ++i)
                if (flag[i]) tmp[i] = tmp[pick[i]] = id[i];
        });
        next += formed;
        left -= 2 * formed;
        if (formed == 0 || left <= kPgmLeftRatio * n) break;
    }
    // rows left over: the strongest aggregated neighbour's aggregate, else alone
    std::vector<int> late(n, -1);
    parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
        for (int i = b; i < e; ++i) {
            if (tmp[i] >= 0) continue;
            double best = 0.0;
            int to = -1;
            for (int k = rp[i]; k < rp[i + 1]; ++k) {
                const int j = ci[k];
                if (j == i || tmp[j] < 0) continue;
                const double w = std::fabs(v[k]);
                if (w > best || (w == best && w > 0.0 && (to < 0 || j < to))) {
                    best = w;
                    to = j;
                }
            }
            late[i] = to >= 0 ? tmp[to] : -1;
            flag[i] = late[i] < 0 ? 1 : 0;
        }
    });
    parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
        for (int i = b; i < e; ++i)
            if (tmp[i] >= 0) flag[i] = 0;
    });
    next += number_flagged(n, flag, id, next);  // rows alone
    parallel_chunks(n, 1 << 15, [&](int b, int e, int) {
        for (int i = b; i < e; ++i)
            if (tmp[i] < 0) tmp[i] = late[i] >= 0 ? late[i] : id[i];
    });
    // number the aggregates by their lowest row
    std::vector<int> renum(next, -1);
    int nc = 0;
    for (int i = 0; i < n; ++i) {
        if (renum[tmp[i]] < 0) renum[tmp[i]] = nc++;
        agg[i] = renum[tmp[i]];
    }
    return nc;
}

// A_c = P^T A P: pattern (columns ascending), values, and for every coarse
// entry the fine entries it sums (gptr/gsrc), in the order they are summed.
void galerkin(const HostCsr& A, const std::vector<int>& agg, int nc, HostCsr& Ac, std::vector<int>& mptr,
              std::vector<int>& mem, std::vector<int>& gptr, std::vector<int>& gsrc) {
    mptr.assign(nc + 1, 0);
    for (int i = 0; i < A.n; ++i) ++mptr[agg[i] + 1];
    for (int c = 0; c < nc; ++c) mptr[c + 1] += mptr[c];
    mem.assign(A.n, 0);
    {
        std::vector<int> fill(mptr.begin(), mptr.end() - 1);
        for (int i = 0; i < A.n; ++i) mem[fill[agg[i]]++] = i;  // ascending within an aggregate
    }
    // coarse rows in chunks, each chunk's rows built apart, then joined in order
    struct Part {
        std::vector<int> rlen, ci, glen, gsrc;
        std::vector<double> v;
    };
    std::vector<Part> parts(16);
    const int nt = parallel_chunks(nc, 4096, [&](int cb, int ce, int t) {
        Part& P = parts[t];
        std::vector<std::pair<int, int>> items;  // (coarse column, fine entry) in summation order
        for (int c = cb; c < ce; ++c) {
            items.clear();
            for (int m = mptr[c]; m < mptr[c + 1]; ++m) {
                const int i = mem[m];
                for (int k = A.rp[i]; k < A.rp[i + 1]; ++k) items.emplace_back(agg[A.ci[k]], k);
            }
            std::stable_sort(items.begin(), items.end(), [](const std::pair<int, int>& a, const std::pair<int, int>& b) {
                return a.first < b.first;
            });
            int len = 0;
            size_t s = 0;
            while (s < items.size()) {
                const int col = items[s].first;
                double sum = 0.0;
                size_t e = s;
                while (e < items.size() && items[e].first == col) {
                    sum += A.v[items[e].second];
                    P.gsrc.push_back(items[e].second);
                    ++e;
                }
                P.ci.push_back(col);
                P.v.push_back(sum);
                P.glen.push_back((int)(e - s));
                ++len;
                s = e;
            }
            P.rlen.push_back(len);
        }
    });
    Ac.n = nc;
    Ac.rp.assign(nc + 1, 0);
    Ac.ci.clear();
    Ac.v.clear();
    gptr.assign(1, 0);
    gsrc.clear();
    gsrc.reserve(A.ci.size());
    int c = 0;
    for (int t = 0; t < nt; ++t) {
        const Part& P = parts[t];
        for (int len : P.rlen) {
            Ac.rp[c + 1] = Ac.rp[c] + len;
            ++c;
        }
        Ac.ci.insert(Ac.ci.end(), P.ci.begin(), P.ci.end());
        Ac.v.insert(Ac.v.end(), P.v.begin(), P.v.end());
        for (int g : P.glen) gptr.push_back(gptr.back() + g);
        gsrc.insert(gsrc.end(), P.gsrc.begin(), P.gsrc.end());
    }
}

// ------------------------------------------------------------ device state
struct AmgState {
    double* x;
    double rel_tol, abs_tol;
    int32_t max_iter;
    double rz, alpha, beta, res0, res, tol;
    int32_t iter, status, done;
    unsigned counter;
    int32_t want_bbase;            // FVGB_SOLVE_RHS_BASELINE: rel_tol is relative to ||b||
    double bbase;                  // ||b|| when asked for (k_bnorm), else -1
    double vinv;                   // FP32 V-cycle: 1/sigma of the residual it was given (sigma_scale)
    fvgb_solver_stats* stats_out;  // device, or null
    fvgb_solver_stats stats;
};

// Levels >= 1 are stored sliced ELL like the system matrix (32-row slices,
// column-major inside a slice, padding slots: column = row, value 0).
struct Level {
    int n = 0, nnz = 0;
    int *sptr = nullptr, *scol = nullptr, *dpos = nullptr;  // levels >= 1 (level 0: the mesh's sliced ELL)
    double *val = nullptr, *dinv = nullptr;
    int* agg = nullptr;                    // [n], when a coarser level follows
    int *mptr = nullptr, *mem = nullptr;   // members of the next level's rows
    int* blk = nullptr;                    // first coarse row of every block of k_resid_restrict (null: an aggregate exceeds a block)
    int nblk = 0;
    int *gptr = nullptr, *gsrc = nullptr;  // sums forming the next level's values
    int* gdst = nullptr;                   // the next level's slot of each sum
    int nnz_next = 0;
    int64_t slots = 0;                     // value slots (level 0: the system's m_len)
    double *b = nullptr, *x = nullptr, *xo = nullptr, *r = nullptr;
    // FP32 copies for the FP32 V-cycle (allocated at the first mixed-precision solve)
    float *valf = nullptr, *dinvf = nullptr, *bf = nullptr, *xf = nullptr, *xof = nullptr, *rf = nullptr;
    // typed views used by the V-cycle builder
    template <class T> T* vals() const;
    template <class T> T* dinvs() const;
    template <class T> T* bs() const;
    template <class T> T* xs() const;
    template <class T> T* xos() const;
    template <class T> T* rs() const;
};
template <> double* Level::vals<double>() const { return val; }
template <> float* Level::vals<float>() const { return valf; }
template <> double* Level::dinvs<double>() const { return dinv; }
template <> float* Level::dinvs<float>() const { return dinvf; }
template <> double* Level::bs<double>() const { return b; }
template <> float* Level::bs<float>() const { return bf; }
template <> double* Level::xs<double>() const { return x; }
template <> float* Level::xs<float>() const { return xf; }
template <> double* Level::xos<double>() const { return xo; }
template <> float* Level::xos<float>() const { return xof; }
template <> double* Level::rs<double>() const { return r; }
template <> float* Level::rs<float>() const { return rf; }

template <class T>
struct TailLevelT;
struct TailPart;

}  // namespace

struct AmgCache {
    const fvgb_ls* ls = nullptr;
    uint64_t version = 0;
    std::vector<Level> lv;
    int nc = 0;            // rows of the coarsest level
    double* ainv = nullptr;  // [nc*nc] inverse of the coarsest matrix
    double *r = nullptr, *p = nullptr, *q = nullptr, *z = nullptr, *part = nullptr;
    AmgState* st = nullptr;
    int cluster = 1;               // blocks of the tail's cluster
    size_t tail_smem = 0;          // shared memory of the largest of them
    TailPart* tail_parts = nullptr;  // [cluster][levels of the tail]
    struct TailIdx {
        int per = 0;
        int *col = nullptr, *acol = nullptr, *agg = nullptr, *mem = nullptr, *mptr = nullptr;
    };
    std::vector<TailIdx> tail_idx;  // encoded columns of the tail's levels
    int tail_from = 1;             // first level run by the tail
    TailLevelT<double>* tail = nullptr;    // device descriptors of levels tail_from..L-1
    cudaGraphExec_t graph = nullptr;
    // the FP32 V-cycle of mixed-precision solves
    bool f32 = false;              // FP32 copies allocated
    uint64_t f32_version = 0;      // matrix version the FP32 copies were made from
    float* ainvf = nullptr;
    TailLevelT<float>* tailf = nullptr;
    cudaGraphExec_t graph32 = nullptr;
    cudaGraphExec_t graph_mg[2] = {nullptr, nullptr};  // the standalone multigrid solver, FP64 / FP32 V-cycle
    std::vector<void*> allocs;
    int nblk = 0;
};

namespace {

template <class T>
cudaError_t dev_alloc(AmgCache* c, T** p, size_t count) {
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
    if (e == cudaSuccess) c->allocs.push_back(*p);
    return e;
}

template <class T>
cudaError_t upload(AmgCache* c, T** p, const std::vector<T>& h) {
    cudaError_t e = dev_alloc(c, p, h.size());
    if (e == cudaSuccess && !h.empty()) e = cudaMemcpy(*p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
    return e;
}

// ------------------------------------------------------------ row access
__device__ __forceinline__ double fmaT(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaT(float a, float b, float c) { return fmaf(a, b, c); }

// Row i of a sliced-ELL matrix with values of type V: sum(i, get) = the fma chain
// over its slots, in slot order from +0, of value * get(column).  Up to 8 slots at a
// time: their column, value and gathered loads are under way together (index array
// chosen once per row), the fmas then run only over the row's own slots (a row's width
// is its slice's, so the branch is the warp's; predicated fmas would all be issued).
template <class V, class G>
__device__ __forceinline__ V chain8(int m, const int* col, const V* a, V s, G get) {
    V x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = k < m ? get(col[k]) : V(0);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k >= m) break;
        s = fmaT(a[k], x[k], s);
    }
    return s;
}

template <class V>
struct EllRowsT {  // level 0: the system's sliced-ELL matrix (or its FP32 copy)
    MeshView m;
    const V* val;
    template <class G>
    __device__ __forceinline__ V sum(int i, G get) const {
        const int slice = i >> 5;
        const int b0 = __ldg(&m.m_ptr[slice]);
        const int base = b0 + (i & 31);
        const int w = (__ldg(&m.m_ptr[slice + 1]) - b0) >> 5;
        V s = V(0);
#pragma unroll 1
        for (int k0 = 0; k0 < w; k0 += 8) {
            const int at = base + 32 * k0, left = w - k0;
            int col[8];
            V a[8];
            if (m.m_off) {
#pragma unroll
                for (int k = 0; k < 8; ++k) col[k] = k < left ? i + (int)__ldg(&m.m_off[at + k * 32]) : i;
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) col[k] = k < left ? __ldg(&m.m_col[at + k * 32]) : i;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = k < left ? __ldg(&val[at + k * 32]) : V(0);
            s = chain8(left, col, a, s, get);
        }
        return s;
    }
};

template <class V>
struct SellRowsT {  // levels >= 1
    const int* ptr;
    const int* col;
    const V* val;
    template <class G>
    __device__ __forceinline__ V sum(int i, G get) const {
        const int slice = i >> 5;
        const int b0 = __ldg(&ptr[slice]);
        const int base = b0 + (i & 31);
        const int w = (__ldg(&ptr[slice + 1]) - b0) >> 5;
        V s = V(0);
#pragma unroll 1
        for (int k0 = 0; k0 < w; k0 += 8) {
            const int at = base + 32 * k0, left = w - k0;
            int c[8];
            V a[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) c[k] = k < left ? __ldg(&col[at + k * 32]) : i;
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = k < left ? __ldg(&val[at + k * 32]) : V(0);
            s = chain8(left, c, a, s, get);
        }
        return s;
    }
};

using EllRows = EllRowsT<double>;
using SellRows = SellRowsT<double>;

// ------------------------------------------------------------ reductions
// (sm[t] += sm[t + s] for s = 128, 64, ..., 1.)  The seven serial additions of the end
// run in one warp, a different one from block to block: a DADD occupies its scheduler
// for 64 clocks, and the blocks of an SM end together.
__device__ __forceinline__ double block_sum(double v, double* sm) {
    __shared__ double out;
    const int t = threadIdx.x, lane = t & 31;
    sm[t] = v;
    __syncthreads();
    if ((t >> 5) == (int)(blockIdx.x & 7)) {
        double q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = sm[lane + 32 * k] + sm[lane + 32 * k + 128];
        double r = (q[0] + q[2]) + (q[1] + q[3]);
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) r += __shfl_down_sync(0xffffffffu, r, s);
        if (lane == 0) out = r;
    }
    __syncthreads();
    return out;
}

// Block partial into part[blockIdx.x]; true in the last block to arrive, which
// then sums part[0..gridDim.x) in index order (the same tree every time).
__device__ __forceinline__ bool arrive(AmgState* st, double* part, double partial, double* sm, double* total) {
    __shared__ bool last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = partial;
        __threadfence();
        last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double s = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kT) s += __ldcg(&part[k]);
    *total = block_sum(s, sm);
    if (threadIdx.x == 0) st->counter = 0;
    return true;
}

// The solve's end, set by an earlier kernel (or by the last block of this one, when
// every block has read it): a plain load, one request per SM.  A volatile one goes to
// L2 from every warp, 8,192 times to one address with 1,024 blocks: 2.2 us a kernel.
__device__ __forceinline__ int done_flag(const AmgState* st) { return st->done; }

// ------------------------------------------------------------ numeric setup
__global__ void __launch_bounds__(kT) k_dinv_ell(MeshView m, const double* __restrict__ val, double* __restrict__ dinv) {
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < m.n) dinv[i] = 1.0 / __ldg(&val[__ldg(&m.diag_pos[i])]);
}

__global__ void __launch_bounds__(kT)
    k_galerkin(int nnz_c, const int* __restrict__ gptr, const int* __restrict__ gsrc, const int* __restrict__ gdst,
               const double* __restrict__ vf, double* __restrict__ vc) {
    const int k = blockIdx.x * kT + threadIdx.x;
    if (k >= nnz_c) return;
    double s = 0.0;
    for (int t = __ldg(&gptr[k]); t < __ldg(&gptr[k + 1]); ++t) s += __ldg(&vf[__ldg(&gsrc[t])]);
    vc[__ldg(&gdst[k])] = s;
}

__global__ void __launch_bounds__(kT)
    k_dinv_csr(int n, const int* __restrict__ dpos, const double* __restrict__ val, double* __restrict__ dinv) {
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) dinv[i] = 1.0 / __ldg(&val[__ldg(&dpos[i])]);
}

// dense copy of the coarsest level (padding slots add 0 to the diagonal)
__global__ void __launch_bounds__(kT) k_dense(int n, SellRows rows, double* __restrict__ a) {
    const int i = blockIdx.x;
    for (int j = threadIdx.x; j < n; j += kT) a[(size_t)i * n + j] = 0.0;
    __syncthreads();
    if (threadIdx.x == 0) {
        const int b0 = __ldg(&rows.ptr[i >> 5]), b1 = __ldg(&rows.ptr[(i >> 5) + 1]);
        for (int pos = b0 + (i & 31); pos < b1; pos += 32) a[(size_t)i * n + __ldg(&rows.col[pos])] += __ldg(&rows.val[pos]);
    }
}

// In-place Gauss-Jordan inverse of an n x n SPD matrix, one block of 1024 threads.
__global__ void __launch_bounds__(1024) k_gauss_jordan(int n, double* __restrict__ a) {
    extern __shared__ double f[];  // [n]: column k of the step
    for (int k = 0; k < n; ++k) {
        const double piv = a[(size_t)k * n + k];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) f[i] = a[(size_t)i * n + k];
        __syncthreads();
        const double ip = 1.0 / piv;
        for (int j = threadIdx.x; j < n; j += blockDim.x) a[(size_t)k * n + j] = (j == k ? 1.0 : a[(size_t)k * n + j]) * ip;
        __syncthreads();
        for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
            const int i = t / n, j = t - i * n;
            if (i == k) continue;
            const double akj = a[(size_t)k * n + j];
            a[(size_t)i * n + j] = fma(-f[i], akj, j == k ? 0.0 : a[(size_t)i * n + j]);
        }
        __syncthreads();
    }
}

// Every thread of the cluster has its stores so far seen by every other (cluster scope).
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same inverse, the rows dealt over one cluster's blocks (row i to block i mod C)
// and held in their shared memory: one block's FP64 pipe needs 16 clocks per warp-wide
// update, 2.4 ms for 221 rows (n^3 / 2 clocks); 16 of them and one cluster barrier per
// step bring the 221-row inverse from 3.7 ms to 0.4.  Same operations on every entry
// in the same order, so the same bits.
constexpr int kGjThreads = 512;
__host__ __device__ inline size_t gj_smem(int n, int C) { return 8 * ((size_t)((n + C - 1) / C) * (n + 1) + 2 * (size_t)n); }

__global__ void __launch_bounds__(kGjThreads) k_gauss_jordan_cluster(int n, double* __restrict__ a) {
    extern __shared__ double sm[];  // [R][n] own rows, [2][n] scaled pivot rows, [R] column k
    const int C = (int)gridDim.x, rank = (int)blockIdx.x, R = (n + C - 1) / C, own = (n - rank + C - 1) / C;
    const int tx = threadIdx.x & 255, ty = threadIdx.x >> 8;
    double* prow = sm + (size_t)R * n;
    double* f = prow + 2 * (size_t)n;
    for (int l = ty; l < own; l += kGjThreads / 256)
        for (int j = tx; j < n; j += 256) sm[(size_t)l * n + j] = a[(size_t)(l * C + rank) * n + j];
    cluster_barrier();  // also: every block runs before its shared memory is written
    for (int k = 0; k < n; ++k) {
        double* cur = prow + (k & 1) * (size_t)n;
        if (rank == k % C) {
            double* row = sm + (size_t)(k / C) * n;
            const double piv = row[k];
            __syncthreads();
            const double ip = 1.0 / piv;
            for (int j = threadIdx.x; j < n; j += kGjThreads) {
                const double v = (j == k ? 1.0 : row[j]) * ip;
                row[j] = v;
                const unsigned at = (unsigned)__cvta_generic_to_shared(&cur[j]);
                for (int q = 0; q < C; ++q) {
                    unsigned ra;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(q));
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
                }
            }
        }
        for (int l = threadIdx.x; l < own; l += kGjThreads) f[l] = sm[(size_t)l * n + k];
        cluster_barrier();
        for (int l = ty; l < own; l += kGjThreads / 256) {
            if (l * C + rank == k) continue;
            const double fl = f[l];
            for (int j = tx; j < n; j += 256) {
                double* e = sm + (size_t)l * n + j;
                *e = fma(-fl, cur[j], j == k ? 0.0 : *e);
            }
        }
        __syncthreads();
    }
    for (int l = ty; l < own; l += kGjThreads / 256)
        for (int j = tx; j < n; j += 256) a[(size_t)(l * C + rank) * n + j] = sm[(size_t)l * n + j];
    cluster_barrier();  // no block leaves while another may write its shared memory
}

// ------------------------------------------------------------ V-cycle
// The V-cycle kernels run in the type T of the V-cycle: double, or float for
// the FP32 V-cycle of a mixed-precision solve (the CG around it stays FP64).

// Level 0's pre-smoothing sweep from zero: x = w D^-1 b
__global__ void __launch_bounds__(kT)
    k_smooth0(const AmgState* st, int n, const double* __restrict__ dinv, const double* __restrict__ b,
              double* __restrict__ x) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) x[i] = kOmega * __ldg(&dinv[i]) * __ldg(&b[i]);
}

// r = b - A x
template <class R, class T>
__global__ void __launch_bounds__(kT)
    k_resid(const AmgState* st, R rows, int n, const T* __restrict__ b, const T* __restrict__ x, T* __restrict__ r) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const T s = rows.sum(i, [&](int j) { return __ldg(&x[j]); });
    r[i] = __ldg(&b[i]) - s;
}

// b_c[I] = sum of r over the rows of aggregate I, and the coarse level's
// pre-smoothing sweep from zero x_c = w D_c^-1 b_c
template <class T>
__global__ void __launch_bounds__(kT)
    k_restrict(const AmgState* st, int nc, const int* __restrict__ mptr, const int* __restrict__ mem,
               const T* __restrict__ r, const T* __restrict__ dinv_c, T* __restrict__ bc, T* __restrict__ xc) {
    if (done_flag(st)) return;
    const int c = blockIdx.x * kT + threadIdx.x;
    if (c >= nc) return;
    T s = T(0);
    for (int k = __ldg(&mptr[c]); k < __ldg(&mptr[c + 1]); ++k) s += __ldg(&r[__ldg(&mem[k])]);
    bc[c] = s;
    xc[c] = T(kOmega) * __ldg(&dinv_c[c]) * s;
}

// Both in one kernel: a block takes whole aggregates of at most kT rows together
// (coarse rows [blk[b], blk[b+1])), a thread per fine row in the aggregates' order; the
// coarse rows then sum their members' residuals from shared memory, in the same order
// as k_restrict.  One launch and the residual's way through memory less.
template <class R, class T>
__global__ void __launch_bounds__(kT)
    k_resid_restrict(const AmgState* st, R rows, const int* __restrict__ blk, const T* __restrict__ b,
                     const T* __restrict__ x, const int* __restrict__ mptr, const int* __restrict__ mem,
                     const T* __restrict__ dinv_c, T* __restrict__ bc, T* __restrict__ xc) {
    __shared__ T sm[kT];
    const int done = done_flag(st);
    const int c0 = __ldg(&blk[blockIdx.x]), c1 = __ldg(&blk[blockIdx.x + 1]);
    const int m0 = __ldg(&mptr[c0]), m1 = __ldg(&mptr[c1]), t = threadIdx.x;
    if (done) return;
    if (m0 + t < m1) {
        const int i = __ldg(&mem[m0 + t]);
        const T s = rows.sum(i, [&](int j) { return __ldg(&x[j]); });
        sm[t] = __ldg(&b[i]) - s;
    }
    __syncthreads();
    const int c = c0 + t;
    if (c >= c1) return;
    const int k1 = __ldg(&mptr[c + 1]) - m0;
    T s = T(0);
    for (int k = __ldg(&mptr[c]) - m0; k < k1; ++k) s += sm[k];
    bc[c] = s;
    xc[c] = T(kOmega) * __ldg(&dinv_c[c]) * s;
}

// The small levels t..L-1 of a V-cycle in one thread-block cluster: each step (a
// residual, a restriction, a sweep) as a kernel of its own costs a launch and a chain
// of waits on L2 (slice, slots, gathered vector, coarse correction) for almost no
// work: 6.6 us apiece in the solve's graph.  Here a block owns a range of slices of
// every level, copies their slots, columns, aggregates and members to shared memory
// at once, and keeps its part of the levels' vectors there; a gather reads the owner's
// shared memory.  A step is then one such read, a row's chain of fmas and a cluster
// barrier.  (With the vectors in global memory a step took 4,000-9,000 clocks, the
// tail of the 512 x 512 cavity's hierarchy 42 us.)  Level t's b and x (its
// pre-smoothing sweep) come from the restriction above it; its xo is handed back up.
template <class T>
struct TailLevelT {
    int n, per;        // rows; slices per block
    const T* val;      // [slots]
    const int* col;    // [slots] owner << 16 | row in the owner's part, of the column
    const int* acol;   // [slots] the same of the column's aggregate (in the level below)
    const int* ptr;    // [slices + 1]
    const int* agg;    // [n] the same of the row's aggregate
    const int* mem;    // the same of the members of this level's rows (in the level above; levels > t)
    const int* mptr;   // [n + 1]
    const T* dinv;
    T *b, *x, *xo;     // level t: global
};
// A block's part of one level: its slices, slots and members, and where they lie in
// shared memory.
struct TailPart {
    int s0, s1, pos0, mem0, len, nmem;
    int o_val, o_col, o_acol, o_ptr, o_mem, o_mptr;  // bytes; of element pos0, s0, mem0, 32 s0
    int o_x, o_b, o_r, o_xo;                         // vectors, the same offsets in every block
    int o_inv, o_rhs;  // coarsest level: its rows of the inverse (-1: read in place), the whole right-hand side
};
constexpr int kTailRowsMax = 65535;  // rows of a block's part: 16 bits of an encoded column
inline size_t tail_round(size_t b) { return (b + 15) / 16 * 16; }

// 16-byte pieces of [first, first + bytes) rounded outwards, to shared memory at dst
// (the piece that holds `first`'s 16-byte line); every thread of the block.
__device__ __forceinline__ void tail_copy(unsigned char* dst, const void* first, size_t bytes) {
    const size_t a = (size_t)first & ~(size_t)15, n = ((size_t)first + bytes - a + 15) >> 4;
    for (size_t k = threadIdx.x; k < n; k += kTailThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + 16 * k)),
                     "l"(a + 16 * k)
                     : "memory");
}
// element e of a vector kept at `base` in its owner's shared memory
template <class T>
__device__ __forceinline__ T tail_get(const T* base, int e, int rank) {
    const int q = e >> 16;
    if (q == rank) return base[e & 0xffff];
    unsigned ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((unsigned)__cvta_generic_to_shared(base + (e & 0xffff))), "r"(q));
    T v;
    if constexpr (sizeof(T) == 8) asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(ra) : "memory");
    else asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
    return v;
}

template <class T>
__global__ void __launch_bounds__(kTailThreads)
    k_tail(const AmgState* st, const TailLevelT<T>* __restrict__ lv, const TailPart* __restrict__ parts, int nl,
           const T* __restrict__ ainv) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ TailPart part[kMaxLevels];
    __shared__ TailLevelT<T> lev[kMaxLevels];
    const int done = done_flag(st);  // the same in every block: only other kernels write it
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = kTailThreads / 32, rank = (int)blockIdx.x;
    for (int k = t; k < (int)(nl * sizeof(TailPart) / 4); k += kTailThreads)
        ((int*)part)[k] = __ldg((const int*)(parts + (size_t)rank * nl) + k);
    for (int k = t; k < (int)(nl * sizeof(TailLevelT<T>) / 4); k += kTailThreads)
        ((int*)lev)[k] = __ldg((const int*)lv + k);
    __syncthreads();
    if (done) return;
    for (int l = 0; l < nl; ++l) {
        const TailLevelT<T>& F = lev[l];
        const TailPart& P = part[l];
        const int rows = min(F.n, P.s1 * 32) - P.s0 * 32;
        if (rows <= 0) continue;
        if (l + 1 < nl) {
            tail_copy(dyn + (P.o_val & ~15), F.val + P.pos0, sizeof(T) * (size_t)P.len);
            tail_copy(dyn + (P.o_col & ~15), F.col + P.pos0, 4 * (size_t)P.len);
            tail_copy(dyn + (P.o_acol & ~15), F.acol + P.pos0, 4 * (size_t)P.len);
            tail_copy(dyn + (P.o_ptr & ~15), F.ptr + P.s0, 4 * (size_t)(P.s1 - P.s0 + 1));
        } else if (P.o_inv >= 0) {
            tail_copy(dyn + P.o_inv, ainv + (size_t)P.s0 * 32 * F.n, sizeof(T) * (size_t)rows * F.n);
        }
        if (l > 0) {
            tail_copy(dyn + (P.o_mem & ~15), F.mem + P.mem0, 4 * (size_t)P.nmem);
            tail_copy(dyn + (P.o_mptr & ~15), F.mptr + P.s0 * 32, 4 * (size_t)(rows + 1));
        }
    }
    {
        const TailLevelT<T>& F = lev[0];
        const TailPart& P = part[0];
        for (int q = t; q < (P.s1 - P.s0) * 32; q += kTailThreads) {
            const int i = min(F.n - 1, P.s0 * 32 + q);
            ((T*)(dyn + P.o_x))[q] = __ldcg(&F.x[i]);
            ((T*)(dyn + P.o_b))[q] = __ldcg(&F.b[i]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_barrier();
    constexpr int G = 8;  // gathers under way per thread
    for (int l = 0; l + 1 < nl; ++l) {  // down
        {
            const TailPart P = part[l];
            const int n = lev[l].n;
            const T *val = (const T*)(dyn + P.o_val), *x = (const T*)(dyn + P.o_x), *b = (const T*)(dyn + P.o_b);
            T* r = (T*)(dyn + P.o_r);
            const int *col = (const int*)(dyn + P.o_col), *ptr = (const int*)(dyn + P.o_ptr);
            for (int sl = wid; sl < P.s1 - P.s0; sl += nw) {
                const int q = sl * 32 + lane, base = ptr[sl] - P.pos0 + lane, w = (ptr[sl + 1] - ptr[sl]) >> 5;
                if (P.s0 * 32 + q >= n) continue;
                T s = T(0);
                for (int k0 = 0; k0 < w; k0 += G) {
                    T v[G];
#pragma unroll
                    for (int k = 0; k < G; ++k) v[k] = tail_get(x, col[base + 32 * min(k0 + k, w - 1)], rank);
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        if (k0 + k >= w) break;
                        s = fmaT(val[base + 32 * (k0 + k)], v[k], s);
                    }
                }
                r[q] = b[q] - s;
            }
        }
        cluster_barrier();
        {
            const TailPart P = part[l + 1];
            const TailLevelT<T>& K = lev[l + 1];
            const T* r = (const T*)(dyn + part[l].o_r);
            T *kb = (T*)(dyn + P.o_b), *kx = (T*)(dyn + P.o_x);
            const int *mem = (const int*)(dyn + P.o_mem), *mptr = (const int*)(dyn + P.o_mptr);
            for (int q = t; q < (P.s1 - P.s0) * 32; q += kTailThreads) {
                if (P.s0 * 32 + q >= K.n) continue;
                const T dc = __ldg(&K.dinv[P.s0 * 32 + q]);
                const int m1 = mptr[q + 1] - P.mem0;
                T s = T(0);
                for (int k0 = mptr[q] - P.mem0; k0 < m1; k0 += G) {
                    T v[G];
#pragma unroll
                    for (int k = 0; k < G; ++k) v[k] = tail_get(r, mem[min(k0 + k, m1 - 1)], rank);
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        if (k0 + k >= m1) break;
                        s += v[k];
                    }
                }
                kb[q] = s;
                kx[q] = T(kOmega) * dc * s;
            }
        }
        cluster_barrier();
    }
    {  // coarsest: xo = A^-1 b, a warp per row
        const TailPart P = part[nl - 1];
        const int n = lev[nl - 1].n, per = lev[nl - 1].per * 32;
        T *xo = (T*)(dyn + P.o_xo), *rhs = (T*)(dyn + P.o_rhs);
        if (P.s1 > P.s0) {  // the whole right-hand side once
            for (int q = 0; q * per < n; ++q)
                for (int k = t; k < min(per, n - q * per); k += kTailThreads)
                    rhs[q * per + k] = tail_get((const T*)(dyn + P.o_b), q << 16 | k, rank);
            __syncthreads();
        }
        for (int row = P.s0 * 32 + wid; row < min(n, P.s1 * 32); row += nw) {
            const T* inv = P.o_inv >= 0 ? (const T*)(dyn + P.o_inv) + (size_t)(row - P.s0 * 32) * n : ainv + (size_t)row * n;
            T s = T(0);
#pragma unroll 4
            for (int j = lane; j < n; j += 32) s = fmaT(inv[j], rhs[j], s);
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) xo[row - P.s0 * 32] = s;
        }
        cluster_barrier();
    }
    for (int l = nl - 2; l >= 0; --l) {  // up: y = x + P xc formed inside the sweep
        const TailLevelT<T>& F = lev[l];
        const TailPart P = part[l];
        const T *val = (const T*)(dyn + P.o_val), *x = (const T*)(dyn + P.o_x), *b = (const T*)(dyn + P.o_b);
        const T* xc = (const T*)(dyn + part[l + 1].o_xo);
        T* xo = (T*)(dyn + P.o_xo);
        const int *col = (const int*)(dyn + P.o_col), *acol = (const int*)(dyn + P.o_acol), *ptr = (const int*)(dyn + P.o_ptr);
        for (int sl = wid; sl < P.s1 - P.s0; sl += nw) {
            const int q = sl * 32 + lane, i = P.s0 * 32 + q, base = ptr[sl] - P.pos0 + lane, w = (ptr[sl + 1] - ptr[sl]) >> 5;
            if (i >= F.n) continue;
            const T di = __ldg(&F.dinv[i]);
            const T yi = x[q] + tail_get(xc, __ldg(&F.agg[i]), rank);
            T s = T(0);
            for (int k0 = 0; k0 < w; k0 += G) {
                T v[G], u[G];
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    const int at = base + 32 * min(k0 + k, w - 1);
                    u[k] = tail_get(xc, acol[at], rank);
                    v[k] = tail_get(x, col[at], rank);
                }
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    if (k0 + k >= w) break;
                    s = fmaT(val[base + 32 * (k0 + k)], v[k] + u[k], s);
                }
            }
            const T out = fmaT(T(kOmega) * di, b[q] - s, yi);
            xo[q] = out;
            if (l == 0) F.xo[i] = out;
        }
        cluster_barrier();  // (the last: no block leaves while another may read its shared memory)
    }
    if (nl == 1) {  // the coarsest level alone
        const TailPart P = part[0];
        for (int q = t; q < (P.s1 - P.s0) * 32; q += kTailThreads)
            if (P.s0 * 32 + q < lev[0].n) lev[0].xo[P.s0 * 32 + q] = ((const T*)(dyn + P.o_xo))[q];
    }
}

// y = x + P xc
template <class T>
__global__ void __launch_bounds__(kT)
    k_prolong(const AmgState* st, int n, const T* __restrict__ x, const T* __restrict__ xc,
              const int* __restrict__ agg, T* __restrict__ y) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) y[i] = __ldg(&x[i]) + __ldg(&xc[__ldg(&agg[i])]);
}

// y = x + P xc; out = y + w D^-1 (b - A y), y formed on the fly (coarse
// levels, where a launch costs more than the extra dependent load)
template <class T>
__global__ void __launch_bounds__(kT)
    k_post_fused(const AmgState* st, SellRowsT<T> rows, int n, const T* __restrict__ dinv, const T* __restrict__ b,
                 const T* __restrict__ x, const T* __restrict__ xc, const int* __restrict__ agg, T* __restrict__ out) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const T yi = __ldg(&x[i]) + __ldg(&xc[__ldg(&agg[i])]);
    const T s = rows.sum(i, [&](int j) { return __ldg(&x[j]) + __ldg(&xc[__ldg(&agg[j])]); });
    out[i] = fmaT(T(kOmega) * __ldg(&dinv[i]), __ldg(&b[i]) - s, yi);
}

// out = y + w D^-1 (b - A y), stored as TO (level 0 hands z back as double;
// from the FP32 V-cycle, times 1/sigma of the residual it was given)
template <class R, class T, class TO>
__global__ void __launch_bounds__(kT)
    k_post(const AmgState* st, R rows, int n, const T* __restrict__ dinv, const T* __restrict__ b,
           const T* __restrict__ y, TO* __restrict__ out) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const T s = rows.sum(i, [&](int j) { return __ldg(&y[j]); });
    const T v = fmaT(T(kOmega) * __ldg(&dinv[i]), __ldg(&b[i]) - s, __ldg(&y[i]));
    if constexpr (std::is_same<T, float>::value && std::is_same<TO, double>::value)
        out[i] = (double)v * st->vinv;
    else
        out[i] = (TO)v;
}

__global__ void __launch_bounds__(kT) k_to_float(int64_t count, const double* __restrict__ src, float* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
    if (i < count) dst[i] = (float)src[i];
}

// ------------------------------------------------------------ CG
__global__ void k_params(AmgState* st, double* x, double rel_tol, double abs_tol, int max_iter,
                         fvgb_solver_stats* out, int want_bbase) {
    st->want_bbase = want_bbase;
    st->bbase = -1.0;
    st->vinv = 1.0;
    st->x = x;
    st->rel_tol = rel_tol;
    st->abs_tol = abs_tol;
    st->max_iter = max_iter;
    st->stats_out = out;
    st->counter = 0;
    st->done = 0;
}

// The FP32 V-cycle runs on sigma r, sigma = 2^-ilogb(|r_prev|) (the previous
// residual norm, known when the new residual is formed): the residual's entries
// sit near 1 whatever the system's scale, so neither underflow nor overflow
// FP32.  The V-cycle is linear and every FP32 operation commutes exactly with a
// power-of-two scale in the normal range, so z = (double)z_sigma / sigma has
// the bits of the unscaled V-cycle wherever that one stays in range.
__device__ __forceinline__ double sigma_scale(double res) {
    return (res > 0.0 && isfinite(res)) ? ldexp(1.0, -ilogb(res)) : 1.0;
}

// The V-cycle's first sweep from the new residual r_i: x0 = w D^-1 r in FP64,
// or, for the FP32 V-cycle (b0f set), b0 = (float)(sigma r) and x0 = w D^-1 b0
// in FP32; neither when both are null (the FP32 first sweep of a solve runs
// after its initial residual norm, k_first_f32).
__device__ __forceinline__ void first_sweep(int i, double ri, const double* __restrict__ dinv0, double* __restrict__ x0,
                                            const float* __restrict__ d0f, float* __restrict__ b0f,
                                            float* __restrict__ x0f, double sigma) {
    if (b0f) {
        const float bf = (float)(ri * sigma);
        b0f[i] = bf;
        x0f[i] = float(kOmega) * __ldg(&d0f[i]) * bf;
    } else if (x0) {
        x0[i] = kOmega * __ldg(&dinv0[i]) * ri;
    }
}

// The FP32 V-cycle's first sweep from the initial residual, once its norm is known
__global__ void __launch_bounds__(kT)
    k_first_f32(AmgState* st, int n, const double* __restrict__ r, const float* __restrict__ d0f,
                float* __restrict__ b0f, float* __restrict__ x0f) {
    if (done_flag(st)) return;
    const double sigma = sigma_scale(st->res0);
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) first_sweep(i, __ldg(&r[i]), nullptr, nullptr, d0f, b0f, x0f, sigma);
    if (i == 0) st->vinv = 1.0 / sigma;
}

// ||b||, the baseline of the relative tolerance when the solve asks for it
// (Ginkgo's ResidualNorm with its default baseline, rhs_norm)
__global__ void __launch_bounds__(kT) k_bnorm(AmgState* st, int n, const double* __restrict__ b, double* part) {
    __shared__ double sm[kT];
    if (!st->want_bbase) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    const double bi = i < n ? __ldg(&b[i]) : 0.0;
    double tot;
    if (arrive(st, part, block_sum(bi * bi, sm), sm, &tot) && threadIdx.x == 0) st->bbase = sqrt(tot);
}

// r = b - A x, ||r||; the V-cycle's first sweep
__global__ void __launch_bounds__(kT)
    k_init(AmgState* st, EllRows A, int n, const double* __restrict__ b, double* __restrict__ r, double* part,
           const double* __restrict__ dinv0, double* __restrict__ x0, const float* __restrict__ d0f,
           float* __restrict__ b0f, float* __restrict__ x0f) {
    __shared__ double sm[kT];
    const int i = blockIdx.x * kT + threadIdx.x;
    const double* x = st->x;
    double ri = 0.0;
    if (i < n) {
        const double s = A.sum(i, [&](int j) { return x[j]; });
        ri = __ldg(&b[i]) - s;
        r[i] = ri;
        first_sweep(i, ri, dinv0, x0, d0f, b0f, x0f, 1.0);
    }
    double tot;
    if (arrive(st, part, block_sum(ri * ri, sm), sm, &tot) && threadIdx.x == 0) {
        const double res = sqrt(tot);
        st->res0 = st->res = res;
        st->iter = 0;
        st->status = FVGB_OK;
        double tol = st->rel_tol * (st->bbase >= 0.0 ? st->bbase : res);
        if (st->abs_tol > tol) tol = st->abs_tol;
        st->tol = tol;
        int done = !(res > tol) || res == 0.0;
        if (!isfinite(res)) {
            done = 1;
            st->status = FVGB_ERR_BREAKDOWN;
        } else if (!done && st->max_iter <= 0) {
            done = 1;
            st->status = FVGB_ERR_NOT_CONVERGED;
        }
        st->done = done;
    }
}

// p = z, rz = r.z (first direction)
__global__ void __launch_bounds__(kT)
    k_first_dir(AmgState* st, int n, const double* __restrict__ r, const double* __restrict__ z, double* __restrict__ p,
                double* part) {
    __shared__ double sm[kT];
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    double v = 0.0;
    if (i < n) {
        const double zi = z[i];
        p[i] = zi;
        v = r[i] * zi;
    }
    double tot;
    if (arrive(st, part, block_sum(v, sm), sm, &tot) && threadIdx.x == 0) st->rz = tot;
}

// q = A p, alpha = rz / p.q
__global__ void __launch_bounds__(kT)
    k_spmv(AmgState* st, EllRows A, int n, const double* __restrict__ p, double* __restrict__ q, double* part) {
    __shared__ double sm[kT];
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    double v = 0.0;
    if (i < n) {
        const double s = A.sum(i, [&](int j) { return __ldg(&p[j]); });
        q[i] = s;
        v = __ldg(&p[i]) * s;
    }
    double tot;
    if (arrive(st, part, block_sum(v, sm), sm, &tot) && threadIdx.x == 0) {
        const double alpha = st->rz / tot;
        st->alpha = alpha;
        if (tot == 0.0 || !isfinite(alpha)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
    }
}

// x += alpha p, r -= alpha q, ||r||, convergence; x0 = w D^-1 r (the V-cycle's first sweep)
__global__ void __launch_bounds__(kT)
    k_update(AmgState* st, int n, const double* __restrict__ p, const double* __restrict__ q, double* __restrict__ r,
             double* part, const double* __restrict__ dinv0, double* __restrict__ x0, const float* __restrict__ d0f,
             float* __restrict__ b0f, float* __restrict__ x0f) {
    __shared__ double sm[kT];
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    const double alpha = st->alpha;
    const double sigma = b0f ? sigma_scale(st->res) : 1.0;  // the previous residual norm (rewritten by the last block below)
    double* x = st->x;
    double v = 0.0;
    if (i < n) {
        x[i] = fma(alpha, __ldg(&p[i]), x[i]);
        const double ri = fma(-alpha, __ldg(&q[i]), r[i]);
        r[i] = ri;
        first_sweep(i, ri, dinv0, x0, d0f, b0f, x0f, sigma);
        v = ri * ri;
    }
    double tot;
    if (arrive(st, part, block_sum(v, sm), sm, &tot) && threadIdx.x == 0) {
        const double res = sqrt(tot);
        st->res = res;
        st->vinv = 1.0 / sigma;
        st->iter += 1;
        if (!isfinite(res)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        } else if (res <= st->tol) {
            st->done = 1;
        } else if (st->iter >= st->max_iter) {
            st->status = FVGB_ERR_NOT_CONVERGED;
            st->done = 1;
        }
    }
}

// p = z + beta p
__global__ void __launch_bounds__(kT)
    k_dir(const AmgState* st, int n, const double* __restrict__ z, double* __restrict__ p) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) p[i] = fma(st->beta, p[i], __ldg(&z[i]));
}

// Level 0's last sweep of the V-cycle inside the CG, z = y + w D^-1 (b - A y), with the
// CG's next step: beta = r.z / rz_old (k_rz, the same blocks and sums) and the loop's
// condition.  FUSED: y = x + P xc formed inside the sweep (as k_post_fused: systems
// whose working set stays in L2 gain the launch, larger ones lose the extra traffic).
template <class R, class T, bool FUSED>
__global__ void __launch_bounds__(kT)
    k_post_rz(AmgState* st, R rows, int n, const T* __restrict__ dinv, const T* __restrict__ b, const T* __restrict__ y,
              const T* __restrict__ xc, const int* __restrict__ agg, double* __restrict__ z,
              const double* __restrict__ r, double* part, cudaGraphConditionalHandle h) {
    __shared__ double sm[kT];
    const int done = done_flag(st);
    const int i = blockIdx.x * kT + threadIdx.x;
    if (done) {
        if (i == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    double v = 0.0;
    if (i < n) {
        T s = T(0);
        T yi = __ldg(&y[i]);
        if (FUSED) {
            yi = yi + __ldg(&xc[__ldg(&agg[i])]);
            s = rows.sum(i, [&](int j) { return __ldg(&y[j]) + __ldg(&xc[__ldg(&agg[j])]); });
        } else {
            s = rows.sum(i, [&](int j) { return __ldg(&y[j]); });
        }
        const T o = fmaT(T(kOmega) * __ldg(&dinv[i]), __ldg(&b[i]) - s, yi);
        double zi;
        if constexpr (std::is_same<T, float>::value) zi = (double)o * st->vinv;
        else zi = o;
        z[i] = zi;
        v = __ldg(&r[i]) * zi;
    }
    double tot;
    if (arrive(st, part, block_sum(v, sm), sm, &tot) && threadIdx.x == 0) {
        const double beta = tot / st->rz;
        st->beta = beta;
        st->rz = tot;
        if (!isfinite(beta)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
        cudaGraphSetConditional(h, st->done ? 0u : 1u);
    }
}

// ------------------------------------------------------------ standalone multigrid
// Ginkgo's solver::Multigrid (OpenFOAM's GAMG as FoamAdapter maps it): one
// V-cycle per iteration on the current residual, x += V(b - A x), the
// residual formed again from x, until the criteria hold.  The iteration starts
// with k_init (r = b - A x, its norm, the tolerance, the V-cycle's first sweep).

// x += z
__global__ void __launch_bounds__(kT) k_mg_add(const AmgState* st, int n, const double* __restrict__ z) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    double* x = st->x;
    if (i < n) x[i] = x[i] + __ldg(&z[i]);
}

// r = b - A x, ||r||, convergence; the V-cycle's first sweep of the next iteration
__global__ void __launch_bounds__(kT)
    k_mg_resid(AmgState* st, EllRows A, int n, const double* __restrict__ b, double* __restrict__ r, double* part,
               const double* __restrict__ dinv0, double* __restrict__ x0, const float* __restrict__ d0f,
               float* __restrict__ b0f, float* __restrict__ x0f) {
    __shared__ double sm[kT];
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    const double sigma = b0f ? sigma_scale(st->res) : 1.0;  // the previous residual norm (rewritten by the last block below)
    const double* x = st->x;
    double ri = 0.0;
    if (i < n) {
        const double s = A.sum(i, [&](int j) { return x[j]; });
        ri = __ldg(&b[i]) - s;
        r[i] = ri;
        first_sweep(i, ri, dinv0, x0, d0f, b0f, x0f, sigma);
    }
    double tot;
    if (arrive(st, part, block_sum(ri * ri, sm), sm, &tot) && threadIdx.x == 0) {
        const double res = sqrt(tot);
        st->res = res;
        st->vinv = 1.0 / sigma;
        st->iter += 1;
        if (!isfinite(res)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        } else if (!(res > st->tol)) {
            st->done = 1;
        } else if (st->iter >= st->max_iter) {
            st->status = FVGB_ERR_NOT_CONVERGED;
            st->done = 1;
        }
    }
}

__global__ void k_cond(AmgState* st, cudaGraphConditionalHandle h) {
    cudaGraphSetConditional(h, st->done ? 0u : 1u);
}

__global__ void k_stats(AmgState* st) {
    fvgb_solver_stats s{};
    s.init_res_norm = st->res0;
    s.final_res_norm = st->res;
    s.num_iter = st->iter;
    s.num_outer = 0;
    s.status = st->status;
    st->stats = s;
    if (st->stats_out) *st->stats_out = s;
}

// ------------------------------------------------------------ host side
template <class T>
std::vector<TailLevelT<T>> tail_levels(const AmgCache* c) {
    std::vector<TailLevelT<T>> tl;
    for (int l = c->tail_from; l < (int)c->lv.size(); ++l) {
        const Level& V = c->lv[l];
        const auto& E = c->tail_idx[l - c->tail_from];
        tl.push_back(TailLevelT<T>{V.n, E.per, V.vals<T>(), E.col, E.acol, V.sptr, E.agg, E.mem, E.mptr, V.dinvs<T>(),
                                   V.bs<T>(), V.xs<T>(), V.xos<T>()});
    }
    return tl;
}

cudaLaunchAttribute cluster_attr(int C) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    return at;
}

// The largest cluster (16, 8, ... blocks) the device runs k_tail and
// k_gauss_jordan_cluster with.
constexpr size_t kGjMaxSmem = 200 * 1024;
int cluster_size() {
    const void* fns[3] = {(const void*)k_tail<double>, (const void*)k_tail<float>, (const void*)k_gauss_jordan_cluster};
    int best = 16;
    for (const void* fn : fns) {
        const bool gj = fn == (const void*)k_gauss_jordan_cluster;
        const size_t smem = gj ? kGjMaxSmem : (size_t)kTailSmem;
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) best = std::min(best, 8);
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) best = 1;
        for (; best > 1; best /= 2) {
            cudaLaunchConfig_t lc{};
            cudaLaunchAttribute at = cluster_attr(best);
            lc.gridDim = dim3((unsigned)best);
            lc.blockDim = dim3(gj ? kGjThreads : kTailThreads);
            lc.dynamicSmemBytes = smem;
            lc.attrs = &at;
            lc.numAttrs = 1;
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, fn, &lc) == cudaSuccess && nc > 0) break;
        }
    }
    cudaGetLastError();
    return best;
}

// Picks the levels of the one-cluster tail (from the coarsest up, as long as every
// block's part fits its shared memory with FP64 values), lays the parts out and
// uploads the encoded columns.
fvgb_status tail_setup(AmgCache* c, const std::vector<std::vector<int>>& h_sptr, const std::vector<std::vector<int>>& h_scol,
                       const std::vector<std::vector<int>>& h_agg, const std::vector<std::vector<int>>& h_mptr,
                       const std::vector<std::vector<int>>& h_mem) {
    const int L = (int)c->lv.size(), C = c->cluster = cluster_size();
    std::vector<int> per(L), ns(L);
    for (int l = 0; l < L; ++l) {
        ns[l] = (c->lv[l].n + 31) / 32;
        per[l] = (ns[l] + C - 1) / C;
    }
    auto s0 = [&](int l, int r) { return std::min(ns[l], r * per[l]); };
    bool inv_in_smem = true;
    // layout of levels t.. for every block; the vectors first, at the same offsets
    auto layout = [&](int t, std::vector<TailPart>& parts) {
        parts.assign((size_t)C * (L - t), TailPart{});
        size_t most = 0, o = 0;
        for (int l = t; l < L; ++l)
            for (int TailPart::*f : {&TailPart::o_x, &TailPart::o_b, &TailPart::o_r, &TailPart::o_xo}) {
                for (int r = 0; r < C; ++r) parts[(size_t)r * (L - t) + l - t].*f = (int)o;
                o += tail_round(8 * 32 * (size_t)per[l]);
            }
        for (int r = 0; r < C; ++r) {
            size_t q = o;
            // an array's copy starts at the 16-byte line of its first element
            auto put = [&](size_t first, size_t count, size_t size) {
                const size_t shift = first * size % 16, at = q + shift;
                q += tail_round(shift + count * size);
                return (int)at;
            };
            for (int l = t; l < L; ++l) {
                TailPart& P = parts[(size_t)r * (L - t) + l - t];
                P.s0 = s0(l, r);
                P.s1 = s0(l, r + 1);
                const int rows = std::max(0, std::min(c->lv[l].n, P.s1 * 32) - P.s0 * 32);
                P.pos0 = h_sptr[l][P.s0];
                const size_t len = l + 1 < L ? h_sptr[l][P.s1] - P.pos0 : 0;
                P.len = (int)len;
                P.o_val = put(P.pos0, len, 8);
                P.o_col = put(P.pos0, len, 4);
                P.o_acol = put(P.pos0, len, 4);
                P.o_ptr = put(P.s0, P.s1 - P.s0 + 1, 4);
                if (l > t) {
                    const int i0 = std::min(c->lv[l].n, P.s0 * 32);
                    P.mem0 = h_mptr[l - 1][i0];
                    P.nmem = h_mptr[l - 1][i0 + rows] - P.mem0;
                    P.o_mem = put(P.mem0, P.nmem, 4);
                    P.o_mptr = put(P.s0 * 32, rows + 1, 4);
                }
            }
            TailPart& B = parts[(size_t)r * (L - t) + L - 1 - t];
            const size_t nc = (size_t)c->lv[L - 1].n, rows = std::max(0, std::min((int)nc, B.s1 * 32) - B.s0 * 32);
            B.o_rhs = put(0, nc, 8);
            B.o_inv = inv_in_smem ? put(0, rows * nc, 8) : -1;
            most = std::max(most, q);
        }
        return most;
    };
    std::vector<TailPart> parts, next;
    int t = L - 1;
    c->tail_smem = layout(t, parts);
    if (c->tail_smem > (size_t)kTailSmem / 2) {  // a large inverse is read in place
        inv_in_smem = false;
        c->tail_smem = layout(t, parts);
    }
    while (t > 1 && 32 * per[t - 1] <= kTailRowsMax) {
        const size_t most = layout(t - 1, next);
        if (most > (size_t)kTailSmem) break;
        parts.swap(next);
        c->tail_smem = most;
        --t;
    }
    if (c->tail_smem > (size_t)kTailSmem) return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: coarsest level too large");
    c->tail_from = t;
    cudaError_t e = upload(c, &c->tail_parts, parts);
    auto enc = [&](int l, int i) { return i / (32 * per[l]) << 16 | i % (32 * per[l]); };
    c->tail_idx.resize(L - t);
    for (int l = t; l < L && e == cudaSuccess; ++l) {
        auto& E = c->tail_idx[l - t];
        E.per = per[l];
        if (l + 1 < L) {
            std::vector<int> col(h_scol[l]), acol(h_scol[l]), agg(h_agg[l]);
            for (int& v : acol) v = enc(l + 1, h_agg[l][v]);
            for (int& v : col) v = enc(l, v);
            for (int& v : agg) v = enc(l + 1, v);
            col.resize(col.size() + 8);  // copies run to the end of a 16-byte line
            acol.resize(acol.size() + 8);
            e = upload(c, &E.col, col);
            if (e == cudaSuccess) e = upload(c, &E.acol, acol);
            if (e == cudaSuccess) e = upload(c, &E.agg, agg);
        }
        if (l > t && e == cudaSuccess) {
            std::vector<int> mem(h_mem[l - 1]), mptr(h_mptr[l - 1]);
            for (int& v : mem) v = enc(l - 1, v);
            mem.resize(mem.size() + 8);
            mptr.resize(mptr.size() + 8);
            e = upload(c, &E.mem, mem);
            if (e == cudaSuccess) e = upload(c, &E.mptr, mptr);
        }
    }
    if (e == cudaSuccess) e = upload(c, &c->tail, tail_levels<double>(c));
    return e == cudaSuccess ? FVGB_OK : cuda_fail(e, "multigrid setup");
}

fvgb_status symbolic(AmgCache* c, cudaStream_t s) {
    const fvgb_ls* ls = c->ls;
    const fvgb_mesh* mesh = ls->mesh;
    const int n = mesh->v.n, nnz = mesh->nnz;
    if ((int)mesh->h_row_offs.size() != n + 1 || (int)mesh->h_col.size() != nnz)
        return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: the mesh keeps no host sparsity pattern (device-built boxes)");
    // level 0 in CSR on the host: pattern from the mesh, values from the device
    std::vector<int> csr_pos(nnz);
    std::vector<double> slots(mesh->m_len);
    FVGB_CUDA_TRY(cudaStreamSynchronize(s));
    FVGB_CUDA_TRY(cudaMemcpy(csr_pos.data(), mesh->csr_pos, sizeof(int) * nnz, cudaMemcpyDeviceToHost));
    FVGB_CUDA_TRY(cudaMemcpy(slots.data(), ls->values, sizeof(double) * mesh->m_len, cudaMemcpyDeviceToHost));
    HostCsr A;
    A.n = n;
    A.rp = mesh->h_row_offs;
    A.ci = mesh->h_col;
    A.v.resize(nnz);
    for (int k = 0; k < nnz; ++k) A.v[k] = slots[csr_pos[k]];
    c->lv.clear();
    c->lv.emplace_back();
    c->lv[0].n = n;
    c->lv[0].nnz = nnz;
    c->lv[0].slots = mesh->m_len;
    std::vector<int> slot_of = csr_pos;  // the current level's slot of each of its CSR entries
    std::vector<std::vector<int>> h_sptr(1), h_scol(1), h_agg, h_mptr, h_mem;  // of every level; members: of the next level's rows
    while ((int)c->lv.size() < kMaxLevels && A.n > kCoarseRows) {
        // two rounds of pairwise matching per level (double pairwise): the pairs
        // of the first round are matched again on their Galerkin matrix, so a
        // level has about a quarter of the rows and half as many levels are
        // needed
        std::vector<int> agg;
        int nc = pgm_aggregate(A.n, A.rp.data(), A.ci.data(), A.v.data(), agg);
        if (nc > 0.9 * A.n) break;
        if (nc > kCoarseRows) {
            HostCsr A1;
            std::vector<int> m1, e1, g1, s1, agg2;
            galerkin(A, agg, nc, A1, m1, e1, g1, s1);
            const int nc2 = pgm_aggregate(A1.n, A1.rp.data(), A1.ci.data(), A1.v.data(), agg2);
            if (nc2 <= 0.9 * nc) {
                for (int& a : agg) a = agg2[a];
                nc = nc2;
                // aggregates numbered by their lowest row again
                std::vector<int> renum(nc, -1);
                int k = 0;
                for (int& a : agg) {
                    if (renum[a] < 0) renum[a] = k++;
                    a = renum[a];
                }
            }
        }
        HostCsr Ac;
        std::vector<int> mptr, mem, gptr, gsrc;
        galerkin(A, agg, nc, Ac, mptr, mem, gptr, gsrc);
        Level& L = c->lv.back();
        for (int& k : gsrc) k = slot_of[k];  // the sums read the fine level's sliced-ELL slots
        cudaError_t e = upload(c, &L.agg, agg);
        if (e == cudaSuccess) e = upload(c, &L.mptr, mptr);
        if (e == cudaSuccess) e = upload(c, &L.mem, mem);
        if (e == cudaSuccess) e = upload(c, &L.gptr, gptr);
        if (e == cudaSuccess) e = upload(c, &L.gsrc, gsrc);
        if (e != cudaSuccess) return cuda_fail(e, "multigrid setup");
        {  // whole aggregates to blocks of k_resid_restrict
            std::vector<int> blk(1, 0);
            bool fits = true;
            for (int I = 0, m0 = 0; I < nc; ++I) {
                fits = fits && mptr[I + 1] - mptr[I] <= kT;
                if (mptr[I + 1] - m0 > kT || I - blk.back() >= kT) {
                    blk.push_back(I);
                    m0 = mptr[I];
                }
            }
            blk.push_back(nc);
            if (fits) {
                L.nblk = (int)blk.size() - 1;
                if ((e = upload(c, &L.blk, blk)) != cudaSuccess) return cuda_fail(e, "multigrid setup");
            }
        }
        L.nnz_next = (int)Ac.ci.size();
        Level C;
        C.n = Ac.n;
        C.nnz = (int)Ac.ci.size();
        // sliced ELL of the coarse matrix; gdst: the slot of each CSR entry
        const int ns = (Ac.n + 31) / 32;
        std::vector<int> sptr(ns + 1, 0);
        for (int sl = 0; sl < ns; ++sl) {
            int w = 0;
            for (int i = sl * 32; i < std::min(Ac.n, sl * 32 + 32); ++i) w = std::max(w, Ac.rp[i + 1] - Ac.rp[i]);
            sptr[sl + 1] = sptr[sl] + 32 * w;
        }
        std::vector<int> scol(sptr[ns]), gdst(C.nnz), dpos(Ac.n, -1);
        for (int i = 0; i < Ac.n; ++i) {
            const int base = sptr[i / 32] + (i & 31), w = (sptr[i / 32 + 1] - sptr[i / 32]) / 32;
            for (int k = 0; k < w; ++k) scol[base + 32 * k] = i;  // padding
            for (int k = Ac.rp[i]; k < Ac.rp[i + 1]; ++k) {
                const int pos = base + 32 * (k - Ac.rp[i]);
                scol[pos] = Ac.ci[k];
                gdst[k] = pos;
                if (Ac.ci[k] == i) dpos[i] = pos;
            }
        }
        for (int i = 0; i < Ac.n; ++i)
            if (dpos[i] < 0) return fvgb_fail(FVGB_ERR_INVALID_ARG, "multigrid: a coarse row without a diagonal entry");
        C.slots = std::max(1, sptr[ns]);
        e = upload(c, &L.gdst, gdst);
        std::vector<int> sptr_pad(sptr);
        sptr_pad.resize(sptr.size() + 8);  // k_tail copies whole 16-byte lines
        if (e == cudaSuccess) e = upload(c, &C.sptr, sptr_pad);
        if (e == cudaSuccess) e = upload(c, &C.scol, scol);
        if (e == cudaSuccess) e = upload(c, &C.dpos, dpos);
        if (e == cudaSuccess) e = dev_alloc(c, &C.val, (size_t)std::max(1, sptr[ns]));
        if (e == cudaSuccess) e = cudaMemset(C.val, 0, sizeof(double) * (size_t)std::max(1, sptr[ns]));
        if (e != cudaSuccess) return cuda_fail(e, "multigrid setup");
        c->lv.push_back(C);
        h_sptr.push_back(std::move(sptr));
        h_scol.push_back(std::move(scol));
        h_agg.push_back(std::move(agg));
        h_mptr.push_back(std::move(mptr));
        h_mem.push_back(std::move(mem));
        slot_of = std::move(gdst);
        A = std::move(Ac);
    }
    if (c->lv.size() < 2) return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: the system does not coarsen (too small?)");
    c->nc = c->lv.back().n;
    if (c->nc > 1024) return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: the coarsest level keeps above 1024 rows");
    for (size_t l = 0; l < c->lv.size(); ++l) {
        Level& L = c->lv[l];
        cudaError_t e = dev_alloc(c, &L.dinv, (size_t)L.n);
        if (e == cudaSuccess) e = dev_alloc(c, &L.x, (size_t)L.n);
        if (e == cudaSuccess) e = dev_alloc(c, &L.xo, (size_t)L.n);
        if (e == cudaSuccess) e = dev_alloc(c, &L.r, (size_t)L.n);
        if (e == cudaSuccess && l > 0) e = dev_alloc(c, &L.b, (size_t)L.n);
        if (e != cudaSuccess) return cuda_fail(e, "multigrid vectors");
    }
    if (fvgb_status ts = tail_setup(c, h_sptr, h_scol, h_agg, h_mptr, h_mem); ts != FVGB_OK) return ts;
    c->nblk = (int)grid_for(n, kT);
    cudaError_t e = dev_alloc(c, &c->ainv, (size_t)c->nc * c->nc + 4);  // k_tail copies whole 16-byte lines
    if (e == cudaSuccess) e = dev_alloc(c, &c->r, (size_t)n);
    if (e == cudaSuccess) e = dev_alloc(c, &c->p, (size_t)n);
    if (e == cudaSuccess) e = dev_alloc(c, &c->q, (size_t)n);
    if (e == cudaSuccess) e = dev_alloc(c, &c->z, (size_t)n);
    if (e == cudaSuccess) e = dev_alloc(c, &c->part, (size_t)c->nblk);
    if (e == cudaSuccess) e = dev_alloc(c, &c->st, 1);
    if (e == cudaSuccess) e = cudaMemset(c->st, 0, sizeof(AmgState));
    if (e != cudaSuccess) return cuda_fail(e, "multigrid vectors");
    FVGB_CUDA_TRY(settle_creation());
    return FVGB_OK;
}

fvgb_status numeric(AmgCache* c, cudaStream_t s) {
    const fvgb_ls* ls = c->ls;
    const MeshView m = ls->mesh->v;
    k_dinv_ell<<<grid_for(m.n, kT), kT, 0, s>>>(m, ls->values, c->lv[0].dinv);
    for (size_t l = 0; l + 1 < c->lv.size(); ++l) {
        const Level& F = c->lv[l];
        Level& C = c->lv[l + 1];
        const double* vf = l == 0 ? ls->values : F.val;
        k_galerkin<<<grid_for(C.nnz, kT), kT, 0, s>>>(C.nnz, F.gptr, F.gsrc, F.gdst, vf, C.val);
        k_dinv_csr<<<grid_for(C.n, kT), kT, 0, s>>>(C.n, C.dpos, C.val, C.dinv);
    }
    const Level& B = c->lv.back();
    k_dense<<<B.n, kT, 0, s>>>(B.n, SellRows{B.sptr, B.scol, B.val}, c->ainv);
    const int C = c->cluster;
    if (C > 1 && gj_smem(B.n, C) <= kGjMaxSmem) {
        cudaLaunchConfig_t lc{};
        cudaLaunchAttribute at = cluster_attr(C);
        lc.gridDim = dim3((unsigned)C);
        lc.blockDim = dim3(kGjThreads);
        lc.dynamicSmemBytes = gj_smem(B.n, C);
        lc.stream = s;
        lc.attrs = &at;
        lc.numAttrs = 1;
        FVGB_CUDA_TRY(cudaLaunchKernelEx(&lc, k_gauss_jordan_cluster, (int)B.n, c->ainv));
    } else {
        k_gauss_jordan<<<1, 1024, sizeof(double) * B.n, s>>>(B.n, c->ainv);
    }
    FVGB_LAUNCH_CHECK("multigrid numeric setup");
    c->version = ls->version;
    return FVGB_OK;
}

// FP32 copies of the level matrices, diagonals and coarsest inverse
fvgb_status to_f32(AmgCache* c, cudaStream_t s) {
    const fvgb_ls* ls = c->ls;
    if (!c->f32) {
        for (size_t l = 0; l < c->lv.size(); ++l) {
            Level& V = c->lv[l];
            cudaError_t e = dev_alloc(c, &V.valf, (size_t)V.slots);
            if (e == cudaSuccess) e = dev_alloc(c, &V.dinvf, (size_t)V.n);
            if (e == cudaSuccess) e = dev_alloc(c, &V.bf, (size_t)V.n);
            if (e == cudaSuccess) e = dev_alloc(c, &V.xf, (size_t)V.n);
            if (e == cudaSuccess) e = dev_alloc(c, &V.xof, (size_t)V.n);
            if (e == cudaSuccess) e = dev_alloc(c, &V.rf, (size_t)V.n);
            if (e != cudaSuccess) return cuda_fail(e, "multigrid FP32 copies");
        }
        cudaError_t e = dev_alloc(c, &c->ainvf, (size_t)c->nc * c->nc + 4);
        const std::vector<TailLevelT<float>> tl = tail_levels<float>(c);
        if (e == cudaSuccess) e = upload(c, &c->tailf, tl);
        if (e != cudaSuccess) return cuda_fail(e, "multigrid FP32 copies");
        c->f32 = true;
    }
    for (size_t l = 0; l < c->lv.size(); ++l) {
        const Level& V = c->lv[l];
        const double* src = l == 0 ? ls->values : V.val;
        k_to_float<<<grid_for(V.slots, kT), kT, 0, s>>>(V.slots, src, V.valf);
        k_to_float<<<grid_for(V.n, kT), kT, 0, s>>>(V.n, V.dinv, V.dinvf);
    }
    k_to_float<<<grid_for((int64_t)c->nc * c->nc, kT), kT, 0, s>>>((int64_t)c->nc * c->nc, c->ainv, c->ainvf);
    FVGB_LAUNCH_CHECK("multigrid FP32 copies");
    c->f32_version = ls->version;
    return FVGB_OK;
}

cudaError_t add_kernel(cudaGraph_t g, cudaGraphNode_t* node, cudaGraphNode_t* dep, void* func, unsigned grid,
                       unsigned block, void** args, unsigned smem = 0) {
    cudaKernelNodeParams kp{};
    kp.func = func;
    kp.gridDim = dim3(grid);
    kp.blockDim = dim3(block);
    kp.sharedMemBytes = smem;
    kp.kernelParams = args;
    kp.extra = nullptr;
    const bool has_dep = dep && *dep;  // a null predecessor node means: no dependency
    return cudaGraphAddKernelNode(node, g, has_dep ? dep : nullptr, has_dep ? 1 : 0, &kp);
}

// The V-cycle z = M r as a chain of kernel nodes after *prev: levels
// 0..t-1 one kernel per step, levels t..L-1 in the one-cluster tail.  T is
// the V-cycle's type; with T = float, level 0's b and x are FP32 copies the
// CG kernels write and z comes back as double.
template <class T>
struct VcycleArgs {
    std::vector<std::vector<void*>> args;
    std::vector<EllRowsT<T>> ell;
    std::vector<SellRowsT<T>> sell;
    std::vector<int> ns;
    std::vector<const T*> bs;
    std::vector<T*> outs;
    std::vector<T*> xcs;
    std::vector<T*> dv, xv, rv, bv;
    int nl_tail = 0;
    const TailLevelT<T>* tail = nullptr;
    const T* ainv = nullptr;
};

template <class T> const T* ainv_of(const AmgCache* c);
template <> const double* ainv_of<double>(const AmgCache* c) { return c->ainv; }
template <> const float* ainv_of<float>(const AmgCache* c) { return c->ainvf; }
template <class T> const TailLevelT<T>* tail_of(const AmgCache* c);
template <> const TailLevelT<double>* tail_of<double>(const AmgCache* c) { return c->tail; }
template <> const TailLevelT<float>* tail_of<float>(const AmgCache* c) { return c->tailf; }

// r_in: level 0's b (double* for T = double; the FP32 copy otherwise).
// z_out: the result (always double).  first_sweep_done: level 0's x was
// formed by the kernel that produced r_in.  h: inside the CG's loop; the last sweep
// then forms beta and sets the loop's condition (k_post_rz).
template <class T>
cudaError_t add_vcycle(AmgCache* c, cudaGraph_t g, cudaGraphNode_t* prev, const T* r_in, double* z_out,
                       VcycleArgs<T>& va, bool first_sweep_done = false, cudaGraphConditionalHandle* h = nullptr) {
    const size_t L = c->lv.size();
    const size_t t = (size_t)c->tail_from;
    if (!first_sweep_done && !std::is_same<T, double>::value) return cudaErrorInvalidValue;  // FP64 only
    va.ell.assign(1, EllRowsT<T>{c->ls->mesh->v, c->lv[0].vals<T>() ? c->lv[0].vals<T>() : nullptr});
    if (std::is_same<T, double>::value) va.ell[0].val = (const T*)c->ls->values;
    va.sell.resize(L);
    for (size_t l = 1; l < L; ++l) va.sell[l] = SellRowsT<T>{c->lv[l].sptr, c->lv[l].scol, c->lv[l].vals<T>()};
    va.ns.resize(L);
    va.bs.resize(L);
    va.outs.resize(L);
    va.xcs.resize(L);
    va.dv.resize(L);
    va.xv.resize(L);
    va.rv.resize(L);
    va.bv.resize(L);
    va.args.clear();
    va.args.reserve(6 * L + 4);
    for (size_t l = 0; l < L; ++l) {
        const Level& V = c->lv[l];
        va.ns[l] = V.n;
        va.bs[l] = l == 0 ? r_in : V.bs<T>();
        va.outs[l] = V.xos<T>();
        va.dv[l] = V.dinvs<T>();
        va.xv[l] = V.xs<T>();
        va.rv[l] = V.rs<T>();
        va.bv[l] = V.bs<T>();
    }
    va.nl_tail = (int)(L - t);
    va.tail = tail_of<T>(c);
    va.ainv = ainv_of<T>(c);
    double* z = z_out;
    cudaError_t e = cudaSuccess;
    cudaGraphNode_t node;
    auto add = [&](void* fn, unsigned grid, unsigned block, unsigned smem = 0) {
        if (e != cudaSuccess) return;
        e = add_kernel(g, &node, prev, fn, grid, block, va.args.back().data(), smem);
        if (e == cudaSuccess) *prev = node;
    };
    for (size_t l = 0; l < t && e == cudaSuccess; ++l) {  // down
        Level& F = c->lv[l];
        if (l == 0) {
            if (!first_sweep_done) {  // the solve's CG kernels form x0 = w D^-1 r themselves
                va.args.push_back({&c->st, &va.ns[0], &F.dinv, &va.bs[0], &F.x});
                add((void*)k_smooth0, grid_for(F.n, kT), kT);
            }
        }
        Level& C = c->lv[l + 1];
        if (F.blk) {
            if (l == 0)
                va.args.push_back({&c->st, &va.ell[0], &F.blk, &va.bs[0], &va.xv[0], &F.mptr, &F.mem, &va.dv[1], &va.bv[1], &va.xv[1]});
            else
                va.args.push_back({&c->st, &va.sell[l], &F.blk, &va.bs[l], &va.xv[l], &F.mptr, &F.mem, &va.dv[l + 1],
                                   &va.bv[l + 1], &va.xv[l + 1]});
            add(l == 0 ? (void*)k_resid_restrict<EllRowsT<T>, T> : (void*)k_resid_restrict<SellRowsT<T>, T>,
                (unsigned)F.nblk, kT);
            continue;
        }
        if (l == 0) {
            va.args.push_back({&c->st, &va.ell[0], &va.ns[0], &va.bs[0], &va.xv[0], &va.rv[0]});
            add((void*)k_resid<EllRowsT<T>, T>, grid_for(F.n, kT), kT);
        } else {
            va.args.push_back({&c->st, &va.sell[l], &va.ns[l], &va.bs[l], &va.xv[l], &va.rv[l]});
            add((void*)k_resid<SellRowsT<T>, T>, grid_for(F.n, kT), kT);
        }
        va.args.push_back({&c->st, &va.ns[l + 1], &F.mptr, &F.mem, &va.rv[l], &va.dv[l + 1], &va.bv[l + 1], &va.xv[l + 1]});
        add((void*)k_restrict<T>, grid_for(C.n, kT), kT);
    }
    va.args.push_back({&c->st, &va.tail, &c->tail_parts, &va.nl_tail, &va.ainv});
    add((void*)k_tail<T>, (unsigned)c->cluster, kTailThreads, (unsigned)c->tail_smem);
    if (e == cudaSuccess) {
        cudaLaunchAttributeValue av{};
        av.clusterDim.x = (unsigned)c->cluster;
        av.clusterDim.y = av.clusterDim.z = 1;
        e = cudaGraphKernelNodeSetAttribute(*prev, cudaLaunchAttributeClusterDimension, &av);
    }
    for (size_t l = t; l-- > 0 && e == cudaSuccess;) {  // up
        Level& F = c->lv[l];
        va.xcs[l] = va.outs[l + 1];
        if (l == 0 && h && F.n <= kFusedPostRows) {
            va.args.push_back({&c->st, &va.ell[0], &va.ns[l], &va.dv[l], &va.bs[l], &va.xv[l], &va.xcs[l], &F.agg, &z, &c->r,
                               &c->part, h});
            add((void*)k_post_rz<EllRowsT<T>, T, true>, grid_for(F.n, kT), kT);
        } else if (l == 0) {
            va.args.push_back({&c->st, &va.ns[l], &va.xv[l], &va.xcs[l], &F.agg, &va.rv[l]});  // y = x + P xc
            add((void*)k_prolong<T>, grid_for(F.n, kT), kT);
            if (h) {
                va.args.push_back({&c->st, &va.ell[0], &va.ns[l], &va.dv[l], &va.bs[l], &va.rv[l], &va.xcs[l], &F.agg, &z, &c->r,
                                   &c->part, h});
                add((void*)k_post_rz<EllRowsT<T>, T, false>, grid_for(F.n, kT), kT);
            } else {
                va.args.push_back({&c->st, &va.ell[0], &va.ns[l], &va.dv[l], &va.bs[l], &va.rv[l], &z});
                add((void*)k_post<EllRowsT<T>, T, double>, grid_for(F.n, kT), kT);
            }
        } else {
            va.args.push_back({&c->st, &va.sell[l], &va.ns[l], &va.dv[l], &va.bs[l], &va.xv[l], &va.xcs[l], &F.agg,
                               &va.outs[l]});
            add((void*)k_post_fused<T>, grid_for(F.n, kT), kT);
        }
    }
    return e;
}

fvgb_status build_graph(AmgCache* c, bool f32) {
    cudaGraphExec_t& out = f32 ? c->graph32 : c->graph;
    if (out) {
        cudaGraphExecDestroy(out);
        out = nullptr;
    }
    const fvgb_ls* ls = c->ls;
    EllRows A{ls->mesh->v, ls->values};
    int n = ls->mesh->v.n;
    const unsigned nb = (unsigned)c->nblk;
    const double* b = ls->rhs;
    cudaGraph_t g = nullptr;
    FVGB_CUDA_TRY(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
    cudaGraphNode_t prev = nullptr, node;
    VcycleArgs<double> v0, v1;
    VcycleArgs<float> f0, f1;
    // FP64 V-cycle: the CG kernels write x0 (double); FP32: b0 and x0 as float
    double* x0 = f32 ? nullptr : c->lv[0].x;
    const float* d0f = f32 ? c->lv[0].dinvf : nullptr;
    float* b0f = f32 ? c->lv[0].bf : nullptr;
    float* x0f = f32 ? c->lv[0].xf : nullptr;
    // FP32: k_init forms no sweep (its norm is not known yet), k_first_f32 follows it
    float* nof = nullptr;
    void* a_init[] = {&c->st, &A, &n, &b, &c->r, &c->part, &c->lv[0].dinv, &x0, &d0f, f32 ? &nof : &b0f, &x0f};
    void* a_f32[] = {&c->st, &n, &c->r, &d0f, &b0f, &x0f};
    void* a_first[] = {&c->st, &n, &c->r, &c->z, &c->p, &c->part};
    void* a_cond[] = {&c->st, &h};
    void* a_spmv[] = {&c->st, &A, &n, &c->p, &c->q, &c->part};
    void* a_upd[] = {&c->st, &n, &c->p, &c->q, &c->r, &c->part, &c->lv[0].dinv, &x0, &d0f, &b0f, &x0f};
    void* a_dir[] = {&c->st, &n, &c->z, &c->p};
    void* a_stats[] = {&c->st};
    void* a_bnorm[] = {&c->st, &n, &b, &c->part};
    if (e == cudaSuccess) e = add_kernel(g, &node, nullptr, (void*)k_bnorm, nb, kT, a_bnorm);
    prev = node;
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_init, nb, kT, a_init);
    prev = node;
    if (e == cudaSuccess && f32) {
        e = add_kernel(g, &node, &prev, (void*)k_first_f32, nb, kT, a_f32);
        prev = node;
    }
    if (e == cudaSuccess)
        e = f32 ? add_vcycle<float>(c, g, &prev, b0f, c->z, f0, true) : add_vcycle<double>(c, g, &prev, c->r, c->z, v0, true);
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_first_dir, nb, kT, a_first);
    prev = node;
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_cond, 1, 1, a_cond);
    prev = node;
    cudaGraph_t body = nullptr;
    if (e == cudaSuccess) {
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        e = cudaGraphAddNode(&node, g, &prev, nullptr, 1, &np);
        if (e == cudaSuccess) body = np.conditional.phGraph_out[0];
        prev = node;
    }
    cudaGraphNode_t bprev = nullptr, bnode;
    if (e == cudaSuccess) e = add_kernel(body, &bnode, nullptr, (void*)k_spmv, nb, kT, a_spmv);
    bprev = bnode;
    if (e == cudaSuccess) e = add_kernel(body, &bnode, &bprev, (void*)k_update, nb, kT, a_upd);
    bprev = bnode;
    if (e == cudaSuccess)
        e = f32 ? add_vcycle<float>(c, body, &bprev, b0f, c->z, f1, true, &h)
                : add_vcycle<double>(c, body, &bprev, c->r, c->z, v1, true, &h);
    if (e == cudaSuccess) e = add_kernel(body, &bnode, &bprev, (void*)k_dir, nb, kT, a_dir);
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_stats, 1, 1, a_stats);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "multigrid CG graph");
    return FVGB_OK;
}

// The standalone multigrid solve as one graph: k_init, then a device-side
// while loop over {V-cycle, x += z, r = b - A x}, bounded by max_iter.
fvgb_status build_graph_mg(AmgCache* c, bool f32) {
    cudaGraphExec_t& out = c->graph_mg[f32 ? 1 : 0];
    if (out) {
        cudaGraphExecDestroy(out);
        out = nullptr;
    }
    const fvgb_ls* ls = c->ls;
    EllRows A{ls->mesh->v, ls->values};
    int n = ls->mesh->v.n;
    const unsigned nb = (unsigned)c->nblk;
    const double* b = ls->rhs;
    cudaGraph_t g = nullptr;
    FVGB_CUDA_TRY(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
    cudaGraphNode_t prev = nullptr, node;
    VcycleArgs<double> v1;
    VcycleArgs<float> f1;
    double* x0 = f32 ? nullptr : c->lv[0].x;
    const float* d0f = f32 ? c->lv[0].dinvf : nullptr;
    float* b0f = f32 ? c->lv[0].bf : nullptr;
    float* x0f = f32 ? c->lv[0].xf : nullptr;
    float* nof = nullptr;
    void* a_init[] = {&c->st, &A, &n, &b, &c->r, &c->part, &c->lv[0].dinv, &x0, &d0f, f32 ? &nof : &b0f, &x0f};
    void* a_f32[] = {&c->st, &n, &c->r, &d0f, &b0f, &x0f};
    void* a_cond[] = {&c->st, &h};
    void* a_add[] = {&c->st, &n, &c->z};
    void* a_res[] = {&c->st, &A, &n, &b, &c->r, &c->part, &c->lv[0].dinv, &x0, &d0f, &b0f, &x0f};
    void* a_stats[] = {&c->st};
    void* a_bnorm[] = {&c->st, &n, &b, &c->part};
    if (e == cudaSuccess) e = add_kernel(g, &node, nullptr, (void*)k_bnorm, nb, kT, a_bnorm);
    prev = node;
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_init, nb, kT, a_init);
    prev = node;
    if (e == cudaSuccess && f32) {
        e = add_kernel(g, &node, &prev, (void*)k_first_f32, nb, kT, a_f32);
        prev = node;
    }
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_cond, 1, 1, a_cond);
    prev = node;
    cudaGraph_t body = nullptr;
    if (e == cudaSuccess) {
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        e = cudaGraphAddNode(&node, g, &prev, nullptr, 1, &np);
        if (e == cudaSuccess) body = np.conditional.phGraph_out[0];
        prev = node;
    }
    cudaGraphNode_t bprev = nullptr, bnode;
    if (e == cudaSuccess)
        e = f32 ? add_vcycle<float>(c, body, &bprev, b0f, c->z, f1, true)
                : add_vcycle<double>(c, body, &bprev, c->r, c->z, v1, true);
    if (e == cudaSuccess) e = add_kernel(body, &bnode, &bprev, (void*)k_mg_add, nb, kT, a_add);
    bprev = bnode;
    if (e == cudaSuccess) e = add_kernel(body, &bnode, &bprev, (void*)k_mg_resid, nb, kT, a_res);
    bprev = bnode;
    if (e == cudaSuccess) e = add_kernel(body, &bnode, &bprev, (void*)k_cond, 1, 1, a_cond);
    if (e == cudaSuccess) e = add_kernel(g, &node, &prev, (void*)k_stats, 1, 1, a_stats);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "multigrid solver graph");
    return FVGB_OK;
}

fvgb_status prepare(fvgb_ls* ls, cudaStream_t s, bool f32 = false) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    FVGB_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
    if (!ls->amg) {
        if (cs != cudaStreamCaptureStatusNone)
            return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: the first solve (setup) cannot be stream-captured");
        AmgCache* c = new AmgCache();
        c->ls = ls;
        fvgb_status st = symbolic(c, s);
        if (st == FVGB_OK) st = build_graph(c, false);
        if (st != FVGB_OK) {
            fvgb_amg_free(c);
            return st;
        }
        ls->amg = c;
    }
    AmgCache* c = ls->amg;
    if (c->version != ls->version) {
        fvgb_status st = numeric(c, s);
        if (st != FVGB_OK) return st;
    }
    if (f32) {
        // the first FP32 V-cycle allocates its copies, uploads their descriptors and
        // builds its graph: none of that may happen inside a caller's capture
        if (!c->f32 && cs != cudaStreamCaptureStatusNone)
            return fvgb_fail(FVGB_ERR_UNSUPPORTED,
                             "multigrid: the first mixed-precision solve (FP32 setup) cannot be stream-captured");
        if (!c->f32 || c->f32_version != ls->version) {
            const bool first = !c->f32;
            fvgb_status st = to_f32(c, s);
            if (st != FVGB_OK) return st;
            if (first) {
                FVGB_CUDA_TRY(cudaStreamSynchronize(s));
                st = build_graph(c, true);
                if (st != FVGB_OK) return st;
            }
        }
    }
    return FVGB_OK;
}

}  // namespace

void fvgb_amg_free(AmgCache* c) {
    if (!c) return;
    if (c->graph) cudaGraphExecDestroy(c->graph);
    if (c->graph32) cudaGraphExecDestroy(c->graph32);
    for (cudaGraphExec_t g : c->graph_mg)
        if (g) cudaGraphExecDestroy(g);
    for (void* p : c->allocs) cudaFree(p);
    delete c;
}

fvgb_status fvgb_amg_solve_async(fvgb_ls* ls, double* x, const fvgb_solver_cfg* cfg, fvgb_solver_stats* stats_dev,
                                 cudaStream_t s) {
    if (ls->ncomp != 1) return fvgb_fail(FVGB_ERR_INVALID_ARG, "fvgb_solve: scalar systems only");
    const bool standalone = cfg->method == FVGB_SOLVER_MULTIGRID;
    if (cfg->method != FVGB_SOLVER_CG && !standalone)
        return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: as the preconditioner of CG only");
    FVGB_CHECK_ARG(cfg->precision == FVGB_PREC_FP64 || cfg->precision == FVGB_PREC_MIXED_IR,
                   "fvgb_solve: unknown precision");
    FVGB_CHECK_ARG(cfg->rel_tol >= 0 && cfg->abs_tol >= 0, "fvgb_solve: negative tolerance");
    FVGB_CHECK_ARG(cfg->max_iter >= 0 && cfg->max_iter <= 100000000, "fvgb_solve: bad max_iter");
    FVGB_CHECK_ARG((cfg->flags & ~(FVGB_SOLVE_NO_TUNE | FVGB_SOLVE_RHS_BASELINE)) == 0, "fvgb_solve: unknown flags");
    // mixed precision: the CG (or the multigrid iteration), its residuals and
    // its stopping test stay FP64; the V-cycle runs in FP32
    const bool f32 = cfg->precision == FVGB_PREC_MIXED_IR;
    fvgb_status st = prepare(ls, s, f32);
    if (st != FVGB_OK) return st;
    AmgCache* c = ls->amg;
    if (standalone && !c->graph_mg[f32 ? 1 : 0]) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        FVGB_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
        if (cs != cudaStreamCaptureStatusNone)
            return fvgb_fail(FVGB_ERR_UNSUPPORTED, "multigrid: the first solve of the multigrid solver cannot be stream-captured");
        st = build_graph_mg(c, f32);
        if (st != FVGB_OK) return st;
    }
    k_params<<<1, 1, 0, s>>>(c->st, x, cfg->rel_tol, cfg->abs_tol, cfg->max_iter, stats_dev,
                             (cfg->flags & FVGB_SOLVE_RHS_BASELINE) ? 1 : 0);
    FVGB_LAUNCH_CHECK("multigrid params");
    FVGB_CUDA_TRY(cudaGraphLaunch(standalone ? c->graph_mg[f32 ? 1 : 0] : (f32 ? c->graph32 : c->graph), s));
    return FVGB_OK;
}

fvgb_status fvgb_amg_sync_stats(fvgb_ls* ls, fvgb_solver_stats* out, cudaStream_t s) {
    AmgCache* c = ls->amg;
    fvgb_solver_stats h{};
    FVGB_CUDA_TRY(cudaMemcpyAsync(&h, &c->st->stats, sizeof h, cudaMemcpyDeviceToHost, s));
    FVGB_CUDA_TRY(cudaStreamSynchronize(s));
    if (out) *out = h;
    return (fvgb_status)(h.status == FVGB_ERR_NOT_CONVERGED ? FVGB_ERR_NOT_CONVERGED
                                                             : (h.status == FVGB_OK ? FVGB_OK : h.status));
}

extern "C" fvgb_status fvgb_amg_apply(fvgb_ls* ls, const double* r, double* z, fvgb_stream stream) {
    FVGB_CHECK_ARG(ls && r && z, "fvgb_amg_apply: null argument");
    FVGB_CHECK_ARG(ls->ncomp == 1, "fvgb_amg_apply: scalar systems only");
    cudaStream_t s = (cudaStream_t)stream;
    fvgb_status st = prepare(ls, s);
    if (st != FVGB_OK) return st;
    AmgCache* c = ls->amg;
    // a one-off graph of the V-cycle alone, with the done flag cleared
    k_params<<<1, 1, 0, s>>>(c->st, nullptr, 0.0, 0.0, 0, nullptr, 0);
    cudaGraph_t g = nullptr;
    FVGB_CUDA_TRY(cudaGraphCreate(&g, 0));
    cudaGraphNode_t prev = nullptr;
    VcycleArgs<double> va;
    cudaError_t e = add_vcycle<double>(c, g, &prev, r, z, va);
    cudaGraphExec_t ge = nullptr;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&ge, g, 0);
    if (e == cudaSuccess) e = cudaGraphLaunch(ge, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (ge) cudaGraphExecDestroy(ge);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "fvgb_amg_apply");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_amg_info(fvgb_ls* ls, int32_t* nlevels, int32_t* rows, int64_t* nnz, int32_t cap) {
    FVGB_CHECK_ARG(ls && nlevels, "fvgb_amg_info: null argument");
    if (!ls->amg) return fvgb_fail(FVGB_ERR_INVALID_ARG, "fvgb_amg_info: no multigrid hierarchy yet (solve first)");
    const AmgCache* c = ls->amg;
    *nlevels = (int32_t)c->lv.size();
    for (int32_t l = 0; l < *nlevels && l < cap; ++l) {
        if (rows) rows[l] = c->lv[l].n;
        if (nnz) nnz[l] = c->lv[l].nnz;
    }
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_pgm_aggregate(int32_t n, const int32_t* row_offs, const int32_t* cols,
                                          const double* values, int32_t* agg, int32_t* n_coarse) {
    FVGB_CHECK_ARG(n >= 0 && row_offs && cols && values && agg && n_coarse, "fvgb_pgm_aggregate: null argument");
    std::vector<int> a;
    *n_coarse = pgm_aggregate(n, row_offs, cols, values, a);
    std::memcpy(agg, a.data(), sizeof(int32_t) * (size_t)n);
    return FVGB_OK;
}
