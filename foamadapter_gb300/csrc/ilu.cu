// ILU(0)-preconditioned CG and BiCGStab (FP64) for a single scalar system.
//
// OpenFOAM's DILU preconditioner maps, through FoamAdapter, to Ginkgo's
// preconditioner::Ilu with a factorization::ParIlu and reverse_apply false
// (src/compatibility/fvSolution.cpp:56-63; the reference's
// test/setup_advection case names it beside PBiCGStab).  ParIlu's fixed-point
// sweeps approach the ILU(0) factors of A's sparsity pattern, and Ginkgo runs
// them asynchronously (not reproducible on a GPU); this file forms those
// factors exactly, which makes the preconditioner deterministic:
//
//  * symbolic (host, once per system, from the mesh's CSR pattern): for every
//    entry (i,k) left of the diagonal the pairs of entries (i,j), (k,j) with
//    j > k in both rows (the IKJ update list), and the rows grouped by level
//    of the lower and of the upper triangle (a row's level is one more than
//    the highest level of the rows it depends on);
//  * factorization (device, inside every solve's graph, so it follows the
//    matrix): level by level, one thread per row, entries k ascending:
//    l_ik = a_ik / u_kk, then a_ij = fma(-l_ik, u_kj, a_ij) over the update
//    list.  On hex meshes (no three cells pairwise adjacent) only the diagonal
//    changes: OpenFOAM's DILU;
//  * application z = U^-1 L^-1 r: forward y_i = r_i - sum_k l_ik y_k, then
//    backward z_i = (y_i - sum_j u_ij z_j) / u_ii, each a single sweep over
//    the rows in level order, fma chains in column order.
//
// On hex meshes the factorization is a sweep over the rows like a triangular solve,
// elsewhere each of its levels is one kernel node of the solve's CUDA graph.  A sweep is
// one launch: rows in level order, each waiting (bounded) for the rows it depends on
// (the sweeps below).
// Every row is computed by the same operations in the same order as the
// sequential restatement (oracle/fvoracle.c or_ilu_*): the bits are those of
// the exact sequential factorization and solves.  A 128^3 box has 382 levels
// per triangle, which bound the sweeps' speed: one dependent row after another.
//
// CG and BiCGStab (right preconditioning) around it follow the Jacobi solvers'
// stopping rules; every dot product uses the solver's reduction tree (256
// threads of R rows, R = 8 from 2^15 rows, else 4; block tree; last-block
// final tree), so the oracle's restatements give the same bits.
#include <algorithm>
#include <cmath>
#include <queue>
#include <utility>
#include <vector>

#include "internal.cuh"

namespace {

constexpr int kT = 256;

struct IluState {
    double* x;
    double rel_tol, abs_tol;
    int32_t max_iter, want_bbase;
    double bbase;
    double res0, res, tol;
    double rz, alpha, beta;           // CG; BiCGStab's alpha and beta
    double rho, rho_prev, omega;      // BiCGStab
    int32_t iter, status, done, half;
    unsigned counter;
    unsigned ticket;      // the next part of a triangular sweep (0 between launches)
    int32_t sweep_abort;  // a sweep's wait ran out: the solve ends with FVGB_ERR_CUDA
    fvgb_solver_stats* stats_out;
    fvgb_solver_stats stats;
};

struct Csr {
    int n;
    const int* ro;
    const int* col;
    const int* dof;  // diagonal offset of every row
};

// Set by an earlier kernel, or by the last block of this one after every block has read
// it: a plain load, one request per SM (a volatile one goes to L2 from every warp).
__device__ __forceinline__ int done_flag(const IluState* st) { return st->done; }

// ------------------------------------------------------------ reduction tree
// Row j of this thread: the solver's tree layout.
__device__ __forceinline__ int tree_row(int R, int j) {
    return blockIdx.x * (kT * R) + (threadIdx.x >> 5) * (32 * R) + j * 32 + (threadIdx.x & 31);
}

// Block sum of one value per thread, in every thread; formed by a warp that differs from
// block to block (solver.cu, block_tree).
__device__ __forceinline__ double block_tree(double v, double* sm) {
    __shared__ double out;
    sm[threadIdx.x] = v;
    __syncthreads();
    if ((threadIdx.x >> 5) == (blockIdx.x & 7u)) {
        const int lane = threadIdx.x & 31;
        double s = sm[lane];
#pragma unroll
        for (int k = 1; k < kT / 32; ++k) s = s + sm[lane + 32 * k];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) out = s;
    }
    __syncthreads();
    return out;
}

__device__ __forceinline__ double final_tree(const double* part, int nb, double* sm) {
    double a = 0.0;
    for (int i = threadIdx.x; i < nb; i += kT) a = a + __ldcg(&part[i]);
    return block_tree(a, sm);
}

// true in the block that arrives last (the counter wraps back to 0)
__device__ __forceinline__ bool arrive_last(unsigned* counter) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    return last;
}

// Up to two tree dots of this launch: the block partials, then in the last
// block the totals (valid in thread 0).  Returns false outside the last block.
__device__ __forceinline__ bool tree_dots(IluState* st, double* pa, double* pb, double a, double b, int ndots,
                                          double* ta, double* tb) {
    __shared__ double sma[kT], smb[kT];
    const double ba = block_tree(a, sma);
    const double bb = ndots > 1 ? block_tree(b, smb) : 0.0;
    if (threadIdx.x == 0) {
        pa[blockIdx.x] = ba;
        if (ndots > 1) pb[blockIdx.x] = bb;
    }
    if (!arrive_last(&st->counter)) return false;
    *ta = final_tree(pa, gridDim.x, sma);
    if (ndots > 1) *tb = final_tree(pb, gridDim.x, smb);
    return true;
}

__device__ __forceinline__ double csr_row(const Csr& A, const double* __restrict__ a, const double* x, int i) {
    double s = 0.0;
    for (int e = __ldg(&A.ro[i]); e < __ldg(&A.ro[i + 1]); ++e) s = fma(__ldg(&a[e]), x[__ldg(&A.col[e])], s);
    return s;
}

// ------------------------------------------------------------ setup kernels
__global__ void k_il_params(IluState* st, double* x, double rel_tol, double abs_tol, int max_iter,
                            fvgb_solver_stats* out, int want_bbase) {
    st->x = x;
    st->rel_tol = rel_tol;
    st->abs_tol = abs_tol;
    st->max_iter = max_iter;
    st->want_bbase = want_bbase;
    st->bbase = -1.0;
    st->stats_out = out;
    st->counter = 0;
    st->ticket = 0;
    st->sweep_abort = 0;
    st->done = 0;
    st->half = 0;
    st->iter = 0;
    st->status = FVGB_OK;
}

// ||b|| when the solve asks for Ginkgo's default ResidualNorm baseline
__global__ void __launch_bounds__(kT)
    k_il_bnorm(IluState* st, int n, int R, const double* __restrict__ b, double* pa) {
    if (!st->want_bbase) return;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i < n) acc = fma(__ldg(&b[i]), __ldg(&b[i]), acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) st->bbase = sqrt(t);
}

// A's values in CSR order, into the matrix copy and the factor
__global__ void __launch_bounds__(kT)
    k_il_gather(int nnz, const int* __restrict__ csr_pos, const double* __restrict__ slots, double* __restrict__ a,
                double* __restrict__ lu) {
    const int k = blockIdx.x * kT + threadIdx.x;
    if (k < nnz) a[k] = lu[k] = __ldg(&slots[__ldg(&csr_pos[k])]);
}

// One level of the factorization: row i's entries left of the diagonal in
// column order, each dividing by the pivot of its row and updating row i.
__global__ void __launch_bounds__(kT)
    k_il_factor(Csr A, const int* __restrict__ rows, int cnt, const int* __restrict__ op_ptr,
                const int* __restrict__ op_f, const int* __restrict__ op_g, double* lu) {
    const int t = blockIdx.x * kT + threadIdx.x;
    if (t >= cnt) return;
    const int i = __ldg(&rows[t]);
    const int b = __ldg(&A.ro[i]), d = b + __ldg(&A.dof[i]);
    for (int e = b; e < d; ++e) {
        const int k = __ldg(&A.col[e]);
        const double l = lu[e] / __ldcg(&lu[__ldg(&A.ro[k]) + __ldg(&A.dof[k])]);
        lu[e] = l;
        for (int o = __ldg(&op_ptr[e]); o < __ldg(&op_ptr[e + 1]); ++o) {
            const int f = __ldg(&op_f[o]);
            lu[f] = fma(-l, __ldcg(&lu[__ldg(&op_g[o])]), lu[f]);
        }
    }
}

// ------------------------------------------------------ triangular sweeps
// One launch per triangle.  The rows are cut into parts, of consecutive rows or, where those
// would have levels of a few rows, by level from groups of consecutive rows (group_rows),
// one part to a block at a time, taken by a ticket in an order in which a row depends only
// on rows of its own part and of parts that running blocks took before, so every wait
// ends.
//
// What bounds a sweep is the chain of levels (197 of them for 77 x 64 x 58 cells, 382
// for 128^3).  Inside a part the levels follow one another through shared memory:
// teams of W warps take them in turn, a team fetches its next level's rows while the
// others have theirs, and hands the turn on by a named barrier.  Between parts a value
// goes through global memory: a row's output holds kPending until the row is computed,
// and the one 64-bit store of the value is the signal (relaxed at GPU scope, no flag and
// no fence).  kHaloWarps warps of the block bring the values that the part needs from
// others into shared memory, in the order in which its rows need them; on large systems
// (kDirectRows) the row warps read them themselves.
//
// BiCGStab on 77 x 64 x 58 cells: 6.1 -> 3.0 ms, on 20^3 1.41 -> 0.70, on 128^3 16.0 ->
// 11.4; before, every value went through L2 (1.6 us a level), and every level of the
// factorization was a kernel of dependent loads (2.2 of the 6.1 ms, now 0.4).  A level
// takes 0.4 us inside a part: the barrier 250 clocks, three dependent multiply-adds 200
// of GB300's FP64; a step to another part 1.3 us.  Rows that poll shared memory without
// a turn were slower: the polls of the waiting warps take the issue slots and the banks.
//
// kPending is a signalling NaN: FP64 arithmetic writes quiet NaNs at most, and every
// value a sweep writes is an arithmetic result.  The forward sweep sets the backward
// sweep's output to kPending row by row, the backward sweep the forward sweep's output
// after reading it; the solve graph fills the latter once at its start.
constexpr unsigned long long kPending = 0x7ff00000deadbeefull;
constexpr int kRowWarps = 16, kHaloWarps = 8;
constexpr int kSweepThreads = 32 * (kRowWarps + kHaloWarps);
constexpr int kMaxTeams = 8;   // named barriers 1 .. kMaxTeams
constexpr int kDeps = 4;       // values a row waits for together; the others one by one
// Rows of a part: few parts make few trips through L2, and a level of more than 128 rows
// leaves two teams, which fetch too late.  BiCGStab on 77 x 64 x 58 cells: 2.98 ms with
// parts of 8,192 rows, 3.45 with 4,096 (levels of up to 128 and 64 rows); on 20^3, 0.70 ms
// with 1,024 and 1.00 in one part (levels of up to 300).  A part of consecutive rows with
// fewer than kThinRows rows a level is too long a chain for its rows: ILU-CG iterations of
// 9000 x 90 x 9 cells 40.7 ms, with groups from 8 rows a level on 13.8, from 16 on 8.4;
// 2048^2 6.62, 4.61 and 4.07; 512^2 (15.5 rows) 0.86 either way.
constexpr int kPart = 8192, kMinPart = 1024, kLevelRows = 128, kThinRows = 16;
// From this size on the row warps read the rows of other parts themselves, before their
// turn: their reads are further ahead of need than the halo warps' when levels are wide.
// ILU-CG on 128^3 cells 162 ms with halo warps and 122 without (144 with every step
// through L2), 96^3 83.8 and 66.9, 64^3 21.5 and 18.3; BiCGStab on 40^3 1.42 and 1.48 ms,
// on 80 x 80 x 9 1.77 and 1.94.  The grid is then twice the SMs, of which one block each
// is resident (123.5 -> 120.0 ms on 128^3, which has 256 parts); without the idle halo
// warps two were, and it took 140.
constexpr int kDirectRows = 1 << 18;
constexpr int kMaxSweepSmem = (3 * kPart + 1) * (int)sizeof(double);

// A triangle's sweep.  Its rows stand at positions 0 .. n - 1, row rows[t] at position t,
// in the order of the parts, in a part by level: part p has the positions first[p] to
// first[p + 1] - 1 and the levels lev[p] to lev[p + 1] - 1, level q the positions
// start[q] to start[q + 1] - 1.  (Levels filled up to whole warps, for aligned loads, took
// 32 times the memory where a level has one row.)  A row's place in its part's shared
// memory is its position less the part's first.  Of the row at position t the values it
// depends on (k < K) are at slot[k n + t]: a place in the part's shared memory (its own
// rows, then what the halo warps bring), -1 none, below -1 the row -2 - slot read from
// global memory.  val[k n + t]: the factor's entries, filled in every solve; from
// val[K n + t] on the pivots and their reciprocals (backward) or the matrix's a_ki and
// a_ii (forward, where the factorization is a sweep: until it is done, and it reads the
// matrix's a_ik at val[k n + t]).
struct Sweep {
    int n, rpp, nparts, K, hcap, W;
    const int* rows;
    const int* first;
    const int* lev;
    const int* start;
    int* pos;    // [n] a row's position
    int* slot;
    double* val;
    int* halo;   // [nparts][hcap] rows of other parts
    int* nhalo;  // [nparts]
};

__device__ __forceinline__ bool pending(double v) { return (unsigned long long)__double_as_longlong(v) == kPending; }

__device__ __forceinline__ double ld_relaxed(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// Bounds of every wait.  The longest one that is no fault: a chain beside wider meshes, a
// part of 8,192 levels of 0.4 us on each of 152 SMs, each waiting for the one before, 0.5 s.
constexpr unsigned long long kWaitNs = 4000000000ull;
constexpr unsigned kWaitPolls = 1u << 28;

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The wait for a pending row value: false when the sweep is aborted, because
// this wait ran out or another one did.
__device__ __noinline__ bool await_pending(const double* p, double& v, IluState* st) {
    const unsigned long long t0 = now_ns();
    for (unsigned k = 1; k < kWaitPolls; ++k) {
        if (k > 2) __nanosleep(k < 16 ? 32 : 256);  // rows far from the wavefront poll less
        v = ld_relaxed(p);
        if (!pending(v)) return true;
        if ((k & 31) == 0) {
            if (*(volatile const int32_t*)&st->sweep_abort) return false;
            if (now_ns() - t0 > kWaitNs) break;
        }
    }
    atomicExch(&st->sweep_abort, 1);
    return false;
}

// Row value of this sweep at p (see await_pending)
__device__ __forceinline__ bool await_row(const double* p, double& v, IluState* st) {
    v = ld_relaxed(p);
    return !pending(v) || await_pending(p, v, st);
}

__global__ void __launch_bounds__(kT) k_il_pending(int n, double* y) {
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) y[i] = __longlong_as_double((long long)kPending);
}

// A value of the block's shared memory that another warp reads or writes; a: 32-bit address
__device__ __forceinline__ double ld_shared(unsigned a) {
    double v;
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared(unsigned a, double v) {
    asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__global__ void __launch_bounds__(kT) k_il_pos(Sweep S) {
    const int t = blockIdx.x * kT + threadIdx.x;
    if (t < S.n) S.pos[__ldg(&S.rows[t])] = t;
}

// Where the values that a part's rows depend on are found: one block per part.
template <bool BWD>
__global__ void __launch_bounds__(kT) k_il_plan(Csr A, Sweep S) {
    __shared__ int wsum[kT / 32], base;
    const int t0 = __ldg(&S.first[blockIdx.x]), t1 = __ldg(&S.first[blockIdx.x + 1]);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int q = t0; q < t1; q += kT) {
        const int t = q + threadIdx.x;
        int e0 = 0, e1 = 0, cnt = 0;
        if (t < t1) {
            const int i = __ldg(&S.rows[t]);
            const int d = __ldg(&A.ro[i]) + __ldg(&A.dof[i]);
            e0 = BWD ? d + 1 : __ldg(&A.ro[i]);
            e1 = min(BWD ? __ldg(&A.ro[i + 1]) : d, e0 + S.K);
            for (int e = e0; e < e1; ++e) {
                const int c = __ldg(&S.pos[__ldg(&A.col[e])]);
                cnt += c < t0 || c >= t1;
            }
        }
        int x = cnt;  // inclusive scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        int at = base + x - cnt;
        for (int k = 0; k < w; ++k) at += wsum[k];
        if (t < t1) {
            for (int k = 0; k < S.K; ++k) {
                int sl = -1;
                if (e0 + k < e1) {
                    const int r = __ldg(&A.col[e0 + k]), c = __ldg(&S.pos[r]);
                    if (c >= t0 && c < t1) {
                        sl = c - t0;
                    } else if (at < S.hcap) {
                        S.halo[(size_t)blockIdx.x * S.hcap + at] = r;
                        sl = S.rpp + at++;
                    } else {
                        sl = -2 - r;
                    }
                }
                S.slot[(size_t)k * S.n + t] = sl;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int k = 0; k < kT / 32; ++k) base += wsum[k];
        __syncthreads();
    }
    if (threadIdx.x == 0) S.nhalo[blockIdx.x] = min(base, S.hcap);
}

enum SweepKind { kFwd = 0, kBwd = 1, kFactor = 2 };

struct Factor {  // of the pivots alone: entry e of the lower triangle updates its row's by a[g[p[e]]]
    const double* a;
    double* lu;
    const int *p, *g;
};

// A factor's entries (kFwd, kBwd) or the matrix's (kFactor) in the order of a sweep.
// piv: the pivots row by row when the factorization was a sweep, else null.
template <int KIND>
__global__ void __launch_bounds__(kT) k_il_pack(Csr A, Sweep S, Factor F, const double* __restrict__ piv) {
    const int t = blockIdx.x * kT + threadIdx.x;
    if (t >= S.n) return;
    const int i = __ldg(&S.rows[t]);
    const int b = __ldg(&A.ro[i]), d = b + __ldg(&A.dof[i]);
    const int e0 = KIND == kBwd ? d + 1 : b, e1 = min(e0 + S.K, KIND == kBwd ? __ldg(&A.ro[i + 1]) : d);
    for (int e = e0; e < e1; ++e) {
        double* v = S.val + (size_t)(e - e0) * S.n + t;
        *v = KIND == kFactor ? __ldg(&F.a[e]) : F.lu[e];
        if (KIND == kFactor) v[(size_t)S.K * S.n] = __ldg(&F.a[__ldg(&F.g[__ldg(&F.p[e])])]);
    }
    if (KIND == kBwd) {
        const double u = piv ? piv[i] : F.lu[d];
        S.val[(size_t)S.K * S.n + t] = u;
        S.val[(size_t)(S.K + 1) * S.n + t] = 1.0 / u;
    }
    if (KIND == kFactor) S.val[(size_t)(2 * S.K) * S.n + t] = __ldg(&F.a[d]);
}

// Part of this block (the same in all its threads), or >= nparts when none is left.
__device__ __forceinline__ int next_part(IluState* st) {
    __shared__ unsigned part;
    __syncthreads();
    if (threadIdx.x == 0) part = atomicAdd(&st->ticket, 1u);
    __syncthreads();
    return (int)part;
}

// The last block resets the ticket and ends an aborted solve.
__device__ __forceinline__ void end_sweep(IluState* st) {
    if (arrive_last(&st->counter) && threadIdx.x == 0) {
        st->ticket = 0;
        if (st->sweep_abort) {
            st->status = FVGB_ERR_CUDA;
            st->done = 1;
        }
    }
}

// What a row needs besides the values it depends on, fetched before its turn.
// kFwd, kBwd: v the entries of the factor; kFactor: v = a_ik, w = a_ki, s = a_ii.
template <int K>
struct RowIn {
    int i, slot[K];
    double v[K], w[K], s, piv, rcp;
};

template <int KIND, int K>
__device__ __forceinline__ void fetch_row(const Sweep& S, const double* src, int t, int i, RowIn<K>& q) {
    q.i = i;
#pragma unroll
    for (int k = 0; k < K; ++k) q.slot[k] = i < 0 ? -1 : __ldg(&S.slot[(size_t)k * S.n + t]);
    q.s = q.piv = q.rcp = 1.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        q.v[k] = q.slot[k] == -1 ? 0.0 : S.val[(size_t)k * S.n + t];
        if (KIND == kFactor) q.w[k] = q.slot[k] == -1 ? 0.0 : S.val[(size_t)(K + k) * S.n + t];
    }
    if (i < 0) return;
    if (KIND == kFactor) {
        q.s = S.val[(size_t)(2 * K) * S.n + t];
    } else {
        q.s = __ldcg(&src[i]);
        if (KIND == kBwd) {
            q.piv = S.val[(size_t)K * S.n + t];
            q.rcp = S.val[(size_t)(K + 1) * S.n + t];
        }
    }
}

// a / b with y = 1 / b rounded to nearest (Markstein, IBM J. Res. Dev. 34, 1990): the
// first correction leaves a quotient within an ulp, the second rounds it correctly, as
// long as nothing over- or underflows.  Five dependent operations where the division
// takes about twice as many.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const unsigned ea = (unsigned)__double2hiint(a) & 0x7ff00000u, eb = (unsigned)__double2hiint(b) & 0x7ff00000u;
    const double q0 = a * y;
    const double q1 = fma(fma(-q0, b, a), y, q0);
    const double q2 = fma(fma(-q1, b, a), y, q1);
    // |a| zero or within 2^-600 .. 2^600, |b| within 2^-300 .. 2^300
    const bool zero = (unsigned long long)__double_as_longlong(a) << 1 == 0;
    if ((zero || ea - (423u << 20) <= (1200u << 20)) && eb - (723u << 20) <= (600u << 20)) return zero ? q0 : q2;
    return a / b;
}

// Waits for the value that a halo warp brings to the shared address a; after an abort it
// may not be there (the teams keep taking their turns, so that no barrier is left short).
__device__ __forceinline__ void await_halo(unsigned a, IluState* st) {
    unsigned long long t0 = 0;
    for (unsigned it = 1; pending(ld_shared(a)); ++it) {
        if ((it & 63) != 0) continue;
        if (it == 64) t0 = now_ns();
        if (*(volatile const int32_t*)&st->sweep_abort) break;
        if (it >= kWaitPolls || now_ns() - t0 > kWaitNs) {
            atomicExch(&st->sweep_abort, 1);
            break;
        }
    }
}

// Rows of one level:
//   kFwd     v_i = src_i - sum_k l_ik v_k
//   kBwd     v_i = (src_i - sum_j u_ij v_j) / u_ii
//   kFactor  l_ik = a_ik / v_k, v_i = a_ii - sum_k l_ik a_ki   (v the pivots)
// the sums in column order.  TURN: the level's turn is still to come; what other parts
// give is waited for before.  Values that are not there have v = 0 and the slot that
// holds +0: fma(-0, +0, s) is s.  Entries past the first K, and values for which shared
// memory had no room (neither on hex meshes), are waited for one by one in global memory.
template <int KIND, int K, bool DIRECT, bool TURN>
__device__ __forceinline__ double sweep_row(IluState* st, const Csr& A, const Sweep& S, const Factor& F,
                                            const double* lu, unsigned sm, RowIn<K>& q, const double* v, int turn,
                                            int count) {
    bool rare = K == kDeps && q.slot[K - 1] != -1;
    unsigned at[K];
    double x[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int sl = q.slot[k];
        at[k] = sm + 8u * (unsigned)(sl < 0 ? S.rpp + S.hcap : sl);
        if (DIRECT) {
            x[k] = 0.0;
            if (sl < -1) await_row(&v[-2 - sl], x[k], st);
        } else {
            rare = rare || sl < -1;
            if (sl >= S.rpp) await_halo(at[k], st);
        }
    }
    rare = __any_sync(0xffffffffu, rare);
    if (TURN) asm volatile("bar.sync %0, %1;" ::"r"(turn), "r"(count) : "memory");
    double s = q.s;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double y = ld_shared(at[k]);
        x[k] = DIRECT && q.slot[k] < -1 ? x[k] : y;
    }
    if (!DIRECT && rare) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (q.slot[k] < -1) {
                x[k] = 0.0;
                await_row(&v[-2 - q.slot[k]], x[k], st);
            }
    }
    if (KIND == kFactor) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (q.slot[k] != -1) q.v[k] = q.v[k] / x[k];
            x[k] = q.w[k];
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) s = fma(-q.v[k], x[k], s);
    if (rare && K == kDeps && q.slot[K - 1] != -1) {
        const int b = __ldg(&A.ro[q.i]), d = b + __ldg(&A.dof[q.i]);
        const int e1 = KIND == kBwd ? __ldg(&A.ro[q.i + 1]) : d;
        for (int e = (KIND == kBwd ? d + 1 : b) + kDeps; e < e1; ++e) {
            double xe = 1.0;
            await_row(&v[__ldg(&A.col[e])], xe, st);
            if (KIND == kFactor) {
                const double l = __ldg(&F.a[e]) / xe;
                F.lu[e] = l;
                s = fma(-l, __ldg(&F.a[__ldg(&F.g[__ldg(&F.p[e])])]), s);
            } else {
                s = fma(-__ldg(&lu[e]), xe, s);
            }
        }
    }
    return KIND == kBwd ? div_by(s, q.piv, q.rcp) : s;
}

// DIRECT: no halo (hcap 0), the row warps read the rows of other parts themselves.
// other_i = pending: the backward sweep's output (kFwd), src once read (kBwd).  A wait
// gives up, raising the abort flag, after kWaitNs (or kWaitPolls polls), or when
// another wait of the sweep did.
template <int KIND, int K, bool DIRECT>
__global__ void __launch_bounds__(kSweepThreads)
    k_il_sweep(IluState* st, Csr A, Sweep S, Factor F, const double* __restrict__ lu, const double* src, double* v,
               double* other) {
    extern __shared__ double smem[];
    const unsigned sm = (unsigned)__cvta_generic_to_shared(smem);
    if (KIND != kFactor && done_flag(st)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double unset = __longlong_as_double((long long)kPending);
    const int T = min(kMaxTeams, kRowWarps / S.W), count = 64 * S.W;
    if (threadIdx.x == 0) smem[S.rpp + S.hcap] = 0.0;
    for (int u = next_part(st); u < S.nparts; u = next_part(st)) {
        const int nh = __ldg(&S.nhalo[u]), t0 = __ldg(&S.first[u]);
        for (int k = threadIdx.x; k < nh; k += kSweepThreads) smem[S.rpp + k] = unset;
        __syncthreads();
        if (w >= kRowWarps) {
            const int* halo = S.halo + (size_t)u * S.hcap;
            for (int h = (w - kRowWarps) * 32 + lane; h < nh; h += 32 * kHaloWarps) {
                const double* p = &v[__ldg(&halo[h])];
                unsigned long long t0 = 0;
                for (unsigned it = 0;; ++it) {
                    const double x = ld_relaxed(p);
                    if (!pending(x)) {
                        st_shared(sm + 8u * (unsigned)(S.rpp + h), x);
                        break;
                    }
                    if (it == 0) t0 = now_ns();
                    if (it > 2) __nanosleep(20);
                    if ((it & 31) == 31) {
                        if (*(volatile const int32_t*)&st->sweep_abort) break;
                        if (it >= kWaitPolls || now_ns() - t0 > kWaitNs) {
                            atomicExch(&st->sweep_abort, 1);
                            break;
                        }
                    }
                }
            }
        } else if (w < T * S.W) {
            const int team = w / S.W, tw = w % S.W;
            const int l0 = __ldg(&S.lev[u]), l1 = __ldg(&S.lev[u + 1]);
            // positions [c, ce) of this warp's level, 32 at a time, the first fetched; [n, ne) of the one after, i the first's rows
            RowIn<K> q;
            int c, ce, n, ne, i = -1;
            const auto level = [&](int l, int& a, int& b) {
                a = b = 0;
                if (l < l1) {
                    a = __ldg(&S.start[l]) + 32 * tw;
                    b = __ldg(&S.start[l + 1]);
                }
            };
            const auto row = [&](int a, int b) { return a + lane < b ? __ldg(&S.rows[a + lane]) : -1; };
            level(l0 + team, c, ce);
            level(l0 + team + T, n, ne);
            if (c < ce) fetch_row<KIND>(S, src, c + lane, row(c, ce), q);
            if (n < ne) i = row(n, ne);
            for (int l = l0 + team; l < l1; l += T) {
                int n2, n2e;
                level(l + 2 * T, n2, n2e);
                const int turn = 1 + team, next = 1 + (team + 1) % T;
                if (c < ce) {
                    double z = l > l0 ? sweep_row<KIND, K, DIRECT, true>(st, A, S, F, lu, sm, q, v, turn, count)
                                      : sweep_row<KIND, K, DIRECT, false>(st, A, S, F, lu, sm, q, v, turn, count);
                    for (;;) {
                        const int t = c + lane;
                        if (q.i >= 0) st_shared(sm + 8u * (unsigned)(t - t0), z);
                        c += 32 * S.W;
                        if (c >= ce) {
                            __syncwarp();
                            if (l + 1 < l1)
                                asm volatile("bar.arrive %0, %1;" ::"r"(next), "r"(count) : "memory");
                        }
                        if (q.i >= 0) {
                            st_relaxed(&v[q.i], z);
                            if (KIND != kFactor) other[q.i] = unset;
                            if (KIND == kFactor) {
#pragma unroll
                                for (int k = 0; k < K; ++k)
                                    if (q.slot[k] != -1) S.val[(size_t)k * S.n + t] = q.v[k];
                            }
                        }
                        if (c >= ce) break;
                        fetch_row<KIND>(S, src, c + lane, row(c, ce), q);
                        z = sweep_row<KIND, K, DIRECT, false>(st, A, S, F, lu, sm, q, v, 0, 0);
                    }
                } else {
                    if (l > l0) asm volatile("bar.sync %0, %1;" ::"r"(turn), "r"(count) : "memory");
                    if (l + 1 < l1) asm volatile("bar.arrive %0, %1;" ::"r"(next), "r"(count) : "memory");
                }
                c = n;
                ce = ne;
                n = n2;
                ne = n2e;
                if (c < ce) fetch_row<KIND>(S, src, c + lane, i, q);
                if (n < ne) i = row(n, ne);
            }
        }
    }
    end_sweep(st);
}

// The tolerance and the first stopping test from the initial residual norm
__device__ void start(IluState* st, double res) {
    st->res0 = st->res = res;
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

// the stopping tests after an iteration's residual norm
__device__ void after_step(IluState* st, double res) {
    st->res = res;
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

// ------------------------------------------------------------ CG
// r = b - A x, |r|
__global__ void __launch_bounds__(kT)
    k_ic_init(IluState* st, Csr A, int R, const double* __restrict__ a, const double* __restrict__ b,
              double* __restrict__ r, double* pa) {
    const double* x = st->x;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= A.n) continue;
        const double ri = __ldg(&b[i]) - csr_row(A, a, x, i);
        r[i] = ri;
        acc = fma(ri, ri, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) start(st, sqrt(t));
}

// p = z, rz = (r, z)
__global__ void __launch_bounds__(kT)
    k_ic_first(IluState* st, int n, int R, const double* __restrict__ r, const double* __restrict__ z,
               double* __restrict__ p, double* pa) {
    if (done_flag(st)) return;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= n) continue;
        const double zi = z[i];
        p[i] = zi;
        acc = fma(r[i], zi, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) st->rz = t;
}

// q = A p, alpha = rz / (p, q)
__global__ void __launch_bounds__(kT)
    k_ic_spmv(IluState* st, Csr A, int R, const double* __restrict__ a, const double* __restrict__ p,
              double* __restrict__ q, double* pa) {
    if (done_flag(st)) return;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= A.n) continue;
        const double qi = csr_row(A, a, p, i);
        q[i] = qi;
        acc = fma(__ldg(&p[i]), qi, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) {
        const double alpha = st->rz / t;
        st->alpha = alpha;
        if (t == 0.0 || !isfinite(alpha)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
    }
}

// x += alpha p, r -= alpha q, |r|, stopping tests
__global__ void __launch_bounds__(kT)
    k_ic_update(IluState* st, int n, int R, const double* __restrict__ p, const double* __restrict__ q,
                double* __restrict__ r, double* pa) {
    if (done_flag(st)) return;
    const double alpha = st->alpha;
    double* x = st->x;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= n) continue;
        x[i] = fma(alpha, __ldg(&p[i]), x[i]);
        const double ri = fma(-alpha, __ldg(&q[i]), r[i]);
        r[i] = ri;
        acc = fma(ri, ri, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) after_step(st, sqrt(t));
}

// beta = (r, z) / rz
__global__ void __launch_bounds__(kT)
    k_ic_rz(IluState* st, int n, int R, const double* __restrict__ r, const double* __restrict__ z, double* pa) {
    if (done_flag(st)) return;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i < n) acc = fma(__ldg(&r[i]), __ldg(&z[i]), acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) {
        st->beta = t / st->rz;
        st->rz = t;
    }
}

// p = z + beta p
__global__ void __launch_bounds__(kT)
    k_ic_dir(const IluState* st, int n, const double* __restrict__ z, double* __restrict__ p) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i < n) p[i] = fma(st->beta, p[i], __ldg(&z[i]));
}

// ------------------------------------------------------------ BiCGStab
// r = b - A x, rr = r, p = v = 0, rho = (rr, r), |r|; rho_prev = alpha = omega = 1
__global__ void __launch_bounds__(kT)
    k_ib_init(IluState* st, Csr A, int R, const double* __restrict__ a, const double* __restrict__ b,
              double* __restrict__ r, double* __restrict__ rr, double* __restrict__ p, double* __restrict__ v,
              double* pa, double* pb) {
    const double* x = st->x;
    double arho = 0.0, arr = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= A.n) continue;
        const double ri = __ldg(&b[i]) - csr_row(A, a, x, i);
        r[i] = ri;
        rr[i] = ri;
        p[i] = 0.0;
        v[i] = 0.0;
        arho = fma(ri, ri, arho);
        arr = fma(ri, ri, arr);
    }
    double rho, rsq;
    if (tree_dots(st, pa, pb, arho, arr, 2, &rho, &rsq) && threadIdx.x == 0) {
        st->rho = rho;
        st->rho_prev = st->alpha = st->omega = 1.0;
        st->beta = rho;
        start(st, sqrt(rsq));
    }
}

// p = r + beta (p - omega v), beta = (rho / rho_prev)(alpha / omega) from the kernel that
// formed rho (its two divisions in every thread here: 11.7 us for 285,824 rows, now 2.5)
__global__ void __launch_bounds__(kT)
    k_ib_p(const IluState* st, int n, const double* __restrict__ r, const double* __restrict__ v,
           double* __restrict__ p) {
    if (done_flag(st)) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    if (i >= n) return;
    const double beta = st->beta;
    p[i] = fma(beta, fma(-st->omega, __ldg(&v[i]), p[i]), __ldg(&r[i]));
}

// v = A y, alpha = rho / (rr, v)
__global__ void __launch_bounds__(kT)
    k_ib_v(IluState* st, Csr A, int R, const double* __restrict__ a, const double* __restrict__ y,
           const double* __restrict__ rr, double* __restrict__ v, double* pa) {
    if (done_flag(st)) return;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= A.n) continue;
        const double vi = csr_row(A, a, y, i);
        v[i] = vi;
        acc = fma(__ldg(&rr[i]), vi, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) {
        const double alpha = st->rho / t;
        st->alpha = alpha;
        if (t == 0.0 || !isfinite(alpha)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
    }
}

// s = r - alpha v, |s|: converged at the half step (x += alpha y follows in k_ib_half)
__global__ void __launch_bounds__(kT)
    k_ib_s(IluState* st, int n, int R, const double* __restrict__ r, const double* __restrict__ v,
           double* __restrict__ s, double* pa) {
    if (done_flag(st)) return;
    const double alpha = st->alpha;
    double acc = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= n) continue;
        const double si = fma(-alpha, __ldg(&v[i]), __ldg(&r[i]));
        s[i] = si;
        acc = fma(si, si, acc);
    }
    double t, u;
    if (tree_dots(st, pa, nullptr, acc, 0.0, 1, &t, &u) && threadIdx.x == 0) {
        const double sres = sqrt(t);
        if (!isfinite(sres)) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->res = sres;
            st->done = 1;
        } else if (!(sres > st->tol)) {
            st->res = sres;
            st->iter += 1;
            st->half = 1;
            st->done = 1;
        }
    }
}

// the half-step convergence's x += alpha y (runs whatever the done flag)
__global__ void __launch_bounds__(kT) k_ib_half(IluState* st, int n, const double* __restrict__ y) {
    if (!st->half) return;
    const int i = blockIdx.x * kT + threadIdx.x;
    double* x = st->x;
    if (i < n) x[i] = fma(st->alpha, __ldg(&y[i]), x[i]);
}

// t = A z, omega = (t, s) / (t, t)
__global__ void __launch_bounds__(kT)
    k_ib_t(IluState* st, Csr A, int R, const double* __restrict__ a, const double* __restrict__ z,
           const double* __restrict__ s, double* __restrict__ t, double* pa, double* pb) {
    if (done_flag(st)) return;
    double ats = 0.0, att = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= A.n) continue;
        const double ti = csr_row(A, a, z, i);
        t[i] = ti;
        ats = fma(ti, __ldg(&s[i]), ats);
        att = fma(ti, ti, att);
    }
    double ts, tt;
    if (tree_dots(st, pa, pb, ats, att, 2, &ts, &tt) && threadIdx.x == 0) {
        const double omega = ts / tt;
        st->omega = omega;
        if (tt == 0.0 || !isfinite(omega) || omega == 0.0) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
    }
}

// x += alpha y + omega z, r = s - omega t, rho = (rr, r), |r|, stopping tests
__global__ void __launch_bounds__(kT)
    k_ib_x(IluState* st, int n, int R, const double* __restrict__ y, const double* __restrict__ z,
           const double* __restrict__ s, const double* __restrict__ t, const double* __restrict__ rr,
           double* __restrict__ r, double* pa, double* pb) {
    if (done_flag(st)) return;
    const double alpha = st->alpha, omega = st->omega;
    double* x = st->x;
    double arho = 0.0, arr = 0.0;
    for (int j = 0; j < R; ++j) {
        const int i = tree_row(R, j);
        if (i >= n) continue;
        x[i] = fma(omega, __ldg(&z[i]), fma(alpha, __ldg(&y[i]), x[i]));
        const double ri = fma(-omega, __ldg(&t[i]), __ldg(&s[i]));
        r[i] = ri;
        arho = fma(__ldg(&rr[i]), ri, arho);
        arr = fma(ri, ri, arr);
    }
    double rho, rsq;
    if (tree_dots(st, pa, pb, arho, arr, 2, &rho, &rsq) && threadIdx.x == 0) {
        st->rho_prev = st->rho;
        st->rho = rho;
        st->beta = (st->rho / st->rho_prev) * (st->alpha / st->omega);
        after_step(st, sqrt(rsq));
        if (!st->done && rho == 0.0) {
            st->status = FVGB_ERR_BREAKDOWN;
            st->done = 1;
        }
    }
}

__global__ void k_il_cond(const IluState* st, cudaGraphConditionalHandle h) {
    cudaGraphSetConditional(h, st->done ? 0u : 1u);
}

__global__ void k_il_stats(IluState* st) {
    fvgb_solver_stats s{};
    s.init_res_norm = st->res0;
    s.final_res_norm = st->res;
    s.num_iter = st->iter;
    s.num_outer = 0;
    s.status = st->status;
    st->stats = s;
    if (st->stats_out) *st->stats_out = s;
}

}  // namespace

// ------------------------------------------------------------ host side
struct IluCache {
    const fvgb_ls* ls = nullptr;
    int n = 0, nnz = 0, R = 4, nb = 1;
    unsigned sweep_grid = 1;  // resident blocks of a triangular sweep
    int sweep_smem = 0;
    bool pivots_only = true;  // the factorization changes the lower triangle and the diagonal alone (hex meshes)
    Sweep fwd{}, bwd{};
    int *ro = nullptr, *col = nullptr, *dof = nullptr;
    int *op_ptr = nullptr, *op_f = nullptr, *op_g = nullptr;
    int* lev_rows = nullptr;   // rows by level of the lower triangle
    std::vector<int> fwd_ptr;  // level offsets into it (host)
    double *a = nullptr, *lu = nullptr;
    double *r = nullptr, *rr = nullptr, *p = nullptr, *q = nullptr, *v = nullptr, *y = nullptr, *z = nullptr,
           *s = nullptr, *t = nullptr, *w = nullptr, *pa = nullptr, *pb = nullptr;
    IluState* st = nullptr;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};  // CG, BiCGStab
    std::vector<void*> allocs;
};

namespace {

unsigned grid_of(int count) { return count > 0 ? (unsigned)((count + kT - 1) / kT) : 1u; }

template <int KIND>
const void* sweep_fn(const Sweep& S) {
    if (S.hcap == 0)
        return S.K == kDeps ? (const void*)k_il_sweep<KIND, kDeps, true> : (const void*)k_il_sweep<KIND, kDeps - 1, true>;
    return S.K == kDeps ? (const void*)k_il_sweep<KIND, kDeps, false> : (const void*)k_il_sweep<KIND, kDeps - 1, false>;
}

template <class T>
cudaError_t il_alloc(IluCache* c, T** p, size_t count) {
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
    if (e == cudaSuccess) c->allocs.push_back(*p);
    return e;
}

template <class T>
cudaError_t il_upload(IluCache* c, T** p, const std::vector<T>& h) {
    cudaError_t e = il_alloc(c, p, h.size());
    if (e == cudaSuccess && !h.empty()) e = cudaMemcpy(*p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
    return e;
}

// rows grouped by level (stable in row order), level offsets in ptr
void by_level(const std::vector<int>& lev, std::vector<int>& ptr, std::vector<int>& rows) {
    const int nl = lev.empty() ? 0 : 1 + *std::max_element(lev.begin(), lev.end());
    ptr.assign((size_t)nl + 1, 0);
    for (int l : lev) ++ptr[(size_t)l + 1];
    for (int l = 0; l < nl; ++l) ptr[(size_t)l + 1] += ptr[(size_t)l];
    rows.assign(lev.size(), 0);
    std::vector<int> at(ptr.begin(), ptr.end() - 1);
    for (int i = 0; i < (int)lev.size(); ++i) rows[(size_t)at[(size_t)lev[(size_t)i]]++] = i;
}

// Rows of a part: the most, halving from kPart to kMinPart, of which a level has no
// more than kLevelRows in a part from the middle.
int part_rows(const std::vector<int>& level) {
    const int n = (int)level.size();
    int rpp = kPart;
    for (std::vector<int> cnt; rpp > kMinPart; rpp /= 2) {
        const int r0 = (n / 2) / rpp * rpp, r1 = std::min(n, r0 + rpp);
        const auto mm = std::minmax_element(level.begin() + r0, level.begin() + r1);
        if (r0 >= r1) break;
        cnt.assign((size_t)(*mm.second - *mm.first + 1), 0);
        for (int i = r0; i < r1; ++i) ++cnt[(size_t)(level[(size_t)i] - *mm.first)];
        if (*std::max_element(cnt.begin(), cnt.end()) <= kLevelRows) break;
    }
    return rpp;
}

// Rows of a group: parts of consecutive rows have levels of few rows when the mesh's lines
// are long (one row, where a line is longer than a part), and a level takes as long for one
// row as for 32.  Such parts are cut from groups of consecutive rows instead, doubled from
// a part's size until a group in the middle has kThinRows rows a level, or is all rows.
int group_rows(const std::vector<int>& level, int rpp) {
    const long n = (long)level.size();
    long group = rpp;
    for (; group < n; group *= 2) {
        const long r0 = (n / 2) / group * group, r1 = std::min(n, r0 + group);
        const auto mm = std::minmax_element(level.begin() + r0, level.begin() + r1);
        if (r1 - r0 >= (long)kThinRows * (*mm.second - *mm.first + 1)) break;
    }
    return (int)std::min(group, n);
}

// The order in which the parts of a sweep are taken: after every part it depends on, the
// one with the lowest first level first.  rows: in the order of groups, in a group by
// level; part p has rpp of them from p rpp on (a group is a multiple, or all rows).
std::vector<int> part_order(const fvgb_mesh* m, const std::vector<int>& rows, const std::vector<int>& level, int rpp,
                            int nparts, bool bwd) {
    const int n = (int)rows.size();
    std::vector<int> part((size_t)n), need((size_t)nparts, 0), seen((size_t)nparts, -1), order;
    std::vector<std::vector<int>> then((size_t)nparts);
    for (int t = 0; t < n; ++t) part[(size_t)rows[(size_t)t]] = t / rpp;
    for (int t = 0; t < n; ++t) {
        const int p = t / rpp, i = rows[(size_t)t], d = m->h_row_offs[i] + m->h_diag_off[i];
        for (int e = bwd ? d + 1 : m->h_row_offs[i]; e < (bwd ? m->h_row_offs[i + 1] : d); ++e) {
            const int q = part[(size_t)m->h_col[e]];
            if (q == p || seen[(size_t)q] == p) continue;
            seen[(size_t)q] = p;
            then[(size_t)q].push_back(p);
            ++need[(size_t)p];
        }
    }
    using Entry = std::pair<int, int>;  // first level, part
    std::priority_queue<Entry, std::vector<Entry>, std::greater<Entry>> ready;
    const auto put = [&](int p) { ready.emplace(level[(size_t)rows[(size_t)p * rpp]], p); };
    for (int p = 0; p < nparts; ++p)
        if (need[(size_t)p] == 0) put(p);
    while (!ready.empty()) {
        const int p = ready.top().second;
        ready.pop();
        order.push_back(p);
        for (int q : then[(size_t)p])
            if (--need[(size_t)q] == 0) put(q);
    }
    return order;
}

// The order of a sweep from the rows' levels: the parts as they are taken, in a part by
// level.  vals: doubles per row of S.val.
cudaError_t il_sweep(IluCache* c, Sweep& S, const std::vector<int>& level, int group, bool bwd, int vals) {
    std::vector<int> rows((size_t)S.n), sorted((size_t)S.n), order, first(1, 0), lev(1, 0), start, at;
    int most = 0;  // rows of the largest level
    for (int r0 = 0; r0 < S.n; r0 += group) {
        const int r1 = (int)std::min((long)S.n, (long)r0 + group);
        const auto mm = std::minmax_element(level.begin() + r0, level.begin() + r1);
        const int lo = *mm.first;
        at.assign((size_t)(*mm.second - lo + 2), 0);
        for (int i = r0; i < r1; ++i) ++at[(size_t)(level[(size_t)i] - lo + 1)];
        at[0] = r0;
        for (size_t k = 1; k < at.size(); ++k) at[k] += at[k - 1];
        for (int i = r0; i < r1; ++i) sorted[(size_t)at[(size_t)(level[(size_t)i] - lo)]++] = i;
        if (r1 == S.n) break;
    }
    if (group <= S.rpp) {
        for (int u = 0; u < S.nparts; ++u) order.push_back(bwd ? S.nparts - 1 - u : u);
    } else {
        order = part_order(c->ls->mesh, sorted, level, S.rpp, S.nparts, bwd);
    }
    for (int p : order) {
        const int t0 = p * S.rpp, t1 = std::min(S.n, t0 + S.rpp);
        int prev = -1;
        for (int t = t0, at = first.back(); t < t1; ++t, ++at) {
            const int i = sorted[(size_t)t];
            rows[(size_t)at] = i;
            if (level[(size_t)i] == prev) continue;
            prev = level[(size_t)i];
            if (start.size() > (size_t)lev.back()) most = std::max(most, at - start.back());
            start.push_back(at);
        }
        first.push_back(first.back() + t1 - t0);
        most = std::max(most, first.back() - start.back());
        lev.push_back((int)start.size());
    }
    start.push_back(S.n);
    S.W = 1;
    while (32 * S.W < most && S.W < kRowWarps / 2) S.W *= 2;
    int *r = nullptr, *fi = nullptr, *lv = nullptr, *sa = nullptr;
    cudaError_t e = il_upload(c, &r, rows);
    if (e == cudaSuccess) e = il_upload(c, &fi, first);
    if (e == cudaSuccess) e = il_upload(c, &lv, lev);
    if (e == cudaSuccess) e = il_upload(c, &sa, start);
    S.rows = r;
    S.first = fi;
    S.lev = lv;
    S.start = sa;
    if (e == cudaSuccess) e = il_alloc(c, &S.pos, (size_t)S.n);
    if (e == cudaSuccess) e = il_alloc(c, &S.slot, (size_t)S.K * S.n);
    if (e == cudaSuccess) e = il_alloc(c, &S.val, (size_t)vals * S.n);
    if (e == cudaSuccess) e = il_alloc(c, &S.halo, (size_t)S.nparts * S.hcap);
    if (e == cudaSuccess) e = il_alloc(c, &S.nhalo, (size_t)S.nparts);
    return e;
}

fvgb_status symbolic(IluCache* c) {
    const fvgb_mesh* m = c->ls->mesh;
    const int n = m->v.n, nnz = m->nnz;
    if ((int)m->h_row_offs.size() != n + 1 || (int)m->h_col.size() != nnz || (int)m->h_diag_off.size() != n)
        return fvgb_fail(FVGB_ERR_UNSUPPORTED, "ILU: the mesh keeps no host sparsity pattern (device-built boxes)");
    const std::vector<int32_t>& ro = m->h_row_offs;
    const std::vector<int32_t>& col = m->h_col;
    const std::vector<int32_t>& dof = m->h_diag_off;
    std::vector<int> op_ptr((size_t)nnz + 1, 0), op_f, op_g, lev_f((size_t)n, 0), lev_b((size_t)n, 0);
    op_f.reserve((size_t)(nnz - n) / 2);
    op_g.reserve((size_t)(nnz - n) / 2);
    int maxl = 0, maxu = 0;
    for (int i = 0; i < n; ++i) {
        const int d = ro[i] + dof[i], end = ro[i + 1];
        maxl = std::max(maxl, d - ro[i]);
        maxu = std::max(maxu, end - d - 1);
        for (int e = ro[i]; e < end; ++e) {
            if (e < d) {
                const int k = col[e];
                lev_f[i] = std::max(lev_f[i], lev_f[k] + 1);
                int f = e + 1, g = ro[k] + dof[k] + 1;
                while (f < end && g < ro[k + 1]) {  // j > k in rows i and k, ascending
                    if (col[f] < col[g]) ++f;
                    else if (col[f] > col[g]) ++g;
                    else {
                        op_f.push_back(f++);
                        op_g.push_back(g++);
                    }
                }
            }
            op_ptr[(size_t)e + 1] = (int)op_f.size();
            if (e < d && (op_ptr[(size_t)e + 1] != op_ptr[(size_t)e] + 1 || op_f.back() != d)) c->pivots_only = false;
        }
    }
    for (int i = n - 1; i >= 0; --i)
        for (int e = ro[i] + dof[i] + 1; e < ro[i + 1]; ++e) lev_b[i] = std::max(lev_b[i], lev_b[col[e]] + 1);
    std::vector<int> lev_rows;
    if (!c->pivots_only) by_level(lev_f, c->fwd_ptr, lev_rows);
    c->n = n;
    c->nnz = nnz;
    c->R = n >= (1 << 15) ? 8 : 4;
    c->nb = std::max(1, (n + kT * c->R - 1) / (kT * c->R));
    int dev = 0, sms = 1;
    FVGB_CUDA_TRY(cudaGetDevice(&dev));
    FVGB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int rpp = std::min((n + 31) / 32 * 32, std::max(32, part_rows(lev_f)));
    const int nparts = (n + rpp - 1) / rpp, group = group_rows(lev_f, rpp);
    // one group of several parts: they follow one another, and more than the next few would
    // only wait (with a part of a chain on every SM, half a second)
    const int blocks = group > rpp && group == n ? 4 : n >= kDirectRows ? 2 * sms : sms;
    c->sweep_grid = (unsigned)std::max(1, std::min(nparts, blocks));
    const auto setup = [&](Sweep& S, int deps) {
        S.n = n;
        S.rpp = rpp;
        S.nparts = nparts;
        S.K = deps < kDeps ? kDeps - 1 : kDeps;
        S.hcap = n >= kDirectRows ? 0 : 2 * rpp;  // a row of a hex mesh needs one value of another part, or two
    };
    setup(c->fwd, maxl);
    setup(c->bwd, maxu);
    c->sweep_smem = (int)sizeof(double) * (rpp + c->fwd.hcap + 1);
    for (const void* f : {sweep_fn<kFwd>(c->fwd), sweep_fn<kBwd>(c->bwd), sweep_fn<kFactor>(c->fwd)})
        FVGB_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSweepSmem));
    cudaError_t e = il_upload(c, &c->ro, ro);
    if (e == cudaSuccess) e = il_upload(c, &c->col, col);
    if (e == cudaSuccess) e = il_upload(c, &c->dof, dof);
    if (e == cudaSuccess) e = il_upload(c, &c->op_ptr, op_ptr);
    if (e == cudaSuccess && !c->pivots_only) e = il_upload(c, &c->op_f, op_f);
    if (e == cudaSuccess) e = il_upload(c, &c->op_g, op_g);
    if (e == cudaSuccess && !c->pivots_only) e = il_upload(c, &c->lev_rows, lev_rows);
    if (e == cudaSuccess) e = il_sweep(c, c->fwd, lev_f, group, false, c->pivots_only ? 2 * c->fwd.K + 1 : c->fwd.K);
    if (e == cudaSuccess) e = il_sweep(c, c->bwd, lev_b, group, true, c->bwd.K + 2);
    if (e == cudaSuccess) e = il_alloc(c, &c->a, (size_t)nnz);
    if (e == cudaSuccess) e = il_alloc(c, &c->lu, (size_t)nnz);
    double** vecs[] = {&c->r, &c->rr, &c->p, &c->q, &c->v, &c->y, &c->z, &c->s, &c->t, &c->w};
    for (double** v : vecs)
        if (e == cudaSuccess) e = il_alloc(c, v, (size_t)n);
    if (e == cudaSuccess) e = il_alloc(c, &c->pa, (size_t)c->nb);
    if (e == cudaSuccess) e = il_alloc(c, &c->pb, (size_t)c->nb);
    if (e == cudaSuccess) e = il_alloc(c, &c->st, 1);
    if (e == cudaSuccess) e = cudaMemset(c->st, 0, sizeof(IluState));
    if (e != cudaSuccess) return cuda_fail(e, "ILU setup");
    const Csr A{n, c->ro, c->col, c->dof};
    if (n > 0) {
        for (const Sweep& S : {c->fwd, c->bwd}) k_il_pos<<<grid_of(n), kT>>>(S);
        k_il_plan<false><<<nparts, kT>>>(A, c->fwd);
        k_il_plan<true><<<nparts, kT>>>(A, c->bwd);
        FVGB_LAUNCH_CHECK("ILU plan");
    }
    FVGB_CUDA_TRY(settle_creation());
    return FVGB_OK;
}

// Graph construction: kernel nodes in a chain.  The arguments are passed by
// value; cudaGraphAddKernelNode copies the values the pointers point to.
struct Chain {
    cudaGraph_t g;
    cudaGraphNode_t prev = nullptr;
    bool has_prev = false;
    cudaError_t e = cudaSuccess;
    int smem = 0;  // of a sweep, which has a block size of its own

    template <class... A>
    void add(void* fn, unsigned grid, A... args) {
        if (e != cudaSuccess) return;
        void* params[] = {(void*)&args...};
        cudaKernelNodeParams kp{};
        kp.func = fn;
        kp.gridDim = dim3(grid);
        kp.blockDim = dim3(fn == (void*)k_il_cond || fn == (void*)k_il_stats ? 1 : smem ? kSweepThreads : kT);
        kp.sharedMemBytes = (unsigned)smem;
        kp.kernelParams = params;
        cudaGraphNode_t node;
        e = cudaGraphAddKernelNode(&node, g, has_prev ? &prev : nullptr, has_prev ? 1 : 0, &kp);
        if (e == cudaSuccess) {
            prev = node;
            has_prev = true;
        }
    }
};

template <int KIND>
void add_sweep(IluCache* c, Chain& ch, const Sweep& S, const double* src, double* v, double* other) {
    const Csr A{c->n, c->ro, c->col, c->dof};
    const Factor F{c->a, c->lu, c->op_ptr, c->op_g};
    ch.smem = c->sweep_smem;
    ch.add((void*)sweep_fn<KIND>(S), c->sweep_grid, c->st, A, S, F, (const double*)c->lu, src, v, other);
    ch.smem = 0;
}

// z = U^-1 L^-1 src through c->w: a forward and a backward sweep
void add_apply(IluCache* c, Chain& ch, const double* src, double* dst) {
    add_sweep<kFwd>(c, ch, c->fwd, src, c->w, dst);
    add_sweep<kBwd>(c, ch, c->bwd, c->w, dst, c->w);
}

fvgb_status build_graph(IluCache* c, bool bicgstab) {
    cudaGraphExec_t& out = c->graph[bicgstab ? 1 : 0];
    const fvgb_ls* ls = c->ls;
    const Csr A{c->n, c->ro, c->col, c->dof};
    const int n = c->n, R = c->R;
    const unsigned nb = (unsigned)c->nb, ng = grid_of(n);
    IluState* st = c->st;
    const double* a = c->a;
    const double* b = ls->rhs;
    cudaGraph_t g = nullptr;
    FVGB_CUDA_TRY(cudaGraphCreate(&g, 0));
    Chain ch;
    ch.g = g;
    cudaGraphConditionalHandle h{};
    ch.e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
    ch.add((void*)k_il_bnorm, nb, st, n, R, b, c->pa);
    ch.add((void*)k_il_pending, ng, n, c->w);  // the forward sweeps' output, pending
    ch.add((void*)k_il_gather, grid_of(c->nnz), c->nnz, (const int*)ls->mesh->csr_pos, (const double*)ls->values,
           c->a, c->lu);
    const Factor F{c->a, c->lu, c->op_ptr, c->op_g};
    if (c->pivots_only) {
        ch.add((void*)k_il_pending, ng, n, c->t);
        ch.add((void*)k_il_pack<kFactor>, grid_of(n), A, c->fwd, F, (const double*)nullptr);
        add_sweep<kFactor>(c, ch, c->fwd, c->a, c->t, c->t);
    } else {
        for (size_t l = 0; l + 1 < c->fwd_ptr.size(); ++l) {
            const int cnt = c->fwd_ptr[l + 1] - c->fwd_ptr[l];
            ch.add((void*)k_il_factor, grid_of(cnt), A, (const int*)(c->lev_rows + c->fwd_ptr[l]), cnt,
                   (const int*)c->op_ptr, (const int*)c->op_f, (const int*)c->op_g, c->lu);
        }
    }
    if (!c->pivots_only) ch.add((void*)k_il_pack<kFwd>, grid_of(n), A, c->fwd, F, (const double*)nullptr);
    ch.add((void*)k_il_pack<kBwd>, grid_of(n), A, c->bwd, F, (const double*)(c->pivots_only ? c->t : nullptr));
    if (!bicgstab) {
        ch.add((void*)k_ic_init, nb, st, A, R, a, b, c->r, c->pa);
        add_apply(c, ch, c->r, c->z);
        ch.add((void*)k_ic_first, nb, st, n, R, (const double*)c->r, (const double*)c->z, c->p, c->pa);
    } else {
        ch.add((void*)k_ib_init, nb, st, A, R, a, b, c->r, c->rr, c->p, c->v, c->pa, c->pb);
    }
    ch.add((void*)k_il_cond, 1, (const IluState*)st, h);
    cudaGraph_t body = nullptr;
    if (ch.e == cudaSuccess) {
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t node;
        ch.e = cudaGraphAddNode(&node, g, &ch.prev, nullptr, 1, &np);
        if (ch.e == cudaSuccess) {
            body = np.conditional.phGraph_out[0];
            ch.prev = node;
        }
    }
    Chain bc;
    bc.g = body;
    if (ch.e == cudaSuccess) {
        if (!bicgstab) {
            bc.add((void*)k_ic_spmv, nb, st, A, R, a, (const double*)c->p, c->q, c->pa);
            bc.add((void*)k_ic_update, nb, st, n, R, (const double*)c->p, (const double*)c->q, c->r, c->pa);
            add_apply(c, bc, c->r, c->z);
            bc.add((void*)k_ic_rz, nb, st, n, R, (const double*)c->r, (const double*)c->z, c->pa);
            bc.add((void*)k_ic_dir, ng, (const IluState*)st, n, (const double*)c->z, c->p);
        } else {
            bc.add((void*)k_ib_p, ng, (const IluState*)st, n, (const double*)c->r, (const double*)c->v, c->p);
            add_apply(c, bc, c->p, c->y);
            bc.add((void*)k_ib_v, nb, st, A, R, a, (const double*)c->y, (const double*)c->rr, c->v, c->pa);
            bc.add((void*)k_ib_s, nb, st, n, R, (const double*)c->r, (const double*)c->v, c->s, c->pa);
            bc.add((void*)k_ib_half, ng, st, n, (const double*)c->y);
            add_apply(c, bc, c->s, c->z);
            bc.add((void*)k_ib_t, nb, st, A, R, a, (const double*)c->z, (const double*)c->s, c->t, c->pa, c->pb);
            bc.add((void*)k_ib_x, nb, st, n, R, (const double*)c->y, (const double*)c->z, (const double*)c->s,
                   (const double*)c->t, (const double*)c->rr, c->r, c->pa, c->pb);
        }
        bc.add((void*)k_il_cond, 1, (const IluState*)st, h);
        ch.e = bc.e;
    }
    ch.add((void*)k_il_stats, 1, st);
    cudaError_t e = ch.e;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&out, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        out = nullptr;
        return cuda_fail(e, "ILU solve graph");
    }
    return FVGB_OK;
}

}  // namespace

void fvgb_ilu_free(IluCache* c) {
    if (!c) return;
    for (cudaGraphExec_t g : c->graph)
        if (g) cudaGraphExecDestroy(g);
    for (void* p : c->allocs) cudaFree(p);
    delete c;
}

fvgb_status fvgb_ilu_solve_async(fvgb_ls* ls, double* x, const fvgb_solver_cfg* cfg, fvgb_solver_stats* stats_dev,
                                 cudaStream_t s) {
    if (ls->ncomp != 1) return fvgb_fail(FVGB_ERR_INVALID_ARG, "fvgb_solve: scalar systems only");
    if (cfg->method != FVGB_SOLVER_CG && cfg->method != FVGB_SOLVER_BICGSTAB)
        return fvgb_fail(FVGB_ERR_UNSUPPORTED, "ILU: the preconditioner of CG and BiCGStab only");
    if (cfg->precision != FVGB_PREC_FP64)
        return fvgb_fail(FVGB_ERR_UNSUPPORTED, "ILU: FP64 only (no mixed-precision ILU solve)");
    FVGB_CHECK_ARG(cfg->rel_tol >= 0 && cfg->abs_tol >= 0, "fvgb_solve: negative tolerance");
    FVGB_CHECK_ARG(cfg->max_iter >= 0 && cfg->max_iter <= 100000000, "fvgb_solve: bad max_iter");
    FVGB_CHECK_ARG((cfg->flags & ~(FVGB_SOLVE_NO_TUNE | FVGB_SOLVE_RHS_BASELINE)) == 0, "fvgb_solve: unknown flags");
    const bool bicgstab = cfg->method == FVGB_SOLVER_BICGSTAB;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    FVGB_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
    if (!ls->ilu || !ls->ilu->graph[bicgstab ? 1 : 0]) {
        // setup allocates, uploads synchronously and builds a graph
        if (cs != cudaStreamCaptureStatusNone)
            return fvgb_fail(FVGB_ERR_UNSUPPORTED, "ILU: the first solve (setup) cannot be stream-captured");
        if (!ls->ilu) {
            IluCache* c = new IluCache();
            c->ls = ls;
            fvgb_status st = symbolic(c);
            if (st != FVGB_OK) {
                fvgb_ilu_free(c);
                return st;
            }
            ls->ilu = c;
        }
        fvgb_status st = build_graph(ls->ilu, bicgstab);
        if (st != FVGB_OK) return st;
    }
    IluCache* c = ls->ilu;
    k_il_params<<<1, 1, 0, s>>>(c->st, x, cfg->rel_tol, cfg->abs_tol, cfg->max_iter, stats_dev,
                                (cfg->flags & FVGB_SOLVE_RHS_BASELINE) ? 1 : 0);
    FVGB_LAUNCH_CHECK("ILU params");
    FVGB_CUDA_TRY(cudaGraphLaunch(c->graph[bicgstab ? 1 : 0], s));
    return FVGB_OK;
}

fvgb_status fvgb_ilu_sync_stats(fvgb_ls* ls, fvgb_solver_stats* out, cudaStream_t s) {
    fvgb_solver_stats h{};
    FVGB_CUDA_TRY(cudaMemcpyAsync(&h, &ls->ilu->st->stats, sizeof h, cudaMemcpyDeviceToHost, s));
    FVGB_CUDA_TRY(cudaStreamSynchronize(s));
    if (out) *out = h;
    return (fvgb_status)h.status;
}
