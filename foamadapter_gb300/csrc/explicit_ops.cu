// Explicit finite-volume operators: surface interpolation (linear, upwind),
// Gauss-Green div / grad / laplacian, uncorrected snGrad and the fused
// upwind-advection forward-Euler step.
//
// The reference's Serial executor scatters face contributions into owner (+)
// and neighbour (-) cells in ascending face order.  Here one thread owns one
// cell and walks that cell's faces in the same ascending order through the
// gather list, so every cell sees the same sequence of IEEE operations and the
// result is bit-identical to the Serial face loop, with no atomics.  This file
// is compiled with -fmad=false so no multiply-add is contracted.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <string>

#include "internal.cuh"
#include "ll.cuh"
#include "tunecache.h"

namespace {

constexpr int kThreads = 256;
constexpr int kFaceThreads = 128;    // face passes: 12 blocks an SM
constexpr int kGatherThreads = 128;  // cell passes over a face buffer

__device__ __forceinline__ int gwidth(const MeshView& m, int slice) {
    return (__ldg(&m.g_ptr[slice + 1]) - __ldg(&m.g_ptr[slice])) >> 5;
}

// F >= 0.0 with IEEE semantics (true for +0 and -0 and +inf, false for NaN),
// decided on the bit pattern so it costs no FP64 instruction: GB300's FP64
// issue rate bounds every FP64 face loop here.
__device__ __forceinline__ bool nonneg(double F) {
    const long long u = __double_as_longlong(F);
    return u >= 0 ? u <= 0x7ff0000000000000LL : u == (long long)0x8000000000000000ULL;
}

// The owner/neighbour accumulation s + x or s - x is ONE fused multiply-add,
// fma(x, +-1, s) (facc): exactly the rounded sum or difference, with no branch
// and no separate negation.  Every other exact sum and product is a DFMA too
// (fadd, fsub, fmul): GB300 retires DFMA faster than DADD and DMUL.

// ---------------------------------------------------------------- interpolation
// Face passes: a thread handles FPT faces spaced a block apart (coalesced across the
// block).  FPT (the face-pass tile: 2, 4 or 8) is the mesh's `face_tile`, 4 unless
// fvgb_explicit_tune measured another; every face is computed alone, so every tile
// gives the same bits.
//
// An operator is a struct: fetch() reads what a face holds (cells, weight, flux),
// gather() the values of its two cells, inner() computes and stores, boundary() does a
// boundary face.  Blocks of internal faces only run the three steps for kBatch faces
// at a time, so that their loads are in flight together without a branch between.
//
// The passes stood at 77 to 88 % of the FP64 pipe, loads and arithmetic hardly
// overlapping, while 10 to 17 % of the issue slots were in use.  So their products run
// on the integer pipes (imul), and the blocks are small and many (12 of 128 threads an
// SM).  Jittered 128^3 box, face pass and cell pass together, before and after: linear
// interpolation 43.7 -> 35.5 us, upwind div 85.6 -> 65.2, linear div 91.8 -> 77.5, of a
// vector 212.6 -> 171.7, gradient 179.8 -> 153.3, Laplacian 87.7 -> 77.5, corrected
// 398.9 -> 312.0 (its gradient buffer no longer zeroed and read), snGrad 39.6 -> 33.4,
// corrected 335.5 -> 259.8 (and written in place of a copy).
#define FVGB_FACE_TILE(tile, ...)          \
    switch (tile) {                         \
        case 2: {                           \
            constexpr int FPT = 2;          \
            __VA_ARGS__;                    \
        } break;                            \
        case 8: {                           \
            constexpr int FPT = 8;          \
            __VA_ARGS__;                    \
        } break;                            \
        default: {                          \
            constexpr int FPT = 4;          \
            __VA_ARGS__;                    \
        } break;                            \
    }

template <int FPT, class Op>
__global__ void __launch_bounds__(kFaceThreads, 12) k_faces(MeshView m, Op op) {
    const int f0 = blockIdx.x * FPT * kFaceThreads + threadIdx.x;
    if ((int)(blockIdx.x + 1) * FPT * kFaceThreads <= m.nif) {
        constexpr int B = Op::kBatch;
#pragma unroll
        for (int g = 0; g < FPT / B; ++g) {
            typename Op::Face a[B];
            typename Op::Cells t[B];
#pragma unroll
            for (int k = 0; k < B; ++k) op.fetch(m, f0 + (g * B + k) * kFaceThreads, a[k]);
#pragma unroll
            for (int k = 0; k < B; ++k) op.gather(a[k], t[k]);
#pragma unroll
            for (int k = 0; k < B; ++k) op.inner(m, f0 + (g * B + k) * kFaceThreads, a[k], t[k]);
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < FPT; ++k) {
            const int f = f0 + k * kFaceThreads;
            if (f < m.nif) {
                typename Op::Face a;
                typename Op::Cells t;
                op.fetch(m, f, a);
                op.gather(a, t);
                op.inner(m, f, a, t);
            } else if (f < m.nif + m.nbf) {
                op.boundary(m, f, f - m.nif);
            }
        }
    }
}

// the values of a face's two cells
template <int NC>
struct PairOf {
    double p[NC], n[NC];
    __device__ __forceinline__ void load(const double* __restrict__ src, int P, int N) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            p[c] = __ldg(&src[P * NC + c]);
            n[c] = __ldg(&src[N * NC + c]);
        }
    }
};

template <int NC>
struct InterpLinear {
    static constexpr int kBatch = 2;
    struct Face { int P, N; double w; };
    using Cells = PairOf<NC>;
    const double *src, *src_b;
    double* dst;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.w = __ldg(&m.w[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const { t.load(src, a.P, a.N); }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) dst[f * NC + c] = fadd(m, imul(a.w, fsub(m, t.p[c], t.n[c])), t.n[c]);
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) dst[f * NC + c] = __ldg(&src_b[b * NC + c]);
    }
};

template <int NC>
struct InterpUpwind {
    static constexpr int kBatch = 2;
    struct Face { int P, N; double F; };
    struct Cells { double v[NC]; };
    const double *flux, *src, *src_b;
    double* dst;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.F = __ldg(&flux[f]);
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const {
        const int u = nonneg(a.F) ? a.P : a.N;
#pragma unroll
        for (int c = 0; c < NC; ++c) t.v[c] = __ldg(&src[u * NC + c]);
    }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) dst[f * NC + c] = t.v[c];
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) dst[f * NC + c] = __ldg(&src_b[b * NC + c]);
    }
};

// ------------------------------------------------------------ gather entries
// A cell's first kG gather entries are fetched together: the entry codes and
// the cells (or boundary faces) across, then every face and cell value they
// point to, so a thread has all its loads in flight at once instead of one
// dependent pair per face.  The arithmetic then runs in ascending face order
// exactly as the one-entry-at-a-time loop did; entries beyond kG (cells with
// more than kG faces) take the per-entry path.
constexpr int kG = 8;

struct Entries {
    int base, width;
    int code[kG], other[kG];  // code FVGB_PAD beyond the cell's row
};

__device__ __forceinline__ void load_entries(const MeshView& m, int c, Entries& e) {
    const int slice = c >> 5;
    e.base = __ldg(&m.g_ptr[slice]) + (c & 31);
    e.width = gwidth(m, slice);
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        e.code[j] = FVGB_PAD;
        e.other[j] = 0;
        if (j < e.width) {
            e.code[j] = __ldg(&m.g_code[e.base + j * 32]);
            e.other[j] = __ldg(&m.g_other[e.base + j * 32]);
        }
    }
}

// face index of an entry (a boundary entry's code is its index in face fields)
__device__ __forceinline__ int entry_face(int code) { return code >= 0 ? code : -code - 1; }

// ------------------------------------------------------------------------ div
// face value seen from cell c across internal face f: owner-side formulas of
// the reference with (P, N) = (owner, neighbour).
template <int NC, int SCHEME>
__device__ __forceinline__ void div_entry(const MeshView& m, int code, double F, const double* To, double wf,
                                          const double* Tc, double* s) {
    if (code >= m.nif) {  // boundary face: value from the boundary field
#pragma unroll
        for (int k = 0; k < NC; ++k) s[k] = fadd(m, s[k], fmul(m, F, To[k]));
        return;
    }
    const bool isOwner = code >= 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const double Town = isOwner ? Tc[k] : To[k];
        const double Tnei = isOwner ? To[k] : Tc[k];
        double tf;
        if (SCHEME == FVGB_SCHEME_UPWIND) tf = nonneg(F) ? Town : Tnei;
        else tf = fadd(m, fmul(m, wf, fsub(m, Town, Tnei)), Tnei);
        s[k] = facc(m, s[k], isOwner, fmul(m, F, tf));
    }
}

template <int NC, int SCHEME>
__device__ __forceinline__ void div_cell(const MeshView& m, int c, const double* __restrict__ flux,
                                         const double* __restrict__ phi,
                                         const double* __restrict__ phi_b, double* s) {
    Entries e;
    load_entries(m, c, e);
    double Tc[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        Tc[k] = __ldg(&phi[c * NC + k]);
        s[k] = 0.0;
    }
    double F[kG], W[kG], T[kG][NC];
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        const int cd = e.code[j];
        F[j] = 0.0;
        W[j] = 0.0;
#pragma unroll
        for (int k = 0; k < NC; ++k) T[j][k] = 0.0;
        if (cd == FVGB_PAD) continue;
        const bool bnd = cd >= m.nif;
        const int f = entry_face(cd);
        F[j] = __ldg(&flux[f]);
        const double* src = bnd ? phi_b : phi;
#pragma unroll
        for (int k = 0; k < NC; ++k) T[j][k] = __ldg(&src[e.other[j] * NC + k]);
        if (SCHEME == FVGB_SCHEME_LINEAR && !bnd) W[j] = __ldg(&m.w[f]);
    }
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        if (e.code[j] == FVGB_PAD) break;
        div_entry<NC, SCHEME>(m, e.code[j], F[j], T[j], W[j], Tc, s);
    }
    for (int j = kG; j < e.width; ++j) {
        const int cd = __ldg(&m.g_code[e.base + j * 32]);
        if (cd == FVGB_PAD) break;
        const int o = __ldg(&m.g_other[e.base + j * 32]);
        const int f = entry_face(cd);
        const double* src = cd >= m.nif ? phi_b : phi;
        double To[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) To[k] = __ldg(&src[o * NC + k]);
        const double wf = (SCHEME == FVGB_SCHEME_LINEAR && cd < m.nif) ? __ldg(&m.w[f]) : 0.0;
        div_entry<NC, SCHEME>(m, cd, __ldg(&flux[f]), To, wf, Tc, s);
    }
}

template <int NC, int SCHEME>
__global__ void __launch_bounds__(kThreads)
    k_div(MeshView m, const double* __restrict__ flux, const double* __restrict__ phi,
          const double* __restrict__ phi_b, double coeff, int unit, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    double s[NC];
    div_cell<NC, SCHEME>(m, c, flux, phi, phi_b, s);
    const double sc = unit ? __ldg(&m.invV[c]) : coeff / __ldg(&m.V[c]);
#pragma unroll
    for (int k = 0; k < NC; ++k) out[c * NC + k] = fadd(m, out[c * NC + k], fmul(m, s[k], sc));
}

// Fused forward-Euler upwind advection step + boundary correction.
__global__ void __launch_bounds__(kThreads)
    k_advect_euler(MeshView m, PatchTable pt, const double* __restrict__ flux,
                   const double* __restrict__ Told, const double* __restrict__ Told_b, double dt,
                   const double* __restrict__ ref, const double* __restrict__ gq, double* __restrict__ Tnew,
                   double* __restrict__ Tnew_b) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    double s[1];
    div_cell<1, FVGB_SCHEME_UPWIND>(m, c, flux, Told, Told_b, s);
    const double dv = facc0(true, fmul(m, s[0], __ldg(&m.invV[c])));  // +0 + s/V
    const double tn = fsub(m, __ldg(&Told[c]), fmul(m, dt, dv));
    Tnew[c] = tn;
    // boundary faces of this cell (they follow its internal faces in the list)
    const int slice = c >> 5, lane = c & 31;
    const int base = __ldg(&m.g_ptr[slice]);
    const int width = gwidth(m, slice);
    for (int j = width - 1; j >= 0; --j) {
        const int code = __ldg(&m.g_code[base + j * 32 + lane]);
        if (code == FVGB_PAD) continue;
        if (code < m.nif) break;
        const int b = code - m.nif;
        const int t = pt.type[__ldg(&m.bpatch[b])];
        double v = __ldg(&Told_b[b]);
        if (t == FVGB_BC_FIXED_VALUE) v = __ldg(&ref[b]);
        else if (t == FVGB_BC_FIXED_GRADIENT) v = tn + (gq ? __ldg(&gq[b]) : __ldg(&ref[b]) / __ldg(&m.bdelta[b]));
        Tnew_b[b] = v;
    }
}

// nsteps of the fused step in one launch: a thread keeps its cell, the cell's fluxes
// and where each face's upwind value comes from (the cell itself or another cell of
// the block in shared memory, or a slot of its own: a boundary value, or a cell of
// another block received with its step beside it, ll.cuh).  Per step a block waits
// only for the cells next to its own, in both directions whatever the flow's (so
// blocks stay within a step of each other and three step buffers suffice: a cell
// seen at step k means its block is done reading step k - 2).  What bounds a step
// is one round trip to L2 (~600 clocks, behind the publishing store's ~500) and a
// cell's chain of 10 DFMAs (64 clocks each with one warp per scheduler).  64 x 64
// cells: 1.3 us a step against 6.2 for a launch per step; 280 x 280: 2.9 against 14.
template <int MAXT, int E>
__global__ void __launch_bounds__(MAXT)
    k_advect_steps(MeshView m, PatchTable pt, const double* __restrict__ flux, double* T, double* T_b, double dt,
                   const double* __restrict__ ref, int nsteps, LLWord* ll, GridBar* gb) {
    // [2][bs] cells of this block by step parity, [E][bs] slots, [E][bs] boundary constants, [E][bs] cells (int)
    extern __shared__ double sm[];
    const int bs = (int)blockDim.x, t = (int)threadIdx.x, c = blockIdx.x * bs + t, first = blockIdx.x * bs;
    double* slot = sm + 2 * bs;
    double* bq = slot + E * bs;
    int* scell = (int*)(bq + E * bs);
    double F[E], Tc = 0.0, iv = 0.0;
    int src[E];  // index into sm; cells of the block (bit in `local`) add the step parity's offset
    unsigned plus = 0u, remote = 0u, bnd = 0u, local = 0u, grad = 0u, fixed = 0u;
    int cnt = 0;
#pragma unroll
    for (int j = 0; j < E; ++j) {
        F[j] = 0.0;
        src[j] = t;
    }
    if (c < m.n) {
        Entries e;
        load_entries(m, c, e);
        Tc = __ldcg(&T[c]);
        iv = __ldg(&m.invV[c]);
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const int cd = e.code[j];
            if (cd == FVGB_PAD) continue;
            cnt = j + 1;
            F[j] = __ldg(&flux[entry_face(cd)]);
            const bool own = cd >= 0;
            if (own) plus |= 1u << j;  // boundary faces are the cell's own too
            const int o = e.other[j], d = o - first, mine = 2 * bs + j * bs + t;
            if (cd >= m.nif) {
                bnd |= 1u << j;
                src[j] = mine;
                sm[mine] = __ldcg(&T_b[o]);
                scell[j * bs + t] = o;
                const int ty = pt.type[__ldg(&m.bpatch[o])];
                if (ty == FVGB_BC_FIXED_VALUE) {
                    fixed |= 1u << j;
                    bq[j * bs + t] = __ldg(&ref[o]);
                } else if (ty == FVGB_BC_FIXED_GRADIENT) {
                    grad |= 1u << j;
                    bq[j * bs + t] = __ldg(&ref[o]) / __ldg(&m.bdelta[o]);
                }
                continue;
            }
            const bool away = (unsigned)d >= (unsigned)bs;
            if (away) {
                remote |= 1u << j;
                scell[j * bs + t] = o;
            }
            if (nonneg(F[j]) != own) src[j] = away ? mine : d;  // the value across, else the cell's own
            if (src[j] < bs) local |= 1u << j;
        }
    }
    sm[t] = Tc;
    bool bad = false;
    const bool full = __all_sync(0xffffffffu, cnt == E);
    LLWord *from = ll, *to = ll + m.n, *spare = ll + 2 * (size_t)m.n;  // step k - 1's cells, step k's, the next's
    __syncthreads();
    for (int k = 1; k <= nsteps; ++k) {
        const int par = ((k - 1) & 1) * bs;
        // Cells of other blocks: the first poll goes out at once, and the boundary
        // values of the step before are formed during its round trip (~600 clocks).
        unsigned long long a[E], b[E];
        unsigned left = k > 1 ? remote : 0u;
#pragma unroll
        for (int j = 0; j < E; ++j)
            if (left >> j & 1u) ll_issue(from + scell[j * bs + t], &a[j], &b[j]);
        if (k == 1) {
            for (int j = 0; j < E; ++j)
                if (remote >> j & 1u) slot[j * bs + t] = __ldcg(&T[scell[j * bs + t]]);
        } else if (grad | fixed) {
#pragma unroll
            for (int j = 0; j < E; ++j) {
                if (grad >> j & 1u) slot[j * bs + t] = Tc + bq[j * bs + t];
                if (fixed >> j & 1u) slot[j * bs + t] = bq[j * bs + t];
            }
        }
#pragma unroll 1
        for (unsigned spins = 0; left; ++spins) {
#pragma unroll
            for (int j = 0; j < E; ++j)
                if ((left >> j & 1u) && ll_take(a[j], b[j], (unsigned)(k - 1), &slot[j * bs + t])) left &= ~(1u << j);
            if (left && ll_give_up(gb, spins)) {
                bad = true;
                break;
            }
#pragma unroll
            for (int j = 0; j < E; ++j)
                if (left >> j & 1u) ll_issue(from + scell[j * bs + t], &a[j], &b[j]);
        }
        LLWord* seen = from;  // from now on `from` is step k's buffer
        from = to;
        to = spare;
        spare = seen;
        double p[E], s;
#pragma unroll
        for (int j = 0; j < E; ++j) p[j] = sm[src[j] + (local >> j & 1u ? par : 0)];
#pragma unroll
        for (int j = 0; j < E; ++j) p[j] = fmul(m, F[j], p[j]);
        s = cnt > 0 ? facc0(plus & 1u, p[0]) : 0.0;
        if (full) {
#pragma unroll
            for (int j = 1; j < E; ++j) s = facc(m, s, plus >> j & 1u, p[j]);
        } else {
#pragma unroll
            for (int j = 1; j < E; ++j) {
                const double a = facc(m, s, plus >> j & 1u, p[j]);
                s = j < cnt ? a : s;
            }
        }
        const double dv = facc0(true, fmul(m, s, iv));  // +0 + s/V
        Tc = fsub(m, Tc, fmul(m, dt, dv));
        if (remote) ll_store(from + c, Tc, (unsigned)k);
        sm[(k & 1) * bs + t] = Tc;
        if (__syncthreads_or(bad)) {
            bad = true;
            break;
        }
    }
#pragma unroll
    for (int j = 0; j < E; ++j) {
        if (grad >> j & 1u) slot[j * bs + t] = Tc + bq[j * bs + t];
        if (fixed >> j & 1u) slot[j * bs + t] = bq[j * bs + t];
    }
    if (c < m.n) {
        // a wait that ran out (seconds) leaves no number that could pass for a result
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        T[c] = bad ? nan : Tc;
        for (int j = 0; j < cnt; ++j)
            if (bnd >> j & 1u) T_b[scell[j * bs + t]] = bad ? nan : slot[j * bs + t];
    }
}

struct AdvectPlan {
    const void* fn = nullptr;  // null: the steps run one launch each
    int threads = 0;
    size_t smem = 0;
};

// One block per SM, from one warp per scheduler (128 threads) up, so that a step's
// DFMA chain shares its scheduler with as few warps as the mesh allows; faces per
// cell 4 (one-cell-thick meshes), 6 or 8.  None for wider cells, for more cells than
// one 1024-thread block per SM holds, or for fewer than 4 steps (a block that is
// done must not overtake a neighbour's first step: at least 3).
inline AdvectPlan advect_plan(const fvgb_mesh* m, int nsteps) {
    AdvectPlan p;
    int dev = 0, sms = 0, coop = 0;
    if (nsteps < 4 || m->g_width > kG || cudaGetDevice(&dev) != cudaSuccess) return p;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    const int64_t per_sm = ((int64_t)m->v.n + sms - 1) / sms;
    const int bs = (int)std::max<int64_t>(128, (per_sm + 127) / 128 * 128);
    if (!coop || per_sm > 1024) return p;
    const int E = m->g_width <= 4 ? 0 : (m->g_width <= 6 ? 1 : 2), r = bs <= 256 ? 0 : (bs <= 512 ? 1 : 2);
    static const void* const fns[3][3] = {
        {(const void*)k_advect_steps<256, 4>, (const void*)k_advect_steps<256, 6>, (const void*)k_advect_steps<256, 8>},
        {(const void*)k_advect_steps<512, 4>, (const void*)k_advect_steps<512, 6>, (const void*)k_advect_steps<512, 8>},
        {(const void*)k_advect_steps<1024, 4>, (const void*)k_advect_steps<1024, 6>,
         (const void*)k_advect_steps<1024, 8>}};
    const void* fn = fns[r][E];
    const int width = 4 + 2 * E, largest = 256 << r;
    const size_t per_thread = 8 * (2 + 2 * width) + 4 * width;
    p.smem = bs * per_thread;
    // the limit belongs to the kernel, not to this call: always its largest block's,
    // so that calls on other threads never lower it under a launch
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(largest * per_thread)) !=
        cudaSuccess) {
        cudaGetLastError();
        return p;
    }
    p.fn = fn;
    p.threads = bs;
    return p;
}

// meshes up to this size advance with the one-pass step kernel (k_advect_euler,
// one launch per step and no face buffer); larger ones with the two-pass step
constexpr int kStepsMaxCells = 1 << 16;

// ----------------------------------------------------------------------- grad
__device__ __forceinline__ void grad_entry(const MeshView& m, int code, double To, double wf, const double* S,
                                           double Tc, double& g0, double& g1, double& g2) {
    if (code >= m.nif) {
        g0 = fadd(m, g0, fmul(m, S[0], To));
        g1 = fadd(m, g1, fmul(m, S[1], To));
        g2 = fadd(m, g2, fmul(m, S[2], To));
        return;
    }
    const bool isOwner = code >= 0;
    const double Town = isOwner ? Tc : To;
    const double Tnei = isOwner ? To : Tc;
    const double tf = fadd(m, fmul(m, wf, fsub(m, Town, Tnei)), Tnei);
    g0 = facc(m, g0, isOwner, fmul(m, S[0], tf));
    g1 = facc(m, g1, isOwner, fmul(m, S[1], tf));
    g2 = facc(m, g2, isOwner, fmul(m, S[2], tf));
}

template <bool ADD>
__global__ void __launch_bounds__(kThreads)
    k_grad(MeshView m, const double* __restrict__ phi, const double* __restrict__ phi_b,
           double coeff, int unit, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    Entries e;
    load_entries(m, c, e);
    const double Tc = __ldg(&phi[c]);
    double T[kG], W[kG], S[kG][3];
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        const int cd = e.code[j];
        T[j] = W[j] = S[j][0] = S[j][1] = S[j][2] = 0.0;
        if (cd == FVGB_PAD) continue;
        const bool bnd = cd >= m.nif;
        const int f = entry_face(cd);
        const double* src = bnd ? phi_b : phi;
        T[j] = __ldg(&src[e.other[j]]);
        const double* sf = bnd ? m.bSf + 3 * (cd - m.nif) : m.Sf + 3 * f;
        S[j][0] = __ldg(&sf[0]);
        S[j][1] = __ldg(&sf[1]);
        S[j][2] = __ldg(&sf[2]);
        if (!bnd) W[j] = __ldg(&m.w[f]);
    }
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        if (e.code[j] == FVGB_PAD) break;
        grad_entry(m, e.code[j], T[j], W[j], S[j], Tc, g0, g1, g2);
    }
    for (int j = kG; j < e.width; ++j) {
        const int cd = __ldg(&m.g_code[e.base + j * 32]);
        if (cd == FVGB_PAD) break;
        const int o = __ldg(&m.g_other[e.base + j * 32]);
        const bool bnd = cd >= m.nif;
        const int f = entry_face(cd);
        const double* sf = bnd ? m.bSf + 3 * (cd - m.nif) : m.Sf + 3 * f;
        const double Sv[3] = {__ldg(&sf[0]), __ldg(&sf[1]), __ldg(&sf[2])};
        grad_entry(m, cd, __ldg(&(bnd ? phi_b : phi)[o]), bnd ? 0.0 : __ldg(&m.w[f]), Sv, Tc, g0, g1, g2);
    }
    const double sc = unit ? __ldg(&m.invV[c]) : coeff / __ldg(&m.V[c]);
    const double t[3] = {fmul(m, g0, sc), fmul(m, g1, sc), fmul(m, g2, sc)};
#pragma unroll
    for (int d = 0; d < 3; ++d) out[3 * c + d] = ADD ? fadd(m, out[3 * c + d], t[d]) : facc0(true, t[d]);
}

// ------------------------------------------------------------------ laplacian
// face flux g*(T_nei - T_own); the owner adds it, the neighbour subtracts it;
// a boundary face adds g_b*(T_b - T_c)
template <int NC>
__device__ __forceinline__ void lap_entry(const MeshView& m, int code, double g, const double* To, const double* Tc,
                                          double* s) {
    if (code >= m.nif) {
#pragma unroll
        for (int k = 0; k < NC; ++k) s[k] = fadd(m, s[k], fmul(m, g, fsub(m, To[k], Tc[k])));
        return;
    }
    const bool isOwner = code >= 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        // owner: s + g*(To - Tc); neighbour: s - g*(Tc - To), the reference's face flux
        const double a = isOwner ? To[k] : Tc[k], b = isOwner ? Tc[k] : To[k];
        s[k] = facc(m, s[k], isOwner, fmul(m, g, fsub(m, a, b)));
    }
}

template <int NC>
__global__ void __launch_bounds__(kThreads)
    k_lap(MeshView m, const double* __restrict__ gamma, const double* __restrict__ phi,
          const double* __restrict__ phi_b, double coeff, int unit, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    Entries e;
    load_entries(m, c, e);
    double Tc[NC], s[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        Tc[k] = __ldg(&phi[c * NC + k]);
        s[k] = 0.0;
    }
    double Gm[kG], Ge[kG], T[kG][NC];
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        const int cd = e.code[j];
        Gm[j] = Ge[j] = 0.0;
#pragma unroll
        for (int k = 0; k < NC; ++k) T[j][k] = 0.0;
        if (cd == FVGB_PAD) continue;
        const bool bnd = cd >= m.nif;
        const int f = entry_face(cd);
        Gm[j] = __ldg(&gamma[f]);
        Ge[j] = bnd ? __ldg(&m.bgeo[cd - m.nif]) : __ldg(&m.geo[f]);
        const double* src = bnd ? phi_b : phi;
#pragma unroll
        for (int k = 0; k < NC; ++k) T[j][k] = __ldg(&src[e.other[j] * NC + k]);
    }
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        if (e.code[j] == FVGB_PAD) break;
        lap_entry<NC>(m, e.code[j], fmul(m, Gm[j], Ge[j]), T[j], Tc, s);
    }
    for (int j = kG; j < e.width; ++j) {
        const int cd = __ldg(&m.g_code[e.base + j * 32]);
        if (cd == FVGB_PAD) break;
        const int o = __ldg(&m.g_other[e.base + j * 32]);
        const bool bnd = cd >= m.nif;
        const int f = entry_face(cd);
        const double g = fmul(m, __ldg(&gamma[f]), bnd ? __ldg(&m.bgeo[cd - m.nif]) : __ldg(&m.geo[f]));
        double To[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) To[k] = __ldg(&(bnd ? phi_b : phi)[o * NC + k]);
        lap_entry<NC>(m, cd, g, To, Tc, s);
    }
    const double sc = unit ? __ldg(&m.invV[c]) : coeff / __ldg(&m.V[c]);
#pragma unroll
    for (int k = 0; k < NC; ++k) out[c * NC + k] = fadd(m, out[c * NC + k], fmul(m, s[k], sc));
}

// --------------------------------------------------------------------- snGrad
struct SnGrad {
    static constexpr int kBatch = 2;
    struct Face { int P, N; double d; };
    using Cells = PairOf<1>;
    const double *phi, *phi_b;
    double* out;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.d = __ldg(&m.delta[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const { t.load(phi, a.P, a.N); }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
        out[f] = imul(a.d, fsub(m, t.n[0], t.p[0]));
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
        out[f] = fmul(m, __ldg(&m.bdelta[b]), fsub(m, __ldg(&phi_b[b]), __ldg(&phi[__ldg(&m.bcells[b])])));
    }
};

// ------------------------------------------------------ face-flux two passes
// Linear div, grad and laplacian: a face pass evaluates each face's flux ONCE
// (face value, then the product), as the reference's face loop does, into a
// face buffer; a cell pass then adds it (owner and boundary faces) or
// subtracts it (neighbour faces) in ascending face order.  The operations are
// those of the one-pass gather above, which evaluated every face from both of
// its cells: same bits, about half the FP64 work per face.  fx holds the faces'
// values component by component, boundary faces after the internal ones (index
// nif + b = entry code): a warp's stores are whole lines, and the three faces that a
// cell owns lie together for the cell pass.
template <int NC>
struct FluxDivLinear {
    static constexpr int kBatch = NC == 1 ? 2 : 1;
    struct Face { int P, N; double F, w; };
    using Cells = PairOf<NC>;
    const double *flux, *phi, *phi_b;
    double* fx;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.F = __ldg(&flux[f]);
        a.w = __ldg(&m.w[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const { t.load(phi, a.P, a.N); }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double d = fsub(m, t.p[c], t.n[c]);
            fx[c * (m.nif + m.nbf) + f] = imul(a.F, fadd(m, imul(a.w, d), t.n[c]));
        }
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
        const double F = __ldg(&flux[f]);
#pragma unroll
        for (int c = 0; c < NC; ++c) fx[c * (m.nif + m.nbf) + f] = fmul(m, F, __ldg(&phi_b[b * NC + c]));
    }
};

template <int NC>
struct FluxDivUpwind {
    static constexpr int kBatch = NC == 1 ? 2 : 1;
    struct Face { int P, N; double F; };
    struct Cells { double v[NC]; };
    const double *flux, *phi, *phi_b;
    double* fx;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.F = __ldg(&flux[f]);
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const {
        const int u = nonneg(a.F) ? a.P : a.N;
#pragma unroll
        for (int c = 0; c < NC; ++c) t.v[c] = __ldg(&phi[u * NC + c]);
    }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) fx[c * (m.nif + m.nbf) + f] = fmul(m, a.F, t.v[c]);
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
        const double F = __ldg(&flux[f]);
#pragma unroll
        for (int c = 0; c < NC; ++c) fx[c * (m.nif + m.nbf) + f] = fmul(m, F, __ldg(&phi_b[b * NC + c]));
    }
};

// S_f T_f of each component, T_f linear: the face terms of the Gauss gradient
template <int NC>
struct FluxGrad {
    static constexpr int kBatch = NC == 1 ? 2 : 1;
    struct Face { int P, N; double w, S[3]; };
    using Cells = PairOf<NC>;
    const double *phi, *phi_b;
    double* fx;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.w = __ldg(&m.w[f]);
#pragma unroll
        for (int d = 0; d < 3; ++d) a.S[d] = __ldg(&m.Sf[3 * f + d]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const { t.load(phi, a.P, a.N); }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double tf = fadd(m, imul(a.w, fsub(m, t.p[c], t.n[c])), t.n[c]);
            fx[3 * c * (m.nif + m.nbf) + f] = imul(a.S[0], tf);
            fx[(3 * c + 1) * (m.nif + m.nbf) + f] = imul(a.S[1], tf);
            fx[(3 * c + 2) * (m.nif + m.nbf) + f] = imul(a.S[2], tf);
        }
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const double tb = __ldg(&phi_b[b * NC + c]);
#pragma unroll
            for (int d = 0; d < 3; ++d) fx[(3 * c + d) * (m.nif + m.nbf) + f] = fmul(m, __ldg(&m.bSf[3 * b + d]), tb);
        }
    }
};

template <int NC>
struct FluxLap {
    static constexpr int kBatch = NC == 1 ? 2 : 1;
    struct Face { int P, N; double gamma, geo; };
    using Cells = PairOf<NC>;
    const double *gamma, *phi, *phi_b;
    double* fx;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.gamma = __ldg(&gamma[f]);
        a.geo = __ldg(&m.geo[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const { t.load(phi, a.P, a.N); }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
        const double g = imul(a.gamma, a.geo);
#pragma unroll
        for (int c = 0; c < NC; ++c) fx[c * (m.nif + m.nbf) + f] = imul(g, fsub(m, t.n[c], t.p[c]));
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
        const int P = __ldg(&m.bcells[b]);
        const double g = fmul(m, __ldg(&gamma[f]), __ldg(&m.bgeo[b]));
#pragma unroll
        for (int c = 0; c < NC; ++c)
            fx[c * (m.nif + m.nbf) + f] = fmul(m, g, fsub(m, __ldg(&phi_b[b * NC + c]), __ldg(&phi[P * NC + c])));
    }
};

// ------------------------------------------- non-orthogonal correction
// OpenFOAM's correctedSnGrad: snGrad_f = delta_f (T_N - T_P) + k_f . (grad T)_f,
// k_f the mesh's correction vector, (grad T)_f the linear interpolation
// w (g_P - g_N) + g_N of the Gauss linear cell gradient; boundary faces of the
// (non-coupled) patches carry no correction.  The gradient of each of the NC
// components comes from FluxGrad + k_gather_fx<3*NC>: for NC = 1 the
// operations of fvgb_grad exactly.
enum CorrMode { kCorrLaplacian = 0, kCorrOnly = 1, kCorrSnGrad = 2 };

// kCorrLaplacian: fma(gamma_f|Sf|delta_f, T_N - T_P, gamma_f|Sf| (k . grad_f)),
//                 boundary faces gamma_b|Sf_b|delta_b (T_b - T_P) (as FluxLap);
// kCorrOnly:      gamma_f|Sf| (k . grad_f), boundary faces 0 (faceFluxCorrection);
// kCorrSnGrad:    fma(delta_f, T_N - T_P, k . grad_f), boundary delta_b (T_b - T_P).
// grad: [n][NC][3]; grad_f = fma(w, g_P - g_N, g_N) per direction and
// k . grad_f = fma(k_z, g_z, fma(k_y, g_y, k_x g_x)): fused multiply-adds, 14
// FP64 operations per face and component where separate roundings took 20 (the
// pass is bound by GB300's FP64 issue rate).  With k = 0 the flux is exactly the
// uncorrected one: fma(a, b, 0) rounds a*b once, as the plain product does.
template <int NC, int MODE>
struct FluxCorr {
    static constexpr int kBatch = 1;
    struct Face { int P, N; double w, k[3], gamma, magSf, geo; };  // geo: delta for kCorrSnGrad
    struct Cells { PairOf<NC> t; PairOf<3 * NC> g; };
    const double *gamma, *phi, *phi_b, *grad;
    double* fx;
    __device__ __forceinline__ void fetch(const MeshView& m, int f, Face& a) const {
        a.P = __ldg(&m.own[f]);
        a.N = __ldg(&m.nei[f]);
        a.w = __ldg(&m.w[f]);
#pragma unroll
        for (int d = 0; d < 3; ++d) a.k[d] = __ldg(&m.corr[3 * f + d]);
        if (MODE != kCorrSnGrad) {
            a.gamma = __ldg(&gamma[f]);
            a.magSf = __ldg(&m.magSf[f]);
        }
        if (MODE != kCorrOnly) a.geo = MODE == kCorrSnGrad ? __ldg(&m.delta[f]) : __ldg(&m.geo[f]);
    }
    __device__ __forceinline__ void gather(const Face& a, Cells& t) const {
        t.g.load(grad, a.P, a.N);
        if (MODE != kCorrOnly) t.t.load(phi, a.P, a.N);
    }
    __device__ __forceinline__ void inner(const MeshView& m, int f, const Face& a, const Cells& t) const {
        const double gm = MODE == kCorrSnGrad ? 1.0 : imul(a.gamma, a.magSf);
        const double gg = MODE == kCorrLaplacian ? imul(a.gamma, a.geo) : a.geo;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            double gf[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) gf[d] = fma(a.w, fsub(m, t.g.p[3 * c + d], t.g.n[3 * c + d]), t.g.n[3 * c + d]);
            const double kg = fma(a.k[2], gf[2], fma(a.k[1], gf[1], imul(a.k[0], gf[0])));
            double v;
            if (MODE == kCorrOnly) v = fmul(m, gm, kg);
            else v = fma(gg, fsub(m, t.t.n[c], t.t.p[c]), MODE == kCorrLaplacian ? imul(gm, kg) : kg);
            fx[c * (m.nif + m.nbf) + f] = v;
        }
    }
    __device__ __forceinline__ void boundary(const MeshView& m, int f, int b) const {
        const int P = __ldg(&m.bcells[b]);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            double v = 0.0;
            if (MODE != kCorrOnly) {
                const double dT = fsub(m, __ldg(&phi_b[b * NC + c]), __ldg(&phi[P * NC + c]));
                const double g = MODE == kCorrLaplacian ? fmul(m, __ldg(&gamma[f]), __ldg(&m.bgeo[b])) : __ldg(&m.bdelta[b]);
                v = fmul(m, g, dT);
            }
            fx[c * (m.nif + m.nbf) + f] = v;
        }
    }
};

// out_f += coeff * fx_f on the internal faces
__global__ void __launch_bounds__(kThreads)
    k_axpy_faces(int64_t count, int nc, int64_t nf, double coeff, const double* __restrict__ fx,
                 double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = out[i] + coeff * __ldg(&fx[i % nc * nf + i / nc]);
}

// out_c += (sum over the cell's faces, ascending, of +-fx_f) * scale, with
// scale = coeff/V_c (mode 0), 1/V_c (mode 1: coeff 1) or coeff (mode 2: volume integrated).
// Blocks of 128 threads, 16 an SM for one component and 8 for three (64 registers):
// with blocks of 256 the registers left room for 48 and 24 warps (128^3 cells: 39 and
// 96 us, now 35 and 85).  ADD false: out_c = +0 + that, for a buffer that would be zeroed.
template <int NC, bool ADD>
__global__ void __launch_bounds__(kGatherThreads, NC == 1 ? 16 : NC == 3 ? 8 : 1)
    k_gather_fx(MeshView m, const double* __restrict__ fx, double coeff, int unit, double* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    Entries e;
    load_entries(m, c, e);
    double v[kG][NC];
#pragma unroll
    for (int j = 0; j < kG; ++j) {
#pragma unroll
        for (int k = 0; k < NC; ++k) v[j][k] = 0.0;
        if (e.code[j] == FVGB_PAD) continue;
        const int f = entry_face(e.code[j]);
#pragma unroll
        for (int k = 0; k < NC; ++k) v[j][k] = __ldg(&fx[k * (m.nif + m.nbf) + f]);
    }
    // owner and boundary faces add, neighbour faces subtract; the sum starts
    // from +0, so its first term is taken exactly on the integer pipes (a
    // padded first entry holds 0 and gives +0)
    double s[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) s[k] = facc0(e.code[0] >= 0, v[0][k]);
#pragma unroll
    for (int j = 1; j < kG; ++j) {
        if (e.code[j] == FVGB_PAD) break;
        const bool plus = e.code[j] >= 0;
#pragma unroll
        for (int k = 0; k < NC; ++k) s[k] = facc(m, s[k], plus, v[j][k]);
    }
    for (int j = kG; j < e.width; ++j) {
        const int cd = __ldg(&m.g_code[e.base + j * 32]);
        if (cd == FVGB_PAD) break;
        const int f = entry_face(cd);
#pragma unroll
        for (int k = 0; k < NC; ++k) s[k] = facc(m, s[k], cd >= 0, __ldg(&fx[k * (m.nif + m.nbf) + f]));
    }
    const double sc = unit == 1 ? __ldg(&m.invV[c]) : unit == 2 ? coeff : coeff / __ldg(&m.V[c]);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const double t = imul(s[k], sc);
        out[c * NC + k] = ADD ? fadd(m, out[c * NC + k], t) : facc0(true, t);
    }
}

// q_b = ref_b / delta_b of every fixed-gradient boundary face, whose boundary
// value is then T_P + q_b.  Formed here by whole warps over the boundary faces:
// in the gather only the one boundary lane of a cell warp needs it (a warp of
// cells along x meets one x wall), and the FP64 division's instruction sequence
// then ran at 1/32 lane use in half the warps, which kept the FP64 pipe busy.
__global__ void __launch_bounds__(kThreads)
    k_bc_gradq(MeshView m, PatchTable pt, const double* __restrict__ ref, double* __restrict__ q) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= m.nbf) return;
    q[b] = pt.type[__ldg(&m.bpatch[b])] == FVGB_BC_FIXED_GRADIENT ? __ldg(&ref[b]) / __ldg(&m.bdelta[b]) : 0.0;
}

// The fused upwind advection step on a face-flux buffer: the divergence as in
// k_gather_fx (coefficient 1), then the forward-Euler update and the boundary
// correction of k_advect_euler (the fixed-gradient quotients from k_bc_gradq).
__global__ void __launch_bounds__(kThreads, 6)
    k_advect_gather(MeshView m, PatchTable pt, const double* __restrict__ fx, const double* __restrict__ Told,
                    const double* __restrict__ Told_b, double dt, const double* __restrict__ ref,
                    const double* __restrict__ gq, double* __restrict__ Tnew, double* __restrict__ Tnew_b) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.n) return;
    Entries e;
    load_entries(m, c, e);
    double v[kG];
#pragma unroll
    for (int j = 0; j < kG; ++j) v[j] = e.code[j] == FVGB_PAD ? 0.0 : __ldg(&fx[entry_face(e.code[j])]);
    double s = facc0(e.code[0] >= 0, v[0]);  // the sum from +0: its first term exactly, on the integer pipes
#pragma unroll
    for (int j = 1; j < kG; ++j) {
        if (e.code[j] == FVGB_PAD) break;
        s = facc(m, s, e.code[j] >= 0, v[j]);
    }
    for (int j = kG; j < e.width; ++j) {
        const int cd = __ldg(&m.g_code[e.base + j * 32]);
        if (cd == FVGB_PAD) break;
        s = facc(m, s, cd >= 0, __ldg(&fx[entry_face(cd)]));
    }
    const double dv = facc0(true, fmul(m, s, __ldg(&m.invV[c])));  // +0 + s/V
    const double tn = fsub(m, __ldg(&Told[c]), fmul(m, dt, dv));
    Tnew[c] = tn;
    // boundary faces of this cell (its last entries): the entries held in
    // registers are tested in an unrolled loop, any beyond them reloaded
#pragma unroll
    for (int j = 0; j < kG; ++j) {
        const int code = e.code[j];
        if (code == FVGB_PAD || code < m.nif) continue;
        const int b = code - m.nif;
        const int t = pt.type[__ldg(&m.bpatch[b])];
        double bv = __ldg(&Told_b[b]);
        if (t == FVGB_BC_FIXED_VALUE) bv = __ldg(&ref[b]);
        else if (t == FVGB_BC_FIXED_GRADIENT) bv = tn + __ldg(&gq[b]);
        Tnew_b[b] = bv;
    }
    for (int j = kG; j < e.width; ++j) {
        const int code = __ldg(&m.g_code[e.base + j * 32]);
        if (code == FVGB_PAD || code < m.nif) continue;
        const int b = code - m.nif;
        const int t = pt.type[__ldg(&m.bpatch[b])];
        double bv = __ldg(&Told_b[b]);
        if (t == FVGB_BC_FIXED_VALUE) bv = __ldg(&ref[b]);
        else if (t == FVGB_BC_FIXED_GRADIENT) bv = tn + __ldg(&gq[b]);
        Tnew_b[b] = bv;
    }
}

template <class Op>
void launch_faces(const fvgb_mesh* m, const Op& op, cudaStream_t s) {
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    FVGB_FACE_TILE(m->face_tile,
                   k_faces<FPT><<<grid_for(nf, kFaceThreads * FPT), kFaceThreads, 0, s>>>(m->v, op))
}

template <int NC, bool ADD = true>
void gather_faces(const fvgb_mesh* m, const double* fx, double coeff, int mode, double* out, cudaStream_t s) {
    k_gather_fx<NC, ADD><<<grid_for(m->v.n, kGatherThreads), kGatherThreads, 0, s>>>(m->v, fx, coeff, mode, out);
}

// Face buffer from the stream-ordered pool (no device synchronisation); the
// pool keeps its memory between calls.  nullptr when it cannot be had: the
// caller then runs the one-pass gather, which needs none.
double* face_buffer(size_t count, cudaStream_t s) {
    static std::atomic<bool> pool_ready{false};  // the setting is idempotent: a racing second setter is harmless
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!pool_ready.load(std::memory_order_acquire) && cudaStreamIsCapturing(s, &cap) == cudaSuccess &&
        cap == cudaStreamCaptureStatusNone) {
        // not while a graph is being captured (there the allocation becomes a graph memory node)
        int dev = 0;
        cudaMemPool_t pool;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
            uint64_t keep = ~0ull;
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        pool_ready.store(true, std::memory_order_release);
    }
    double* p = nullptr;
    if (cudaMallocAsync((void**)&p, sizeof(double) * (count ? count : 1), s) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

// Div, gradient and Laplacian of a small mesh take the one-pass gather: one launch
// and no face buffer instead of two launches and an allocation, and its doubled FP64
// work hides behind latency as long as every block of cells has an SM to itself.
// Measured per call, two passes and one: 24,389 cells, scalar div 13.2 and 9.1 us,
// vector div 15.1 and 13.1, gradient 14.4 and 11.1; 64,000 cells 12.6 and 11.1, 16.9 and
// 23.1, 16.3 and 19.0; 262,144 cells 17.2 and 27.3, 31.6 and 64.6, 27.4 and 49.4.
constexpr int kOnePassCells = 152 * kThreads;
bool one_pass(const fvgb_mesh* m) { return m->v.n <= kOnePassCells; }

// The Gauss linear gradient of every component of psi into grad [n*nc*3], on a face
// buffer.
fvgb_status gauss_grad_components(const fvgb_mesh* m, int nc, const double* psi, const double* psi_b, double* grad,
                                  cudaStream_t s) {
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    if (nc == 1 && one_pass(m)) {
        k_grad<false><<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(m->v, psi, psi_b, 1.0, 1, grad);
        return FVGB_OK;
    }
    double* fx = face_buffer((size_t)(nf * nc * 3), s);
    if (!fx) return fvgb_fail(FVGB_ERR_OOM, "non-orthogonal correction: no face buffer");
    if (nc == 1) {
        launch_faces(m, FluxGrad<1>{psi, psi_b, fx}, s);
        gather_faces<3, false>(m, fx, 1.0, 1, grad, s);
    } else {
        launch_faces(m, FluxGrad<3>{psi, psi_b, fx}, s);
        gather_faces<9, false>(m, fx, 1.0, 1, grad, s);
    }
    cudaFreeAsync(fx, s);
    return FVGB_OK;
}

// One corrected face pass (MODE) of psi into `dst` [nf*nc], or into a face buffer that
// the caller frees when that is null.  nullptr with the error set when buffers cannot
// be had.
template <int MODE>
double* corrected_faces(const fvgb_mesh* m, int nc, const double* gamma, const double* psi, const double* psi_b,
                        cudaStream_t s, double* dst = nullptr) {
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    double* grad = face_buffer((size_t)m->v.n * nc * 3, s);
    if (!grad) {
        fvgb_fail(FVGB_ERR_OOM, "non-orthogonal correction: no gradient buffer");
        return nullptr;
    }
    if (gauss_grad_components(m, nc, psi, psi_b, grad, s) != FVGB_OK) {
        cudaFreeAsync(grad, s);
        return nullptr;
    }
    double* fx = dst ? dst : face_buffer((size_t)(nf * nc), s);
    if (fx) {
        if (nc == 1)
            launch_faces(m, FluxCorr<1, MODE>{gamma, psi, psi_b, grad, fx}, s);
        else
            launch_faces(m, FluxCorr<3, MODE>{gamma, psi, psi_b, grad, fx}, s);
    } else {
        fvgb_fail(FVGB_ERR_OOM, "non-orthogonal correction: no face buffer");
    }
    cudaFreeAsync(grad, s);
    return fx;
}

}  // namespace

fvgb_status nonorth_rhs(const fvgb_mesh* m, int nc, const double* gamma, const double* psi, const double* psi_b,
                        double coeff, double* out, cudaStream_t s) {
    double* fx = corrected_faces<kCorrOnly>(m, nc, gamma, psi, psi_b, s);
    if (!fx) return FVGB_ERR_OOM;
    if (nc == 1) gather_faces<1>(m, fx, coeff, 2, out, s);
    else gather_faces<3>(m, fx, coeff, 2, out, s);
    cudaFreeAsync(fx, s);
    FVGB_LAUNCH_CHECK("non-orthogonal correction");
    return FVGB_OK;
}

// ==================================================================== C ABI
#define CHECK_MESH_NC(m, nc, name)                                                         \
    FVGB_CHECK_ARG(m, name ": null mesh");                                                 \
    FVGB_CHECK_ARG((nc) == 1 || (nc) == 3, name ": ncomp must be 1 or 3")

extern "C" fvgb_status fvgb_interp_linear(const fvgb_mesh* m, int32_t nc, const double* src,
                                          const double* src_b, double* dst, fvgb_stream stream) {
    CHECK_MESH_NC(m, nc, "fvgb_interp_linear");
    FVGB_CHECK_ARG(src && dst && (src_b || m->v.nbf == 0), "fvgb_interp_linear: null field");
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    if (nf == 0) return FVGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (nc == 1)
        launch_faces(m, InterpLinear<1>{src, src_b, dst}, s);
    else
        launch_faces(m, InterpLinear<3>{src, src_b, dst}, s);
    FVGB_LAUNCH_CHECK("fvgb_interp_linear");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_interp_upwind(const fvgb_mesh* m, int32_t nc, const double* flux,
                                          const double* src, const double* src_b, double* dst,
                                          fvgb_stream stream) {
    CHECK_MESH_NC(m, nc, "fvgb_interp_upwind");
    FVGB_CHECK_ARG(flux && src && dst && (src_b || m->v.nbf == 0), "fvgb_interp_upwind: null field");
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    if (nf == 0) return FVGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (nc == 1)
        launch_faces(m, InterpUpwind<1>{flux, src, src_b, dst}, s);
    else
        launch_faces(m, InterpUpwind<3>{flux, src, src_b, dst}, s);
    FVGB_LAUNCH_CHECK("fvgb_interp_upwind");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_div_explicit(const fvgb_mesh* m, int32_t scheme, int32_t nc,
                                         const double* flux, const double* phi,
                                         const double* phi_b, double coeff, double* out,
                                         fvgb_stream stream) {
    CHECK_MESH_NC(m, nc, "fvgb_div_explicit");
    FVGB_CHECK_ARG(scheme == FVGB_SCHEME_LINEAR || scheme == FVGB_SCHEME_UPWIND,
                   "fvgb_div_explicit: unknown scheme");
    FVGB_CHECK_ARG(flux && phi && out && (phi_b || m->v.nbf == 0), "fvgb_div_explicit: null field");
    const int unit = coeff == 1.0;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned g = grid_for(m->v.n, kThreads);
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    double* fx = one_pass(m) ? nullptr : face_buffer((size_t)(nf * nc), s);
    if (fx) {
        const bool up = scheme == FVGB_SCHEME_UPWIND;
        if (nc == 1) {
            if (up)
                launch_faces(m, FluxDivUpwind<1>{flux, phi, phi_b, fx}, s);
            else
                launch_faces(m, FluxDivLinear<1>{flux, phi, phi_b, fx}, s);
            gather_faces<1>(m, fx, coeff, unit, out, s);
        } else {
            if (up)
                launch_faces(m, FluxDivUpwind<3>{flux, phi, phi_b, fx}, s);
            else
                launch_faces(m, FluxDivLinear<3>{flux, phi, phi_b, fx}, s);
            gather_faces<3>(m, fx, coeff, unit, out, s);
        }
        FVGB_LAUNCH_CHECK("fvgb_div_explicit");
        cudaFreeAsync(fx, s);
        return FVGB_OK;
    }
    if (nc == 1 && scheme == FVGB_SCHEME_UPWIND)
        k_div<1, FVGB_SCHEME_UPWIND><<<g, kThreads, 0, s>>>(m->v, flux, phi, phi_b, coeff, unit, out);
    else if (nc == 1)
        k_div<1, FVGB_SCHEME_LINEAR><<<g, kThreads, 0, s>>>(m->v, flux, phi, phi_b, coeff, unit, out);
    else if (scheme == FVGB_SCHEME_UPWIND)
        k_div<3, FVGB_SCHEME_UPWIND><<<g, kThreads, 0, s>>>(m->v, flux, phi, phi_b, coeff, unit, out);
    else
        k_div<3, FVGB_SCHEME_LINEAR><<<g, kThreads, 0, s>>>(m->v, flux, phi, phi_b, coeff, unit, out);
    FVGB_LAUNCH_CHECK("fvgb_div_explicit");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_grad(const fvgb_mesh* m, const double* phi, const double* phi_b,
                                 double coeff, double* out, fvgb_stream stream) {
    FVGB_CHECK_ARG(m, "fvgb_grad: null mesh");
    FVGB_CHECK_ARG(phi && out && (phi_b || m->v.nbf == 0), "fvgb_grad: null field");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    double* fx = one_pass(m) ? nullptr : face_buffer((size_t)(3 * nf), s);
    if (fx) {
        launch_faces(m, FluxGrad<1>{phi, phi_b, fx}, s);
        gather_faces<3>(m, fx, coeff, coeff == 1.0, out, s);
        FVGB_LAUNCH_CHECK("fvgb_grad");
        cudaFreeAsync(fx, s);
        return FVGB_OK;
    }
    k_grad<true><<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(m->v, phi, phi_b, coeff, coeff == 1.0, out);
    FVGB_LAUNCH_CHECK("fvgb_grad");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_laplacian_explicit(const fvgb_mesh* m, int32_t nc, const double* gamma,
                                               const double* phi, const double* phi_b,
                                               double coeff, double* out, fvgb_stream stream) {
    CHECK_MESH_NC(m, nc, "fvgb_laplacian_explicit");
    FVGB_CHECK_ARG(gamma && phi && out && (phi_b || m->v.nbf == 0),
                   "fvgb_laplacian_explicit: null field");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned g = grid_for(m->v.n, kThreads);
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    double* fx = one_pass(m) ? nullptr : face_buffer((size_t)(nf * nc), s);
    if (fx) {
        if (nc == 1) {
            launch_faces(m, FluxLap<1>{gamma, phi, phi_b, fx}, s);
            gather_faces<1>(m, fx, coeff, coeff == 1.0, out, s);
        } else {
            launch_faces(m, FluxLap<3>{gamma, phi, phi_b, fx}, s);
            gather_faces<3>(m, fx, coeff, coeff == 1.0, out, s);
        }
        FVGB_LAUNCH_CHECK("fvgb_laplacian_explicit");
        cudaFreeAsync(fx, s);
        return FVGB_OK;
    }
    if (nc == 1) k_lap<1><<<g, kThreads, 0, s>>>(m->v, gamma, phi, phi_b, coeff, coeff == 1.0, out);
    else k_lap<3><<<g, kThreads, 0, s>>>(m->v, gamma, phi, phi_b, coeff, coeff == 1.0, out);
    FVGB_LAUNCH_CHECK("fvgb_laplacian_explicit");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_sngrad(const fvgb_mesh* m, const double* phi, const double* phi_b,
                                   double* out, fvgb_stream stream) {
    FVGB_CHECK_ARG(m, "fvgb_sngrad: null mesh");
    FVGB_CHECK_ARG(phi && out && (phi_b || m->v.nbf == 0), "fvgb_sngrad: null field");
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    if (nf == 0) return FVGB_OK;
    launch_faces(m, SnGrad{phi, phi_b, out}, (cudaStream_t)stream);
    FVGB_LAUNCH_CHECK("fvgb_sngrad");
    return FVGB_OK;
}

#define CHECK_CORRECTED(m, name) \
    FVGB_CHECK_ARG((m)->v.corr || (m)->v.nif == 0, name ": the mesh was created without cell centres")

extern "C" fvgb_status fvgb_laplacian_explicit_corrected(const fvgb_mesh* m, int32_t nc, const double* gamma,
                                                         const double* phi, const double* phi_b, double coeff,
                                                         double* out, fvgb_stream stream) {
    fvgb_clear_error();
    CHECK_MESH_NC(m, nc, "fvgb_laplacian_explicit_corrected");
    CHECK_CORRECTED(m, "fvgb_laplacian_explicit_corrected");
    FVGB_CHECK_ARG(gamma && phi && out && (phi_b || m->v.nbf == 0), "fvgb_laplacian_explicit_corrected: null field");
    cudaStream_t s = (cudaStream_t)stream;
    double* fx = corrected_faces<kCorrLaplacian>(m, nc, gamma, phi, phi_b, s);
    if (!fx) return FVGB_ERR_OOM;
    if (nc == 1) gather_faces<1>(m, fx, coeff, coeff == 1.0, out, s);
    else gather_faces<3>(m, fx, coeff, coeff == 1.0, out, s);
    cudaFreeAsync(fx, s);
    FVGB_LAUNCH_CHECK("fvgb_laplacian_explicit_corrected");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_sngrad_corrected(const fvgb_mesh* m, const double* phi, const double* phi_b, double* out,
                                             fvgb_stream stream) {
    fvgb_clear_error();
    FVGB_CHECK_ARG(m, "fvgb_sngrad_corrected: null mesh");
    CHECK_CORRECTED(m, "fvgb_sngrad_corrected");
    FVGB_CHECK_ARG(phi && out && (phi_b || m->v.nbf == 0), "fvgb_sngrad_corrected: null field");
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    if (nf == 0) return FVGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (!corrected_faces<kCorrSnGrad>(m, 1, nullptr, phi, phi_b, s, out)) return FVGB_ERR_OOM;
    FVGB_LAUNCH_CHECK("fvgb_sngrad_corrected");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_nonorth_flux(const fvgb_mesh* m, int32_t nc, const double* gamma, const double* phi,
                                         const double* phi_b, double coeff, double* out, fvgb_stream stream) {
    fvgb_clear_error();
    CHECK_MESH_NC(m, nc, "fvgb_nonorth_flux");
    CHECK_CORRECTED(m, "fvgb_nonorth_flux");
    FVGB_CHECK_ARG(gamma && phi && out && (phi_b || m->v.nbf == 0), "fvgb_nonorth_flux: null field");
    if (m->v.nif == 0) return FVGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    double* fx = corrected_faces<kCorrOnly>(m, nc, gamma, phi, phi_b, s);
    if (!fx) return FVGB_ERR_OOM;
    const int64_t cnt = (int64_t)m->v.nif * nc;
    k_axpy_faces<<<grid_for(cnt, kThreads), kThreads, 0, s>>>(cnt, nc, (int64_t)m->v.nif + m->v.nbf, coeff, fx, out);
    cudaFreeAsync(fx, s);
    FVGB_LAUNCH_CHECK("fvgb_nonorth_flux");
    return FVGB_OK;
}

// One forward-Euler upwind step: the face pass and the fused gather on a
// face buffer (with the boundary quotients gq, formed here when null), or the
// one-pass step kernel when no face buffer can be had.
static fvgb_status advect_two_pass(const fvgb_mesh* m, const PatchTable& pt, const double* flux, const double* T_old,
                            const double* T_old_b, double dt, const double* ref, const double* gq, double* T_new,
                            double* T_new_b, cudaStream_t s) {
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    double* fx = face_buffer((size_t)(nf + (gq ? 0 : m->v.nbf)), s);  // face fluxes, then the quotients
    if (fx) {
        if (!gq) {
            double* q = fx + nf;
            k_bc_gradq<<<grid_for(m->v.nbf, kThreads), kThreads, 0, s>>>(m->v, pt, ref, q);
            gq = q;
        }
        launch_faces(m, FluxDivUpwind<1>{flux, T_old, T_old_b, fx}, s);
        k_advect_gather<<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(m->v, pt, fx, T_old, T_old_b, dt, ref, gq,
                                                                          T_new, T_new_b);
        FVGB_LAUNCH_CHECK("fvgb_advect_euler_step");
        cudaFreeAsync(fx, s);
        return FVGB_OK;
    }
    k_advect_euler<<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(m->v, pt, flux, T_old, T_old_b, dt, ref, gq,
                                                                   T_new, T_new_b);
    FVGB_LAUNCH_CHECK("fvgb_advect_euler_step");
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_advect_euler_steps(const fvgb_mesh* m, const double* flux, double* T, double* T_b,
                                               double dt, const fvgb_bc* bc, int32_t nsteps, double* work,
                                               double* work_b, fvgb_stream stream) {
    FVGB_CHECK_ARG(m && bc && nsteps >= 0, "fvgb_advect_euler_steps: bad argument");
    FVGB_CHECK_ARG(flux && T && work && ((T_b && work_b) || m->v.nbf == 0), "fvgb_advect_euler_steps: null field");
    FVGB_CHECK_ARG(T != work && (m->v.nbf == 0 || T_b != work_b), "fvgb_advect_euler_steps: work must not alias T");
    PatchTable pt;
    FVGB_CHECK_ARG(make_patch_table(m, bc->patch_type, &pt), "fvgb_advect_euler_steps: bad patch types");
    FVGB_CHECK_ARG(bc->ref || !patch_table_needs_ref(pt), "fvgb_advect_euler_steps: ref is null");
    if (nsteps == 0) return FVGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const AdvectPlan plan = advect_plan(m, nsteps);
    // GridBar, then the step buffers of the cells that cross blocks
    const size_t ex_bytes = 128 + sizeof(LLWord) * 3 * (size_t)m->v.n;
    char* ex = plan.fn ? (char*)face_buffer(ex_bytes / sizeof(double), s) : nullptr;
    if (ex) {
        MeshView v = m->v;
        const double* ref = bc->ref;
        GridBar* gb = (GridBar*)ex;
        LLWord* ll = (LLWord*)(ex + 128);
        cudaError_t e = cudaMemsetAsync(ex, 0, ex_bytes, s);
        void* args[] = {&v, &pt, &flux, &T, &T_b, &dt, &ref, &nsteps, &ll, &gb};
        if (e == cudaSuccess)
            e = cudaLaunchCooperativeKernel(plan.fn, dim3(grid_for(v.n, plan.threads)), dim3(plan.threads), args,
                                            plan.smem, s);
        cudaFreeAsync(ex, s);
        if (e == cudaSuccess) return FVGB_OK;
        cudaGetLastError();  // not launched (fewer SMs than the device's): a launch per step needs no co-residency
    }
    // the fixed-gradient boundary quotients ref/delta do not change between
    // steps: formed once for the whole call
    // (without the buffer each step forms its quotients itself)
    double* gq = m->v.nbf > 0 ? face_buffer((size_t)m->v.nbf, s) : nullptr;
    if (gq) k_bc_gradq<<<grid_for(m->v.nbf, kThreads), kThreads, 0, s>>>(m->v, pt, bc->ref, gq);
    fvgb_status st = FVGB_OK;
    if (m->v.n <= kStepsMaxCells) {
        for (int k = 0; k < nsteps; ++k) {
            const bool even = (k & 1) == 0;
            k_advect_euler<<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(
                m->v, pt, flux, even ? T : work, even ? T_b : work_b, dt, bc->ref, gq, even ? work : T,
                even ? work_b : T_b);
        }
    } else {
        for (int k = 0; k < nsteps && st == FVGB_OK; ++k) {
            const bool even = (k & 1) == 0;
            st = advect_two_pass(m, pt, flux, even ? T : work, even ? T_b : work_b, dt, bc->ref, gq,
                                 even ? work : T, even ? work_b : T_b, s);
        }
    }
    if (gq) cudaFreeAsync(gq, s);
    if (st != FVGB_OK) return st;
    FVGB_LAUNCH_CHECK("fvgb_advect_euler_steps");
    if (nsteps & 1) {  // the last step wrote the work buffers
        FVGB_CUDA_TRY(cudaMemcpyAsync(T, work, sizeof(double) * (size_t)m->v.n, cudaMemcpyDeviceToDevice, s));
        if (m->v.nbf > 0)
            FVGB_CUDA_TRY(cudaMemcpyAsync(T_b, work_b, sizeof(double) * (size_t)m->v.nbf, cudaMemcpyDeviceToDevice, s));
    }
    return FVGB_OK;
}

extern "C" fvgb_status fvgb_advect_euler_step(const fvgb_mesh* m, const double* flux,
                                              const double* T_old, const double* T_old_b,
                                              double dt, const fvgb_bc* bc, double* T_new,
                                              double* T_new_b, fvgb_stream stream) {
    FVGB_CHECK_ARG(m && bc, "fvgb_advect_euler_step: null argument");
    FVGB_CHECK_ARG(flux && T_old && T_new && ((T_old_b && T_new_b) || m->v.nbf == 0),
                   "fvgb_advect_euler_step: null field");
    FVGB_CHECK_ARG(T_new != T_old, "fvgb_advect_euler_step: T_new must not alias T_old");
    PatchTable pt;
    FVGB_CHECK_ARG(make_patch_table(m, bc->patch_type, &pt), "fvgb_advect_euler_step: bad patch types");
    FVGB_CHECK_ARG(bc->ref || !patch_table_needs_ref(pt), "fvgb_advect_euler_step: ref is null");
    cudaStream_t s = (cudaStream_t)stream;
    if (m->v.n <= kStepsMaxCells) {  // small meshes: one launch of the one-pass step kernel
        k_advect_euler<<<grid_for(m->v.n, kThreads), kThreads, 0, s>>>(m->v, pt, flux, T_old, T_old_b, dt, bc->ref,
                                                                       nullptr, T_new, T_new_b);
        FVGB_LAUNCH_CHECK("fvgb_advect_euler_step");
        return FVGB_OK;
    }
    return advect_two_pass(m, pt, flux, T_old, T_old_b, dt, bc->ref, nullptr, T_new, T_new_b, s);
}

// ------------------------------------------------------- face-pass tile
extern "C" fvgb_status fvgb_mesh_face_tile(fvgb_mesh* m, int32_t tile) {
    FVGB_CHECK_ARG(m, "fvgb_mesh_face_tile: null mesh");
    FVGB_CHECK_ARG(tile == 0 || tile == 2 || tile == 4 || tile == 8, "fvgb_mesh_face_tile: the tile is 2, 4 or 8");
    m->face_tile = tile == 0 ? 4 : tile;
    return FVGB_OK;
}

namespace {
// The tuning cache's key of a mesh shape for the face passes
std::string face_tune_key(const fvgb_mesh* m) {
    int dev = 0, sms = 0, cmaj = 0, cmin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&cmaj, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&cmin, cudaDevAttrComputeCapabilityMinor, dev);
    const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
    const int lg = nf > 0 ? (int)std::lround(std::log2((double)nf)) : 0;
    return "faces/sm" + std::to_string(cmaj * 10 + cmin) + "x" + std::to_string(sms) + "/faces2^" + std::to_string(lg);
}
constexpr int kTiles[3] = {2, 4, 8};
}  // namespace

// Times the face passes of grad and upwind div (the FP64-issue-bound and the
// memory-latency-bound kind) with each tile on scratch fields of this mesh and
// keeps the fastest; a tile cached for this mesh shape is taken untimed.
// Synchronises `stream`.
extern "C" fvgb_status fvgb_explicit_tune(fvgb_mesh* m, fvgb_stream stream, int32_t* tile_out, float* ms_out) {
    FVGB_CHECK_ARG(m, "fvgb_explicit_tune: null mesh");
    cudaStream_t s = (cudaStream_t)stream;
    const std::string key = face_tune_key(m);
    int cached = -1;
    float ms[4] = {0, 0, 0, 0};
    if (tune_cache_get(key, 0, &cached) && cached >= 0 && cached < 3) {
        m->face_tile = kTiles[cached];
    } else {
        const int64_t nf = (int64_t)m->v.nif + m->v.nbf;
        double *phi = nullptr, *phi_b = nullptr, *flux = nullptr, *fx = nullptr;
        cudaError_t e = cudaMallocAsync(&phi, sizeof(double) * (size_t)std::max<int64_t>(1, m->v.n), s);
        if (e == cudaSuccess) e = cudaMallocAsync(&phi_b, sizeof(double) * (size_t)std::max<int32_t>(1, m->v.nbf), s);
        if (e == cudaSuccess) e = cudaMallocAsync(&flux, sizeof(double) * (size_t)std::max<int64_t>(1, nf), s);
        if (e == cudaSuccess) e = cudaMallocAsync(&fx, sizeof(double) * 3 * (size_t)std::max<int64_t>(1, nf), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(phi, 0, sizeof(double) * (size_t)std::max<int64_t>(1, m->v.n), s);
        if (e == cudaSuccess)
            e = cudaMemsetAsync(phi_b, 0, sizeof(double) * (size_t)std::max<int32_t>(1, m->v.nbf), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(flux, 0, sizeof(double) * (size_t)std::max<int64_t>(1, nf), s);
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (e == cudaSuccess) e = cudaEventCreate(&e0);
        if (e == cudaSuccess) e = cudaEventCreate(&e1);
        int best = 1;
        for (int t = 0; t < 3 && e == cudaSuccess; ++t) {
            float times[3];
            for (int r = 0; r < 4 && e == cudaSuccess; ++r) {  // the first run warms up
                cudaEventRecord(e0, s);
                FVGB_FACE_TILE(kTiles[t],
                               k_faces<FPT><<<grid_for(nf, kFaceThreads * FPT), kFaceThreads, 0, s>>>(m->v, FluxGrad<1>{phi, phi_b, fx});
                               k_faces<FPT><<<grid_for(nf, kFaceThreads * FPT), kFaceThreads, 0, s>>>(m->v, FluxDivUpwind<1>{flux, phi, phi_b, fx}))
                cudaEventRecord(e1, s);
                e = cudaEventSynchronize(e1);
                if (e == cudaSuccess && r > 0) e = cudaEventElapsedTime(&times[r - 1], e0, e1);
            }
            std::sort(times, times + 3);
            ms[t] = times[1];
        }
        for (int t = 0; t < 3; ++t)
            if (ms[t] < ms[best]) best = t;
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        cudaFreeAsync(phi, s);
        cudaFreeAsync(phi_b, s);
        cudaFreeAsync(flux, s);
        cudaFreeAsync(fx, s);
        if (e != cudaSuccess) return cuda_fail(e, "fvgb_explicit_tune");
        m->face_tile = kTiles[best];
        tune_cache_put(key, 0, best, ms);
    }
    if (tile_out) *tile_out = m->face_tile;
    if (ms_out)
        for (int t = 0; t < 3; ++t) ms_out[t] = ms[t];
    return FVGB_OK;
}
