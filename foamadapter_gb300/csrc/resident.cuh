// Resident persistent solves: one cooperative launch runs a whole single-case
// solve with every block's part of the system held on its SM.  Included by
// solver.cu inside its anonymous namespace.
//
// Block b is virtual block b of the reduction tree: 256 threads, thread t owning
// its R tree rows row0 + (t/32)*32R + j*32 + t%32 (j < R), so every vector of a
// row lives in the registers of the thread that sums it and no dot product is
// staged.  The block's matrix slots are copied to shared memory once per solve,
// with each column as an index into the block's shared direction vector: own
// rows first, then one entry per slot that reaches into another block (a halo
// entry).  Only the halo and the dot products cross blocks.
//
// Everything that crosses blocks carries its epoch beside the data (ll.cuh).
//  * Halo: an owner publishes the preconditioned residual z of its rows; a
//    reader keeps its own copy of the halo's direction and forms the new one,
//    p = z + beta p, with the owner's arithmetic.
//  * Reductions: every block publishes its partial on a 128-byte line of its own
//    and a warp of every block polls all of them and forms the final tree and
//    the solver's scalars itself.  (With 128 blocks this hop takes 2,600-2,900
//    clocks; with the partials packed 8 to a line, 6,600: every write makes all
//    pollers fetch the line again.  A block that collects and answers takes
//    3,800.)
// Every wait is bounded; on time-out a block raises the abort flag, every block
// leaves at its next wait and the solve reports FVGB_ERR_CUDA.
#pragma once

constexpr int kResMaxBlocks = 160;       // 5 partials per polling lane
// Most dynamic shared memory of a resident block.  A launch asks only for what its
// largest block needs: what is left stays L1, and a poll of 128 lines through an L1
// of a few KB takes 2,700 clocks instead of 1,400.
constexpr int kResSmem = 220 * 1024;

struct alignas(128) LLLine {
    LLWord w;  // an FP64 partial; an FP32 one takes w.w0 alone
};
struct ResMail {
    LLLine part[2][3][kResMaxBlocks];  // [epoch parity][dot product][block]
};
// Two parities suffice: a block publishes epoch e after it has every block's
// partial of e - 1, and a block publishes that after it is done with epoch e - 2.

// v, or +0 for a zero of either sign: the sum 0.0 + v
__device__ __forceinline__ double plus_zero(double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return __longlong_as_double((u << 1) == 0 ? 0ll : (long long)u);
}

__device__ __forceinline__ bool ll_get(const LLLine* p, unsigned epoch, double* v) { return ll_load(&p->w, epoch, v); }
__device__ __forceinline__ bool ll_get(const LLLine* p, unsigned epoch, float* v) { return ll_load(&p->w.w0, epoch, v); }

// One warp: the final tree over every block's partial, in all lanes.
// With at most 256 blocks a tree thread holds one partial, so lane l adds
// partials l, l+32, ... and the butterfly finishes, exactly final_tree.
template <class V = double>
__device__ __forceinline__ bool res_collect(GridBar* gb, const LLLine* part, unsigned epoch, int nblk, double* out) {
    constexpr int NS = kResMaxBlocks / 32;
    const int lane = threadIdx.x & 31;
    double v[NS];
    bool have[NS], good = true;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        v[s] = 0.0;
        have[s] = lane + 32 * s >= nblk;
    }
#pragma unroll 1
    for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            V t;
            if (!have[s] && ll_get(&part[lane + 32 * s], epoch, &t)) {
                v[s] = plus_zero((double)t);
                have[s] = true;
            }
            all = all && have[s];
        }
        if (__all_sync(0xffffffffu, all)) break;
        if (__any_sync(0xffffffffu, ll_give_up(gb, spins))) {
            good = false;
            break;
        }
    }
    double s = v[0];
#pragma unroll
    for (int k = 1; k < NS; ++k)
        if (32 * k < nblk) s = s + v[k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
    *out = s;
    return good;
}

// One warp: the block's partial from its 256 thread partials (block_tree)
template <class V>
__device__ __forceinline__ V res_block_tree(const V* sm) {
    const int lane = threadIdx.x & 31;
    V s = sm[lane];
#pragma unroll
    for (int k = 1; k < kT / 32; ++k) s = s + sm[lane + 32 * k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// Slots and halo entries of the largest block of a system, by which every block lays its
// part out; zh: with room for the halo's z.
struct ResSize {
    int len, nh;
    bool zh;
};

// The block's part of the system in shared memory (V: double, or float for the
// FP32 inner solve).
template <class V>
struct ResMatrix {
    V* sp;                 // [rows + size.nh] own directions, then the halo's
    V* sval;               // [size.len]
    V* zh;                 // [size.nh] the halo's z, fetched while a reduction is under way (null: no room)
    int* hcol;             // [size.nh] column of every halo entry
    unsigned short* scol;  // [size.len] index into sp
    int rows, nh, pos0;
    bool fits;             // else nothing of it may be used
};

// bytes of that part: value size v, with or without the staged z (with FP32 values
// it starts with one FP64 residual per row)
__host__ __device__ inline size_t res_bytes(int v, int rows, int len, int nh, bool zh) {
    return (v == 4 ? 8 * (size_t)rows : 0) + (size_t)v * ((size_t)rows + nh + len + (zh ? nh : 0)) + 4 * (size_t)nh +
           2 * (size_t)len;
}

// Slots and halo entries of the largest block of `rows` rows, from the pattern on the
// host: the rows' columns, or the boxes of a mesh built on the device.
inline ResSize res_count(const fvgb_mesh* m, int rows) {
    ResSize z{0, 0, false};
    const int64_t n = m->v.n;
    if (!m->h_boxes.empty()) {
        for (int64_t r0 = 0; r0 < n; r0 += rows) {
            const int64_t r1 = r0 + rows;
            int64_t nh = 0;
            for (const HostBox& b : m->h_boxes) {
                const int64_t cells = (int64_t)b.nx * b.ny * b.nz, a0 = r0 - b.cell0, a1 = r1 - b.cell0;
                if (a1 <= 0 || a0 >= cells) continue;
                int64_t s = 1;  // the neighbour's distance
                for (int64_t d : {b.nx, b.ny, b.nz}) {
                    // cells below c that have an upper neighbour
                    const auto below = [&](int64_t c) {
                        c = std::min(std::max<int64_t>(c, 0), cells);
                        return c / (s * d) * (s * (d - 1)) + std::min(c % (s * d), s * (d - 1));
                    };
                    // pairs (c, c + s) with only c, or only c + s, in the block
                    nh += below(a1) - below(std::max(a0, a1 - s));
                    nh += below(std::min(a0, a1 - s)) - below(a0 - s);
                    s *= d;
                }
            }
            z.len = std::max(z.len, (int)(std::min((int64_t)rows, n - r0) * m->m_width));
            z.nh = (int)std::max<int64_t>(z.nh, nh);
        }
        return z;
    }
    const std::vector<int32_t>&ro = m->h_row_offs, &col = m->h_col;
    for (int64_t r0 = 0; r0 < n; r0 += rows) {
        const int64_t r1 = std::min(n, r0 + rows);
        int64_t len = 0, nh = 0;
        for (int64_t s = r0; s < r1; s += 32) {
            int w = 0;
            for (int64_t i = s; i < std::min(r1, s + 32); ++i) {
                const int b = ro[(size_t)i], e = ro[(size_t)i + 1];
                w = std::max(w, e - b);
                for (int k = b; k < e && col[(size_t)k] < r0; ++k) ++nh;  // ascending columns
                for (int k = e; k > b && col[(size_t)k - 1] >= r0 + rows; --k) ++nh;
            }
            len += 32 * w;
            // slots of the lanes past the last row name row 0 (where columns are stored)
            if (r0 > 0 && s + 32 > n && !m->v.m_off) nh += (s + 32 - n) * w;
        }
        z.len = (int)std::max<int64_t>(z.len, len);
        z.nh = (int)std::max<int64_t>(z.nh, nh);
    }
    return z;
}

inline ResSize res_size(const fvgb_mesh* m, int rows) {
    ResSize z = res_count(m, rows);
    z.nh = (z.nh + 3) & ~3;  // the values start on a 16-byte boundary
    return z;
}

// Lays the block's part out and fills the columns; the values are the caller's.
template <class V>
__device__ __forceinline__ ResMatrix<V> res_load(const MeshView& m, unsigned char* dyn, int row0, int rows,
                                                 const ResSize& size, int* counter) {
    const int T = threadIdx.x, lane = T & 31, wid = T >> 5, nw = (int)blockDim.x >> 5;
    const int ns = (m.n + 31) >> 5, s0 = min(ns, row0 >> 5), s1 = min(ns, s0 + rows / 32);
    ResMatrix<V> M;
    M.rows = rows;
    M.pos0 = __ldg(&m.m_ptr[s0]);
    M.sp = (V*)(dyn + (sizeof(V) == 4 ? 8 * rows : 0));
    M.sval = M.sp + rows + size.nh;
    M.zh = size.zh ? M.sval + size.len : nullptr;
    M.hcol = (int*)(M.sval + size.len + (size.zh ? size.nh : 0));
    M.scol = (unsigned short*)(M.hcol + size.nh);
    M.fits = __ldg(&m.m_ptr[s1]) - M.pos0 <= size.len;
    if (T == 0) *counter = 0;
    __syncthreads();
    // a slice's columns are fetched while the one before is laid out
    int next[8], w0 = 0, b0 = 0;
    const auto fetch = [&](int s) {
        if (s >= s1) return;
        b0 = __ldg(&m.m_ptr[s]);
        w0 = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5;
        slot_cols(m, b0 + lane, w0, s * 32 + lane, next);
    };
    int s = M.fits ? s0 + wid : s1;
    fetch(s);
#pragma unroll 1
    for (; s < s1; s += nw) {
        const int w = w0, at = b0 + lane;
        int col[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) col[k] = next[k];
        fetch(s + nw);
        const auto place = [&](int k, int c) {
            const int d = c - row0;
            const bool halo = (unsigned)d >= (unsigned)rows;
            const unsigned ball = __ballot_sync(0xffffffffu, halo);
            int base = 0;
            if (ball) {
                const int lead = __ffs(ball) - 1;
                if (lane == lead) base = atomicAdd(counter, __popc(ball));
                base = __shfl_sync(0xffffffffu, base, lead);
            }
            int idx = d;
            if (halo) {
                const int h = base + __popc(ball & ((1u << lane) - 1));
                if (h < size.nh) M.hcol[h] = c;
                idx = rows + h;
            }
            M.scol[at + 32 * k - M.pos0] = (unsigned short)idx;
        };
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k < w) place(k, col[k]);
#pragma unroll 1
        for (int k = 8; k < w; ++k) place(k, slot_col(m, at + 32 * k, s * 32 + lane));
    }
    __syncthreads();
    M.nh = *counter;
    M.fits = M.fits && M.nh <= size.nh;
    return M;
}

// put(h, z) of every halo entry h = first, first + step, ..., as its z of `epoch` arrives;
// four loads in flight (60^3 cells, whose halo has no room to be staged: 18.8 -> 16.0 us an
// iteration against one at a time).
template <class V, class W, class F>
__device__ __forceinline__ bool res_halo_get(GridBar* gb, const ResMatrix<V>& M, const W* z, unsigned epoch, int first,
                                             int step, F put) {
#pragma unroll 1
    for (int h0 = first; h0 < M.nh; h0 += 4 * step) {
        bool have[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) have[u] = h0 + u * step >= M.nh;
#pragma unroll 1
        for (unsigned spins = 0;; ++spins) {
            bool all = true;
            V v[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                ok[u] = false;
                if (!have[u]) ok[u] = ll_load(z + M.hcol[h0 + u * step], epoch, &v[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (ok[u]) {
                    put(h0 + u * step, v[u]);
                    have[u] = true;
                }
                all = all && have[u];
            }
            if (all) break;
            if (ll_give_up(gb, spins)) return false;
        }
    }
    return true;
}

// The halo's z of `epoch` into M.zh, by threads T0 <= T < kT.
template <class V, class W>
__device__ __forceinline__ bool res_halo(GridBar* gb, const ResMatrix<V>& M, const W* z, unsigned epoch, int T0) {
    return res_halo_get(gb, M, z, epoch, (int)threadIdx.x - T0, kT - T0, [&](int h, V v) { M.zh[h] = v; });
}

__device__ __forceinline__ double res_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float res_fma(float a, float b, float c) { return fmaf(a, b, c); }

// The halo's new direction, z (restart) or z + beta p, in M.sp (all threads).
template <class V, class W>
__device__ __forceinline__ bool res_halo_dir(GridBar* gb, const ResMatrix<V>& M, const W* z, unsigned epoch,
                                             bool restart, V beta) {
    if (!M.zh) return res_halo_get(gb, M, z, epoch, (int)threadIdx.x, kT, [&](int h, V v) {  // no room to stage it
        V* p = M.sp + M.rows + h;
        *p = restart ? v : res_fma(beta, *p, v);
    });
#pragma unroll 1
    for (int h = threadIdx.x; h < M.nh; h += kT) {
        V* p = M.sp + M.rows + h;
        *p = restart ? M.zh[h] : res_fma(beta, *p, M.zh[h]);
    }
    return true;
}

// The matrix rows of one thread: slot bases (in the block's arrays) and widths of
// its R slices, one per j.
template <int R>
struct ResRows {
    int base[R], w[R], kmin, kmax;
    __device__ __forceinline__ ResRows(const MeshView& m, int first_row, int pos0) {
        kmin = INT_MAX;
        kmax = 0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int s = (first_row >> 5) + j;
            base[j] = w[j] = 0;
            if (s * 32 < m.n) {
                const int b0 = __ldg(&m.m_ptr[s]);
                base[j] = b0 - pos0 + (threadIdx.x & 31);
                w[j] = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5;
            }
            kmin = min(kmin, w[j]);
            kmax = max(kmax, w[j]);
        }
    }
    // q[j] = sum over the row's slots of value * f(own[j], x[column]): fma chains from
    // +0 in slot order, the R rows interleaved.  A branch per row would serialise the
    // dependent shared-memory loads, so the slots all R rows have go without one.
    template <class V, class F>
    __device__ __forceinline__ void product(const ResMatrix<V>& M, V* q, F f, const V* own) const {
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = (V)0;
#pragma unroll 1
        for (int k = 0; k < kmin; ++k) {
            int c[R];
            V a[R], x[R];
#pragma unroll
            for (int j = 0; j < R; ++j) c[j] = M.scol[base[j] + 32 * k];
#pragma unroll
            for (int j = 0; j < R; ++j) a[j] = M.sval[base[j] + 32 * k];
#pragma unroll
            for (int j = 0; j < R; ++j) x[j] = M.sp[c[j]];
#pragma unroll
            for (int j = 0; j < R; ++j) q[j] = res_fma(a[j], f(own[j], x[j]), q[j]);
        }
#pragma unroll 1
        for (int k = kmin; k < kmax; ++k) {
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (k < w[j])
                    q[j] = res_fma(M.sval[base[j] + 32 * k], f(own[j], M.sp[M.scol[base[j] + 32 * k]]), q[j]);
        }
    }
};

// A block whose part is larger than the host counted ends the solve: every block leaves at
// its next wait.
__device__ __forceinline__ void res_refuse(const Layout& L, GridBar* gb) {
    if (threadIdx.x != 0) return;
    atomicExch(&gb->abort, 1);
    if (blockIdx.x == 0) L.cases[0].status = FVGB_ERR_CUDA;
}

struct ResShared {
    double value, res0, res;
    int code, status, iter, bad, counter;
};

// FP64 Jacobi-CG of one case on its blocks (one per SM); mail and z are zero at
// launch.  512 x 512 cavity pressure (262,144 rows, 128 blocks, 3,050 iterations):
// 12.5 us per iteration against 20.1 for k_pcg_persistent (three grid barriers,
// every vector through L2); of its 25,600 clocks 12,500 are DFMA issue, 7,500 the
// two hops and 4,500 the block and final trees and the scalars' divisions (64
// clocks per dependent FP64 instruction).  1,600 rows: 7.9 us against 15.2.
//
// Before the first iteration (50 us at 60^3 cells, of which 33 are the grid-barrier
// kernel's too): columns fetched a slice ahead, the matrix copied asynchronously beside
// them, the first residual from the block's own part.  A load at a time these took 74 us,
// more than a warm-started solve of seven iterations gains.
template <int R>
__global__ void __launch_bounds__(kT, 1)
    k_pcg_resident(Layout L, MeshView m, const double* __restrict__ val, const double* __restrict__ b, LLWord* z,
                   ResMail* mail, GridBar* gb, ResSize size) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double sma[kT], smb[kT];
    __shared__ ResShared sh;
    constexpr int ROWS = kT * R;
    const int n = m.n, T = threadIdx.x, lane = T & 31, wid = T >> 5, nblk = (int)gridDim.x, blk = (int)blockIdx.x;
    const int row0 = blk * ROWS;
    const int loc0 = wid * (32 * R) + lane;  // this thread's rows: loc0 + 32 j
    const SolverParams prm = L.bs->prm;
    double* x = prm.x;
    if (T == 0) sh.bad = 0;
    const ResMatrix<double> M = res_load<double>(m, dyn, row0, ROWS, size, &sh.counter);
    if (!M.fits) return res_refuse(L, gb);
    {  // the block's slots, 16 bytes at a time
        const int len = min(size.len, __ldg(&m.m_ptr[min((n + 31) >> 5, (row0 + ROWS) >> 5)]) - M.pos0);
        const unsigned at = (unsigned)__cvta_generic_to_shared(M.sval);
        for (int k = 2 * T; k < len; k += 2 * kT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + 8u * k), "l"(val + M.pos0 + k) : "memory");
    }
    double xr[R], rv[R], pr[R], di[R], zr[R];
    ResRows<R> W(m, row0 + wid * (32 * R), M.pos0);
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j;
        xr[j] = i < n ? x[i] : 0.0;
        rv[j] = i < n ? __ldg(&b[i]) : 0.0;
        di[j] = i < n ? __ldg(&val[__ldg(&m.diag_pos[i])]) : 0.0;
        M.sp[loc0 + 32 * j] = xr[j];
    }
#pragma unroll 4
    for (int h = T; h < M.nh; h += kT) M.sp[ROWS + h] = __ldcg(&x[M.hcol[h]]);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    W.product(M, zr, [](double, double xk) { return xk; }, xr);  // b - A x, the chains of the graph's row sums
#pragma unroll
    for (int j = 0; j < R; ++j) {
        rv[j] = row0 + loc0 + 32 * j < n ? rv[j] - zr[j] : 0.0;
        pr[j] = 0.0;
    }
    // (cold code stays in rolled loops: unrolled over the rows the kernel was 97 KB, and its
    // iteration has to stay in the instruction cache)
#pragma unroll 1
    for (int j = 0; j < R; ++j) {  // 1 / diagonal, one division's code
        double d = 1.0;
#pragma unroll
        for (int u = 0; u < R; ++u) d = u == j ? di[u] : d;
        d = 1.0 / d;
#pragma unroll
        for (int u = 0; u < R; ++u) di[u] = u == j && row0 + loc0 + 32 * u < n ? d : di[u];
    }
    unsigned epoch = 0;
    double rz = 0.0, tol = 0.0, res0 = 0.0, res = 0.0;  // warp 0: rz; warp 1: the others
    int iter = 0, status = FVGB_OK;
    double alpha = 0.0;
    bool first = true;
    for (;;) {
        // z = dinv r, r.z, r.r; every other product on the integer pipes (512 x 512
        // cavity: 78.6 -> 77.4 ms; all of them there, 78.7)
        ++epoch;
        double arz = 0.0, arr = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int i = row0 + loc0 + 32 * j;
            zr[j] = j & 1 ? __fma_rn(di[j], rv[j], m.k_nzero) : imul(di[j], rv[j]);
            if (i < n) ll_store(z + i, zr[j], epoch);
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            if (row0 + loc0 + 32 * j < n) {
                arz = fma(rv[j], zr[j], arz);
                arr = fma(rv[j], rv[j], arr);
            }
        }
        sma[T] = arz;
        smb[T] = arr;
        __syncthreads();
        LLLine(*part)[kResMaxBlocks] = mail->part[epoch & 1u];
        if (wid < 2) {
            const double v = res_block_tree(wid == 0 ? sma : smb);
            if (lane == 0) ll_store(&part[wid][blk].w, v, epoch);
        }
        // x += alpha p off the reduction's path: the warps that share a scheduler
        // with a tree warp wait until it has published (their DFMAs would double
        // the tree's 12 dependent additions)
        if (wid < 2) asm volatile("bar.arrive %0, 64;" ::"r"(1 + wid) : "memory");
        else if (wid == 4 || wid == 5) asm volatile("bar.sync %0, 64;" ::"r"(wid - 3) : "memory");
        if (!first) {
#pragma unroll
            for (int j = 0; j < R; ++j) xr[j] = fma(alpha, pr[j], xr[j]);
        }
        if (wid < 2) {
            double v;
            const bool good = res_collect(gb, part[wid], epoch, nblk, &v);
            if (wid == 0) {
                const double beta = v / rz;
                rz = v;
                if (lane == 0) sh.value = beta;
            } else {
                res = sqrt(v);
                int d = 0;
                if (first) {
                    res0 = res;
                    tol = prm.rel_tol * tol_base(&L.cases[0], res);
                    if (prm.abs_tol > tol) tol = prm.abs_tol;
                    d = !(res > tol) || res == 0.0;
                    if (!isfinite(res)) {
                        d = 1;
                        status = FVGB_ERR_BREAKDOWN;
                    } else if (!d && prm.max_iter <= 0) {
                        d = 1;
                        status = FVGB_ERR_NOT_CONVERGED;
                    }
                } else {
                    ++iter;
                    if (!isfinite(res)) {
                        status = FVGB_ERR_BREAKDOWN;
                        d = 1;
                    } else if (!(res > tol)) {
                        d = 1;
                    } else if (iter >= prm.max_iter) {
                        status = FVGB_ERR_NOT_CONVERGED;
                        d = 1;
                    }
                }
                if (lane == 0) sh.code = d;
            }
            if (!good && lane == 0) sh.bad = 1;
        } else if (M.zh) {
            if (!res_halo(gb, M, z, epoch, 64)) sh.bad = 1;
        }
        __syncthreads();
        if (sh.code || sh.bad) break;
        // p = z + beta p: the halo's copies, then the own rows
        const double beta = sh.value;
        if (!res_halo_dir(gb, M, z, epoch, first, beta)) sh.bad = 1;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            pr[j] = first ? zr[j] : fma(beta, pr[j], zr[j]);
            M.sp[loc0 + 32 * j] = pr[j];
        }
        __syncthreads();
        // q = A p: fma chains in slot order, R rows interleaved; p.q
        double q[R];
        W.product(M, q, [](double, double xk) { return xk; }, pr);
        double apq = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (row0 + loc0 + 32 * j < n) apq = fma(pr[j], q[j], apq);
        sma[T] = apq;
        ++epoch;
        __syncthreads();
        if (wid == 0) {
            part = mail->part[epoch & 1u];
            const double v = res_block_tree(sma);
            if (lane == 0) ll_store(&part[2][blk].w, v, epoch);
            double pq;
            const bool good = res_collect(gb, part[2], epoch, nblk, &pq);
            const double a = rz / pq;
            if (lane == 0) {
                sh.value = a;
                if (pq == 0.0 || !isfinite(a)) sh.code = 2;
                if (!good) sh.bad = 1;
            }
        }
        __syncthreads();
        if (sh.code || sh.bad) break;
        alpha = sh.value;
#pragma unroll
        for (int j = 0; j < R; ++j) rv[j] = fma(-alpha, q[j], rv[j]);
        first = false;
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j;
        if (i < n) x[i] = xr[j];
    }
    if (blk == 0 && wid == 1 && lane == 0) {
        CaseState* cs = &L.cases[0];
        cs->res0 = res0;
        cs->res = res;
        cs->iter = iter;
        cs->status = sh.bad ? FVGB_ERR_CUDA : (sh.code == 2 ? FVGB_ERR_BREAKDOWN : status);
    }
}

struct IrResShared {
    double v[3];       // collected sums of a residual
    double nsig, isig;
    float fa, fbeta;
    int restart, done, inner, brk, bad, counter;
    unsigned int flags;
};

// Mixed-precision solve of one case on its blocks: the algorithm, arithmetic and
// decisions of k_ir_persistent with the layout of k_pcg_resident.  The FP32 matrix
// copy, the vectors of the inner CG and x are resident; a refinement step writes x
// for the other blocks behind a fence and reads the FP64 matrix through L2.  An
// inner iteration is two hops (2 x 1.4 us with 128 blocks on both dies), two final
// trees and divisions in FP64 (2 x 0.7 us) and 1.5 us of FP32 work on shared
// memory.  512 x 512 cavity step: 128 -> 66 ms against k_ir_persistent.
template <int R>
__global__ void __launch_bounds__(kT, 1)
    k_ir_resident(Layout L, MeshView m, const double* __restrict__ val, const double* __restrict__ b, float* a32,
                  float* ev, float* dinv, unsigned long long* z, ResMail* mail, GridBar* gb, ResSize size) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double sma[kT], smb[kT];
    __shared__ float smf[kT];
    __shared__ IrResShared sh;
    constexpr int ROWS = kT * R;
    const int n = m.n, T = threadIdx.x, lane = T & 31, wid = T >> 5, nblk = (int)gridDim.x, blk = (int)blockIdx.x;
    const int row0 = blk * ROWS;
    const int loc0 = wid * (32 * R) + lane;  // this thread's rows: loc0 + 32 j
    const SolverParams prm = L.bs->prm;
    double* x = prm.x;
    if (T == 0) {
        sh.bad = 0;
        sh.flags = 0u;
    }
    double* stage = (double*)dyn;  // [rows] FP64 residuals
    const ResMatrix<float> M = res_load<float>(m, dyn, row0, ROWS, size, &sh.counter);
    if (!M.fits) return res_refuse(L, gb);
    // prepare: dinv, a32, ev (formed, or those of the unchanged matrix), sign flags, |D^-1/2 (b - A x0)|
    unsigned int f = 0u;
    double asr = 0.0;
    ResRows<R> W(m, row0 + wid * (32 * R), M.pos0);
    if (!prm.convert) {  // the block's slots, 16 bytes at a time
        const int len = min(size.len, __ldg(&m.m_ptr[min((n + 31) >> 5, (row0 + ROWS) >> 5)]) - M.pos0);
        const unsigned at = (unsigned)__cvta_generic_to_shared(M.sval);
        for (int k = 4 * T; k < len; k += 4 * kT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + 4u * k), "l"(a32 + M.pos0 + k) : "memory");
    }
#pragma unroll 1
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j, s = i >> 5;
        if (s * 32 >= n || !prm.convert) break;
        const int b0 = __ldg(&m.m_ptr[s]), wj = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5;
        float* sv = M.sval + (b0 - M.pos0);
        if (i >= n) {
#pragma unroll 1
            for (int k = 0; k < wj; ++k) sv[lane + 32 * k] = 0.0f;
            continue;
        }
        const double d = __ldg(&val[__ldg(&m.diag_pos[i])]);
        dinv[i] = (float)(1.0 / d);
        const double sg = d < 0.0 ? -1.0 : 1.0;
        double e = 0.0;
#pragma unroll 1
        for (int k0 = 0; k0 < wj; k0 += 8) {
            const int at = b0 + lane + 32 * k0, left = wj - k0;
            int code[8];
            double av[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                code[k] = k < left ? __ldg(&m.m_code[at + 32 * k]) : FVGB_PAD;
                av[k] = k < left ? __ldg(&val[at + 32 * k]) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (k >= left) break;
                float a = 0.0f;
                if (code[k] != FVGB_PAD) {
                    e = e + av[k];
                    if (code[k] != -1) a = (float)(sg * av[k]);
                }
                a32[at + 32 * k] = a;
                sv[lane + 32 * (k0 + k)] = a;
            }
        }
        ev[i] = (float)(sg * e);
    }
#pragma unroll 4
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j;
        if (i >= n) continue;
        const double d = __ldg(&val[__ldg(&m.diag_pos[i])]);
        f |= d > 0.0 ? 1u : (d < 0.0 ? 2u : 4u);
        const double r = __ldg(&b[i]) - spmv_row_cg(m, val, x, i);
        stage[loc0 + 32 * j] = r;
        asr = fma(r * (double)fabsf(dinv[i]), r, asr);
    }
    double xr[R];
    float yv[R], rh[R], pr[R], zr[R], di[R], ei[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j;
        xr[j] = i < n ? x[i] : 0.0;
        di[j] = i < n ? dinv[i] : 0.0f;
        ei[j] = i < n ? ev[i] : 0.0f;
        yv[j] = rh[j] = pr[j] = zr[j] = 0.0f;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (f) atomicOr(&sh.flags, f);
    sma[T] = asr;
    unsigned epoch = 1;
    // refinement state: warp 0
    double sres = 0.0, sig = 1.0, isig = 1.0, res0 = 0.0, res = 0.0, tol = 0.0, rho = 0.0, rho_prev = 0.0, itol = 0.0;
    int total = 0, outer = 0, inner_it = 0, status = FVGB_OK;
    unsigned int flags = 0u;
    __syncthreads();
    if (wid < 2) {
        // the sign flags of all blocks travel as an exact sum of 1, 2^10 and 2^20 per block
        double v;
        if (wid == 0) {
            v = res_block_tree(sma);
        } else {
            const unsigned int g = sh.flags;
            v = (double)((g & 1u) | ((g & 2u) << 9) | ((g & 4u) << 18));
        }
        if (lane == 0) ll_store(&mail->part[epoch & 1u][wid][blk].w, v, epoch);
        double t;
        const bool good = res_collect(gb, mail->part[epoch & 1u][wid], epoch, nblk, &t);
        if (lane == 0) {
            sh.v[wid] = t;
            if (!good) sh.bad = 1;
        }
    }
    __syncthreads();
    bool done = sh.bad != 0, first = true;
    if (wid == 0) {
        sres = sqrt(sh.v[0]);
        const unsigned int g = (unsigned)sh.v[1];
        flags = ((g & 1023u) ? 1u : 0u) | ((g >> 10) & 1023u ? 2u : 0u) | ((g >> 20) ? 4u : 0u);
    }
    while (!done) {
        if (!first) {
            // x += y / sig, published behind a fence
            const double is = sh.isig;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int i = row0 + loc0 + 32 * j;
                xr[j] = fma((double)yv[j], is, xr[j]);
                if (i < n) x[i] = xr[j];
            }
            ++epoch;
            __syncthreads();
            if (wid == 0) {
                if (lane == 0) {
                    __threadfence();
                    ll_store(&mail->part[epoch & 1u][0][blk].w, 0.0, epoch);
                }
                double t;
                const bool good = res_collect(gb, mail->part[epoch & 1u][0], epoch, nblk, &t);
                __threadfence();
                if (!good && lane == 0) sh.bad = 1;
            }
        }
        double nsig = 1.0, nisig = 1.0;
        if (wid == 0) {
            residual_scale(sres, &nsig, &nisig);
            if (lane == 0) sh.nsig = nsig;
        }
        __syncthreads();
        if (sh.bad) break;
        // residual: r = b - A x (FP64), rh = sign*(float)(sig r), y = 0, z = |dinv| rh
        const double ns = sh.nsig;
        ++epoch;
        if (!first) {
#pragma unroll 4
            for (int j = 0; j < R; ++j) {
                const int i = row0 + loc0 + 32 * j;
                if (i < n) stage[loc0 + 32 * j] = __ldg(&b[i]) - spmv_row_cg(m, val, x, i);
            }
        }
        double arr = 0.0;
        asr = 0.0;
        float arho = 0.0f;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int i = row0 + loc0 + 32 * j;
            if (i >= n) continue;
            const double r = stage[loc0 + 32 * j];
            float t = (float)(r * ns);
            if (di[j] < 0.0f) t = -t;
            rh[j] = t;
            yv[j] = 0.0f;
            zr[j] = fabsf(di[j]) * t;
            ll_store(z + i, zr[j], epoch);
            arr = fma(r, r, arr);
            asr = fma(r * (double)fabsf(di[j]), r, asr);
            arho = fmaf(t, zr[j], arho);
        }
        sma[T] = arr;
        smb[T] = asr;
        smf[T] = arho;
        __syncthreads();
        if (wid < 3) {
            LLLine* part = mail->part[epoch & 1u][wid];
            const double v = wid == 0 ? res_block_tree(sma) : (wid == 1 ? res_block_tree(smb) : (double)res_block_tree(smf));
            if (lane == 0) ll_store(&part[blk].w, v, epoch);
            double t;
            const bool good = res_collect(gb, part, epoch, nblk, &t);
            if (lane == 0) {
                sh.v[wid] = t;
                if (!good) sh.bad = 1;
            }
        } else if (M.zh) {
            if (!res_halo(gb, M, z, epoch, 96)) sh.bad = 1;
        }
        __syncthreads();
        if (sh.bad) break;
        if (wid == 0) {
            const double rr = sh.v[0], sr2 = sh.v[1], nrho = sh.v[2];
            bool d = false;
            res = sqrt(rr);
            if (!first) outer += 1;
            if (first) {
                res0 = res;
                tol = prm.rel_tol * tol_base(&L.cases[0], res);
                if (prm.abs_tol > tol) tol = prm.abs_tol;
                if ((flags & 4u) || flags == 3u) {
                    status = FVGB_ERR_UNSUPPORTED;
                    d = true;
                }
            }
            if (!d) {
                if (!isfinite(res)) {
                    status = FVGB_ERR_BREAKDOWN;
                    d = true;
                } else if (!(res > tol) || res == 0.0) {
                    d = true;
                } else if (outer >= prm.max_outer || total >= prm.max_iter) {
                    status = FVGB_ERR_NOT_CONVERGED;
                    d = true;
                }
            }
            const double g = nsig * isig;
            const double rho_rec = rho * g * g;
            const bool restart = first || inner_it == 0 || nrho > 4.0 * rho_rec;
            const float frel = restart ? -1.0f : (float)((nrho / rho_prev) * (sig * nisig));
            sig = nsig;
            isig = nisig;
            sres = sqrt(sr2);
            rho = nrho;
            const double dr = prm.inner_rel_tol * prm.inner_rel_tol;
            const double dt = (tol / res) * (tol / res);
            itol = rho * (dr > dt ? dr : dt);
            inner_it = 0;
            if (lane == 0) {
                sh.inner = !d && rho > itol && prm.inner_max_iter > 0 && total < prm.max_iter;
                sh.done = d;
                sh.isig = isig;
                sh.restart = frel < 0.0f;
                sh.fbeta = frel;
            }
        }
        __syncthreads();
        first = false;
        done = sh.done;
        if (done) break;
        while (sh.inner) {
            // p = z + beta p: the halo's copies, then the own rows
            const bool restart = sh.restart;
            const float fb = sh.fbeta;
            if (!res_halo_dir(gb, M, z, epoch, restart, fb)) sh.bad = 1;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                pr[j] = restart ? zr[j] : fmaf(fb, pr[j], zr[j]);
                M.sp[loc0 + 32 * j] = pr[j];
            }
            __syncthreads();
            // q = A p in the difference form, R rows interleaved; p.q
            float q[R];
            W.product(M, q, [](float xi, float xk) { return xk - xi; }, pr);
            float acc = 0.0f;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                q[j] = fmaf(ei[j], pr[j], q[j]);
                if (row0 + loc0 + 32 * j < n) acc = fmaf(pr[j], q[j], acc);
            }
            smf[T] = acc;
            ++epoch;
            __syncthreads();
            if (wid == 0) {
                LLLine* part = mail->part[epoch & 1u][2];
                const float v = res_block_tree(smf);
                if (lane == 0) ll_store(&part[blk].w.w0, v, epoch);
                double pq;
                const bool good = res_collect<float>(gb, part, epoch, nblk, &pq);
                const double alpha = rho / pq;
                const bool brk = pq == 0.0 || !isfinite(alpha);
                if (brk && inner_it == 0) status = FVGB_ERR_BREAKDOWN;
                if (lane == 0) {
                    sh.fa = (float)alpha;
                    sh.brk = brk;
                    if (brk) sh.inner = 0;
                    if (brk && inner_it == 0) sh.done = 1;
                    if (!good) sh.bad = 1;
                }
            }
            __syncthreads();
            if (sh.brk || sh.bad) break;
            const float fa = sh.fa;
            // y += alpha p, rh -= alpha q, z = |dinv| rh, rh.z
            ++epoch;
            acc = 0.0f;
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const int i = row0 + loc0 + 32 * j;
                yv[j] = fmaf(fa, pr[j], yv[j]);
                rh[j] = fmaf(-fa, q[j], rh[j]);
                zr[j] = fabsf(di[j]) * rh[j];
                if (i < n) {
                    ll_store(z + i, zr[j], epoch);
                    acc = fmaf(rh[j], zr[j], acc);
                }
            }
            smf[T] = acc;
            __syncthreads();
            if (wid == 0) {
                LLLine* part = mail->part[epoch & 1u][2];
                const float v = res_block_tree(smf);
                if (lane == 0) ll_store(&part[blk].w.w0, v, epoch);
                double rhon;
                const bool good = res_collect<float>(gb, part, epoch, nblk, &rhon);
                const float fbeta = (float)(rhon / rho);
                rho_prev = rho;
                rho = rhon;
                inner_it += 1;
                total += 1;
                if (lane == 0) {
                    sh.inner = rhon > itol && inner_it < prm.inner_max_iter && total < prm.max_iter;
                    sh.restart = 0;
                    sh.fbeta = fbeta;
                    if (!good) sh.bad = 1;
                }
            } else if (M.zh) {
                if (!res_halo(gb, M, z, epoch, 32)) sh.bad = 1;
            }
            __syncthreads();
            if (sh.bad) break;
        }
        if (sh.bad) break;
        done = sh.done;
    }
    if (blk == 0 && T == 0) {
        CaseState* cs = &L.cases[0];
        cs->res0 = res0;
        cs->res = res;
        cs->iter = 0;
        cs->total = total;
        cs->outer = outer;
        cs->status = sh.bad ? FVGB_ERR_CUDA : status;
    }
}

// ---------------------------------------------------------- one cluster (small systems)
// FP64 CG of at most kClMaxUnits tree warps (4-row tree) in ONE thread-block cluster:
// the reduction tree's warps ("units", 128 consecutive rows) are spread over its
// blocks, a thread holding one row, so the rows of a virtual block share out over up
// to 8 SMs' FP64 pipes.  Everything that crosses blocks is a word with its epoch
// (ll.cuh) in distributed shared memory: a unit sends its 32 lane partials to the
// block that forms its virtual block's tree, that block sends the result to all, and
// the halo's z is polled where its owner keeps it.  What bounds an iteration is its
// ~55 dependent FP64 instructions (64 clocks each) in the chains, trees and
// divisions, then four hops of 700 clocks.  40 x 40 cavity pressure (1,600 rows, 13
// of 16 blocks): 4.4 us an iteration against 7.5 for k_pcg_resident's two blocks.
// Measured slower: every unit's partials to every block (one hop less, but a
// warp's 16 stores of 512 bytes take 450 clocks; 4.9 us with the trees in every
// block), cluster barriers in place of the words (5.2), partials read by the trees
// across the cluster (5.1).
constexpr int kClRows = 128;     // rows of a unit: 32 lanes x 4 rows
constexpr int kClMaxUnits = 32;  // two per block of a 16-block cluster
constexpr int kClMaxVb = kClMaxUnits / 8;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// address of this block's shared object p in block `rank`
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cl_store(unsigned at, double v, unsigned epoch) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.cluster.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(at), "l"(e | (u & 0xffffffffull)),
                 "l"(e | (u >> 32))
                 : "memory");
}
__device__ __forceinline__ bool cl_load(unsigned at, unsigned epoch, double* v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.cluster.shared::cluster.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(at) : "memory");
    return ll_take(a, b, epoch, v);
}
// the same of this block's own words (through the cluster's window each poll would
// take the network's latency)
__device__ __forceinline__ bool cl_load_own(unsigned at, unsigned epoch, double* v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(at) : "memory");
    return ll_take(a, b, epoch, v);
}
constexpr unsigned kClSpins = 1u << 23;  // bound of every wait: seconds

struct ClShared {
    LLWord part[2][2][8][32];            // [epoch parity][dot product][unit of the virtual block formed here][lane]
    LLWord val[2][2][kClMaxVb];          // [epoch parity][dot product][virtual block]
    LLWord z[2 * kClRows];               // this block's z, polled by the others
    double a[2 * kClRows], b[2 * kClRows];  // staged operands of the dot products
    double value;
    int code, bad, counter;
};

// One warp: lane partials of the block's unit u as the tree thread sums them, sent to
// `at` (the slot of lane 0).
__device__ __forceinline__ void cl_chain(unsigned at, unsigned epoch, const double* a, const double* b, int u,
                                         int row0, int n) {
    const int lane = threadIdx.x & 31;
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int l = u * kClRows + 32 * j + lane;
        if (row0 + l < n) acc = fma(a[l], b[l], acc);
    }
    cl_store(at + 16u * lane, acc, epoch);
}

// One warp: a virtual block's partial from its k1 units' lanes as they arrive at
// `part` (block_tree), sent to `val`, lane r's address in block r.
__device__ __forceinline__ bool cl_tree(unsigned part, unsigned epoch, int k1, unsigned val, int ncta) {
    const int lane = threadIdx.x & 31;
    const unsigned at = part + 16u * lane;
    double t[8];
    bool good = true;
#pragma unroll 1
    for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < 8; ++k) all = (cl_load_own(at + 512u * k, epoch, &t[k]) || k >= k1) && all;
        if (__all_sync(0xffffffffu, all)) break;
        if (spins > kClSpins) {
            good = false;
            break;
        }
    }
    double s = t[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) {
        if (k >= k1) break;
        s = s + t[k];
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
    if (lane < ncta) cl_store(val, s, epoch);
    return good;
}

// One warp: final_tree over the virtual blocks' partials as they arrive (the
// butterfly's other terms are +0).
__device__ __forceinline__ bool cl_final(const LLWord* val, unsigned epoch, int nvb, double* out) {
    const unsigned at = (unsigned)__cvta_generic_to_shared(val);
    double v[kClMaxVb];
    bool good = true;
#pragma unroll 1
    for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int k = 0; k < kClMaxVb; ++k) all = (cl_load_own(at + 16u * k, epoch, &v[k]) || k >= nvb) && all;
        if (__all_sync(0xffffffffu, all)) break;
        if (spins > kClSpins) {
            good = false;
            break;
        }
    }
    static_assert(kClMaxVb == 4, "two butterfly steps");
#pragma unroll
    for (int k = 0; k < kClMaxVb; ++k) v[k] = k < nvb ? plus_zero(v[k]) : 0.0;
    if (nvb > 2) {
        v[0] = v[0] + v[2];
        v[1] = v[1] + v[3];
    }
    *out = nvb > 1 ? v[0] + v[1] : v[0];
    return good;
}

__global__ void __launch_bounds__(2 * kClRows, 1)
    k_pcg_cluster(Layout L, MeshView m, const double* __restrict__ val, const double* __restrict__ b, int units) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ ClShared sh;
    const int n = m.n, T = threadIdx.x, lane = T & 31, wid = T >> 5, nw = (int)blockDim.x >> 5;
    const int rows = (int)blockDim.x, lg = rows == kClRows ? 7 : 8;  // one unit per block, or two
    // The cluster's size is a power of two, `ncta` of its blocks hold rows.  The others
    // take no part: a word is written again two epochs on, when every block that sends
    // partials has read it, and a block without rows sends none, so nothing would make
    // the others wait for it.
    const int rank = (int)blockIdx.x, ncta = (units * kClRows + rows - 1) / rows;
    const int row0 = rank * rows, i = row0 + T, nvb = (units + 7) / 8;
    if (rank >= ncta) {
        cluster_arrive();
        cluster_wait();
        cluster_arrive();
        cluster_wait();
        return;
    }
    const SolverParams prm = L.bs->prm;
    double* x = prm.x;
    for (int k = T; k < (int)(offsetof(ClShared, a) / sizeof(LLWord)); k += rows) ((LLWord*)&sh)[k] = LLWord{0ull, 0ull};
    if (T == 0) sh.code = sh.bad = 0;
    const ResMatrix<double> M = res_load<double>(m, dyn, row0, rows, ResSize{rows * 8, rows * 8, false}, &sh.counter);
    // this thread's row, its slots (at most 8) in registers
    double xr = 0.0, rv = 0.0, pr = 0.0, di = 0.0, v8[8];
    int c8[8], w = 0, b0 = 0;
    if ((i & ~31) < n) {
        b0 = __ldg(&m.m_ptr[i >> 5]);
        w = (__ldg(&m.m_ptr[(i >> 5) + 1]) - b0) >> 5;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        v8[k] = k < w ? __ldg(&val[b0 + lane + 32 * k]) : 0.0;
        c8[k] = k < w ? M.scol[b0 - M.pos0 + lane + 32 * k] : 0;
    }
    if (i < n) {
        xr = x[i];
        di = 1.0 / __ldg(&val[__ldg(&m.diag_pos[i])]);
        rv = __ldg(&b[i]) - spmv_row_cg(m, val, x, i);
    }
    // where this thread's first halo entry lives
    unsigned hat = 0u;
    if (T < M.nh) hat = cluster_addr(&sh.z[M.hcol[T] & (rows - 1)], M.hcol[T] >> lg);
    double rz = 0.0, tol = 0.0, res0 = 0.0, res = 0.0, alpha = 0.0;  // warp 0: rz; the last warp: the residual's
    int iter = 0, status = FVGB_OK;
    // chain warps: a unit's two dot products on warps of different schedulers; the tree
    // of dot product d of virtual block v is formed by warp 2 of block d * nvb + v (or
    // that modulo the cluster's size: at most 8 trees, and never two on one warp when
    // the cluster has as many blocks)
    const int cu = wid >> 2, first_w = 4 * cu + (cu & 1) * 2;  // of the unit this warp belongs to
    const int unit = rank * (rows / kClRows) + cu;
    const int chain = unit < units ? wid - first_w : -1;  // the dot product this warp's chain forms (0, 1), if any
    int tree2 = -1, tree1 = -1;                           // the trees this warp forms: dot * nvb + virtual block
    for (int q = rank, k = 2; q < 2 * nvb; q += ncta, ++k)
        if (wid == k % nw) {
            tree2 = q;
            if (q < nvb) tree1 = q;
        }
    const int tdot = tree2 >= nvb, tv = tree2 - tdot * nvb, tk = min(units - 8 * tv, 8);
    // addresses with epoch parity 0; parity 1 is one array further
    constexpr unsigned kPartPar = sizeof(LLWord) * 2 * 8 * 32, kValPar = sizeof(LLWord) * 2 * kClMaxVb;
    unsigned to2 = 0u, to1 = 0u, tval = 0u;
    if (chain == 0 || chain == 1)
        to2 = cluster_addr(sh.part[0][chain][unit & 7], (chain * nvb + (unit >> 3)) % ncta);
    if (chain == 0) to1 = to2;
    if (tree2 >= 0 && lane < ncta) tval = cluster_addr(&sh.val[0][tdot][tv], lane);
    const unsigned tpart = (unsigned)__cvta_generic_to_shared(sh.part[0][tdot]);
    bool first = true;
    unsigned epoch = 0;
    cluster_arrive();  // every block has cleared its words
    cluster_wait();
    for (;;) {
        // z = dinv r, r.z, r.r
        ++epoch;
        const unsigned par = epoch & 1u;
        const double z = __fma_rn(di, rv, m.k_nzero);
        sh.a[T] = z;
        sh.b[T] = rv;
        cl_store((unsigned)__cvta_generic_to_shared(&sh.z[T]), z, epoch);
        __syncthreads();
        if (chain == 0 || chain == 1) cl_chain(to2 + par * kPartPar, epoch, sh.b, chain ? sh.b : sh.a, cu, row0, n);
        if (!first) xr = fma(alpha, pr, xr);  // off the reduction's path
        bool good = true;
        if (tree2 >= 0) good = cl_tree(tpart + par * kPartPar, epoch, tk, tval + par * kValPar, ncta);
        double rr = 0.0;
        if (wid == 0) {
            double t;
            good = cl_final(sh.val[par][0], epoch, nvb, &t) && good;
            const double beta = t / rz;
            rz = t;
            if (lane == 0) sh.value = beta;
        } else if (wid == nw - 1) {
            good = cl_final(sh.val[par][1], epoch, nvb, &rr) && good;
        }
        // the halo's z
        double hz = 0.0;
        if (T < M.nh) {
            unsigned spins = 0;
            while (!cl_load(hat, epoch, &hz))
                if (++spins > kClSpins) {
                    good = false;
                    break;
                }
        }
        if (!good) sh.bad = 1;
        __syncthreads();
        // p = z + beta p: the halo's copies and the own row
        const double beta = sh.value;
        if (T < M.nh) M.sp[rows + T] = first ? hz : fma(beta, M.sp[rows + T], hz);
#pragma unroll 1
        for (int h = T + rows; h < M.nh; h += rows) {
            const unsigned at = cluster_addr(&sh.z[M.hcol[h] & (rows - 1)], M.hcol[h] >> lg);
            unsigned spins = 0;
            while (!cl_load(at, epoch, &hz))
                if (++spins > kClSpins) {
                    sh.bad = 1;
                    break;
                }
            M.sp[rows + h] = first ? hz : fma(beta, M.sp[rows + h], hz);
        }
        pr = first ? z : fma(beta, pr, z);
        M.sp[T] = pr;
        __syncthreads();
        // q = A p, p.q
        double q = 0.0, x8[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x8[k] = M.sp[c8[k]];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k >= w) break;  // w is the warp's
            q = fma(v8[k], x8[k], q);
        }
        sh.b[T] = q;
        ++epoch;
        const unsigned par1 = epoch & 1u;
        __syncthreads();
        if (chain == 0) cl_chain(to1 + par1 * kPartPar, epoch, M.sp, sh.b, cu, row0, n);
        if (tree1 >= 0 && !cl_tree(tpart + par1 * kPartPar, epoch, tk, tval + par1 * kValPar, ncta)) sh.bad = 1;
        // the stopping test of the residual, while the partials are under way: x is
        // already the iterate it belongs to, and nothing of this product is used
        // when it ends the solve
        if (wid == nw - 1) {
            res = sqrt(rr);
            int d = 0;
            if (first) {
                res0 = res;
                tol = prm.rel_tol * tol_base(&L.cases[0], res);
                if (prm.abs_tol > tol) tol = prm.abs_tol;
                d = !(res > tol) || res == 0.0;
                if (!isfinite(res)) {
                    d = 1;
                    status = FVGB_ERR_BREAKDOWN;
                } else if (!d && prm.max_iter <= 0) {
                    d = 1;
                    status = FVGB_ERR_NOT_CONVERGED;
                }
            } else {
                ++iter;
                if (!isfinite(res)) {
                    status = FVGB_ERR_BREAKDOWN;
                    d = 1;
                } else if (!(res > tol)) {
                    d = 1;
                } else if (iter >= prm.max_iter) {
                    status = FVGB_ERR_NOT_CONVERGED;
                    d = 1;
                }
            }
            if (d && lane == 0) sh.code = 1;
        }
        int brk = 0;
        if (wid == 0) {
            double pq;
            if (!cl_final(sh.val[par1][0], epoch, nvb, &pq)) sh.bad = 1;
            const double a = rz / pq;
            const long long ua = __double_as_longlong(a), up = __double_as_longlong(pq);
            brk = (up << 1) == 0 || (ua & 0x7ff0000000000000ll) == 0x7ff0000000000000ll;
            if (lane == 0) sh.value = a;
        }
        brk = __syncthreads_or(brk);
        if (sh.code || sh.bad) break;
        if (brk) {
            status = FVGB_ERR_BREAKDOWN;
            break;
        }
        alpha = sh.value;
        rv = fma(-alpha, q, rv);
        first = false;
    }
    if (i < n) x[i] = xr;
    if (rank == 0 && wid == nw - 1 && lane == 0) {
        CaseState* cs = &L.cases[0];
        cs->res0 = res0;
        cs->res = res;
        cs->iter = iter;
        cs->status = sh.bad ? FVGB_ERR_CUDA : status;
    }
    cluster_arrive();  // no block leaves while another may read its shared memory
    cluster_wait();
}
