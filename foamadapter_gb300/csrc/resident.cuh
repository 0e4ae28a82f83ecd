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
// Everything that crosses blocks carries its epoch beside the data: a value
// travels as two 8-byte words, each half the value and the 32-bit epoch, so a
// reader polls the data itself and no fence, counter or second read is needed
// (a fence behind the vector stores costs 930 clocks here, one such hop 570).
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
constexpr int kResSmem = 220 * 1024;     // dynamic shared memory of a resident block

struct alignas(16) LLWord {  // one published value
    unsigned long long w0, w1;  // epoch << 32 | low half, epoch << 32 | high half
};
struct alignas(128) LLLine {
    LLWord w;
};
struct ResMail {
    LLLine part[2][3][kResMaxBlocks];  // [epoch parity][dot product][block]
};
// Two parities suffice: a block publishes epoch e after it has every block's
// partial of e - 1, and a block publishes that after it is done with epoch e - 2.

__device__ __forceinline__ void ll_store(LLWord* p, double v, unsigned epoch) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(e | (u & 0xffffffffull)),
                 "l"(e | (u >> 32))
                 : "memory");
}
__device__ __forceinline__ bool ll_load(const LLWord* p, unsigned epoch, double* v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    *v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (unsigned)(a >> 32) == epoch && (unsigned)(b >> 32) == epoch;
}

// Bound of every wait: true when it has run out, here or in another block.
__device__ __forceinline__ bool res_give_up(GridBar* gb, unsigned spins) {
    if ((spins & 63u) != 63u) return false;
    int ab;
    asm volatile("ld.relaxed.gpu.s32 %0, [%1];" : "=r"(ab) : "l"(&gb->abort) : "memory");
    if (ab) return true;
    if (spins < (1u << 23)) return false;  // seconds
    atomicExch(&gb->abort, 1);
    return true;
}

// v, or +0 for a zero of either sign: the sum 0.0 + v
__device__ __forceinline__ double plus_zero(double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return __longlong_as_double((u << 1) == 0 ? 0ll : (long long)u);
}

// One warp: the final tree over every block's partial, in all lanes.
// With at most 256 blocks a tree thread holds one partial, so lane l adds
// partials l, l+32, ... and the butterfly finishes, exactly final_tree.
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
    for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            double t;
            if (!have[s] && ll_load(&part[lane + 32 * s].w, epoch, &t)) {
                v[s] = plus_zero(t);
                have[s] = true;
            }
            all = all && have[s];
        }
        if (__all_sync(0xffffffffu, all)) break;
        if (__any_sync(0xffffffffu, res_give_up(gb, spins))) {
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
__device__ __forceinline__ double res_block_tree(const double* sm) {
    const int lane = threadIdx.x & 31;
    double s = sm[lane];
#pragma unroll
    for (int k = 1; k < kT / 32; ++k) s = s + sm[lane + 32 * k];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// The block's part of the system in shared memory.
struct ResMatrix {
    double* sp;            // [rows + nh] own directions, then the halo's
    double* sval;          // [len]
    double* zh;            // [nh] the halo's z, fetched while a reduction is under way (null: no room)
    int* hcol;             // [nh] column of every halo entry
    unsigned short* scol;  // [len] index into sp
    int nh, pos0;
};

__host__ __device__ inline size_t res_bytes(int rows, int len, int nh, bool zh) {
    return 8 * (size_t)(rows + nh) + 8 * (size_t)len + (zh ? 8 * (size_t)nh : 0) + 4 * (size_t)nh + 2 * (size_t)len;
}

// Slots and halo entries of block row0's rows (all threads; counter: shared).
template <int R>
__device__ __forceinline__ void res_count(const MeshView& m, int row0, int* counter, int* len, int* nh) {
    constexpr int ROWS = kT * R;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int s0 = row0 >> 5, s1 = min((m.n + 31) >> 5, s0 + ROWS / 32);
    *len = __ldg(&m.m_ptr[s1]) - __ldg(&m.m_ptr[s0]);
    if (threadIdx.x == 0) *counter = 0;
    __syncthreads();
    for (int s = s0 + wid; s < s1; s += kT / 32) {
        const int b0 = __ldg(&m.m_ptr[s]), w = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5, i = s * 32 + lane;
        int c = 0;
        for (int k = 0; k < w; ++k)
            c += (unsigned)(slot_col(m, b0 + k * 32 + lane, i) - row0) >= (unsigned)ROWS;
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(counter, c);
    }
    __syncthreads();
    *nh = *counter;
    __syncthreads();
}

// Whether every block's part fits in shared memory: the largest need, in bytes.
template <int R>
__global__ void __launch_bounds__(kT) k_res_need(MeshView m, unsigned int* need) {
    __shared__ int counter;
    int len, nh;
    res_count<R>(m, (int)blockIdx.x * (kT * R), &counter, &len, &nh);
    if (threadIdx.x == 0) {
        const size_t b = kT * R + nh > 65536 ? ~(size_t)0 : res_bytes(kT * R, len, nh, false);
        atomicMax(need, b > 0xffffffffull ? 0xffffffffu : (unsigned)b);
    }
}

template <int R>
__device__ __forceinline__ ResMatrix res_load(const MeshView& m, const double* __restrict__ val, unsigned char* dyn,
                                              int row0, int* counter) {
    constexpr int ROWS = kT * R;
    const int T = threadIdx.x, lane = T & 31, wid = T >> 5;
    const int s0 = row0 >> 5, s1 = min((m.n + 31) >> 5, s0 + ROWS / 32);
    ResMatrix M;
    int len;
    res_count<R>(m, row0, counter, &len, &M.nh);
    M.pos0 = __ldg(&m.m_ptr[s0]);
    const bool zh = res_bytes(ROWS, len, M.nh, true) <= (size_t)kResSmem;
    M.sp = (double*)dyn;
    M.sval = M.sp + ROWS + M.nh;
    M.zh = zh ? M.sval + len : nullptr;
    M.hcol = (int*)(M.sval + len + (zh ? M.nh : 0));
    M.scol = (unsigned short*)(M.hcol + M.nh);
    if (T == 0) *counter = 0;
    __syncthreads();
    for (int s = s0 + wid; s < s1; s += kT / 32) {
        const int b0 = __ldg(&m.m_ptr[s]), w = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5, i = s * 32 + lane;
        for (int k = 0; k < w; ++k) {
            const int pos = b0 + k * 32 + lane;
            const int c = slot_col(m, pos, i), d = c - row0;
            const bool halo = (unsigned)d >= (unsigned)ROWS;
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
                M.hcol[h] = c;
                idx = ROWS + h;
            }
            M.scol[pos - M.pos0] = (unsigned short)idx;
            M.sval[pos - M.pos0] = __ldg(&val[pos]);
        }
    }
    __syncthreads();
    return M;
}

// The halo's z of `epoch` into dst, by threads T0 <= T < kT; four loads in flight each.
__device__ __forceinline__ bool res_halo(GridBar* gb, const ResMatrix& M, const LLWord* z, unsigned epoch, int T0,
                                         double* dst) {
    for (int h0 = (int)threadIdx.x - T0; h0 < M.nh; h0 += 4 * (kT - T0)) {
        bool have[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) have[u] = h0 + u * (kT - T0) >= M.nh;
        for (unsigned spins = 0;; ++spins) {
            bool all = true;
            double v[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                ok[u] = false;
                if (!have[u]) ok[u] = ll_load(z + M.hcol[h0 + u * (kT - T0)], epoch, &v[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (ok[u]) {
                    dst[h0 + u * (kT - T0)] = v[u];
                    have[u] = true;
                }
                all = all && have[u];
            }
            if (all) break;
            if (res_give_up(gb, spins)) return false;
        }
    }
    return true;
}

struct ResShared {
    double value, res0, res;
    int code, status, iter, bad, counter;
};

// FP64 Jacobi-CG of one case on its blocks (one per SM); mail and z are zero at
// launch.  512 x 512 cavity pressure (262,144 rows, 128 blocks, 3,050 iterations):
// 13.1 us per iteration against 20.1 for k_pcg_persistent (three grid barriers,
// every vector through L2); of its 25,600 clocks 12,500 are DFMA issue, 7,500 the
// two hops and 4,500 the block and final trees and the scalars' divisions (64
// clocks per dependent FP64 instruction).  1,600 rows: 7.9 us against 15.2.
template <int R>
__global__ void __launch_bounds__(kT, 1)
    k_pcg_resident(Layout L, MeshView m, const double* __restrict__ val, const double* __restrict__ b, LLWord* z,
                   ResMail* mail, GridBar* gb) {
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
    const ResMatrix M = res_load<R>(m, val, dyn, row0, &sh.counter);
    double xr[R], rv[R], pr[R], di[R], zr[R];
    int base[R], w[R];
    int wmax = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        const int i = row0 + loc0 + 32 * j, s = (row0 >> 5) + wid * R + j;
        base[j] = w[j] = 0;
        if (s * 32 < n) {
            const int b0 = __ldg(&m.m_ptr[s]);
            base[j] = b0 - M.pos0 + lane;
            w[j] = (__ldg(&m.m_ptr[s + 1]) - b0) >> 5;
        }
        wmax = max(wmax, w[j]);
        xr[j] = rv[j] = pr[j] = di[j] = 0.0;
        if (i < n) {
            xr[j] = x[i];
            di[j] = 1.0 / __ldg(&val[__ldg(&m.diag_pos[i])]);
            rv[j] = __ldg(&b[i]) - spmv_row_cg(m, val, x, i);
        }
    }
    unsigned epoch = 0;
    double rz = 0.0, tol = 0.0, res0 = 0.0, res = 0.0;  // warp 0: rz; warp 1: the others
    int iter = 0, status = FVGB_OK;
    double alpha = 0.0;
    bool first = true;
    for (;;) {
        // z = dinv r, r.z, r.r
        ++epoch;
        double arz = 0.0, arr = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int i = row0 + loc0 + 32 * j;
            zr[j] = __fma_rn(di[j], rv[j], m.k_nzero);
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
            if (!res_halo(gb, M, z, epoch, 64, M.zh)) sh.bad = 1;
        }
        __syncthreads();
        if (sh.code || sh.bad) break;
        // p = z + beta p: the halo's copies, then the own rows
        const double beta = sh.value;
        if (!M.zh) {  // no room to stage it
            for (int h = T; h < M.nh; h += kT) {
                double v;
                unsigned spins = 0;
                while (!ll_load(z + M.hcol[h], epoch, &v))
                    if (res_give_up(gb, spins++)) {
                        sh.bad = 1;
                        break;
                    }
                M.sp[ROWS + h] = first ? v : fma(beta, M.sp[ROWS + h], v);
            }
        } else {
            for (int h = T; h < M.nh; h += kT)
                M.sp[ROWS + h] = first ? M.zh[h] : fma(beta, M.sp[ROWS + h], M.zh[h]);
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            pr[j] = first ? zr[j] : fma(beta, pr[j], zr[j]);
            M.sp[loc0 + 32 * j] = pr[j];
        }
        __syncthreads();
        // q = A p: fma chains in slot order, R rows interleaved; p.q
        double q[R];
#pragma unroll
        for (int j = 0; j < R; ++j) q[j] = 0.0;
        for (int k = 0; k < wmax; ++k) {
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (k < w[j]) q[j] = fma(M.sval[base[j] + 32 * k], M.sp[M.scol[base[j] + 32 * k]], q[j]);
        }
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
