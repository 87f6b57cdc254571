// mg_persist.cuh -- a multigrid solve, or the coarse part of a V-cycle, as one
// kernel.
//
// What bounds a solve of these sizes is not memory but the number of
// dependent steps: a V(2,2) cycle over six levels is 38 sweeps and
// transfers, nearly all of them 2-4 us long as kernels although their data
// (a 1025 x 1025 level is 4 MB in FP32) stays in L2 and would stream in
// 0.1-2 us.  Here one kernel walks through them and its blocks meet at a
// barrier between two steps instead of at a kernel boundary:
//
//   * levels whose vectors fit the shared memory of one block (the "tail")
//     are worked by block 0 alone, between two barriers;
//   * a problem that is nothing but tail runs in one block (kSyncBlock);
//   * up to kClusterRows rows, in one cluster of 16 blocks, whose barrier is
//     a hardware one (kSyncCluster);
//   * above, in one block per SM, launched cooperatively (all blocks
//     resident), with a counter barrier in global memory (kSyncGrid).
//
// The refinement loop runs inside the kernel, so a solve ends with the cycle
// that met the residual bound and no gated launch follows it.
//
// Every row is computed by the operations of k_level_op, k_restrict,
// k_prolong_add, k_dense_mv and k_residual64 in their order, and the norms
// are summed in the order of k_residual64's fixed grid, so iterates and
// residuals are those of the launched kernels bit for bit.
//
// Waits: a cluster barrier cannot spin; a grid barrier polls a counter at
// most `polls` times, then records a stall and no later barrier of the block
// waits.  The host reports a stall as PSUM_ERR_INTERNAL.
#pragma once

#include "mg_kernels.cuh"

namespace psum_b200 {

// Threads per block: a 27-point FP64 row keeps twice the registers in flight.
// All stencil shapes share a kernel, so it has 80 (FP32) and 128 (FP64)
// registers a thread and spills 140-200 and 644 bytes at its largest shape.
template <class T>
constexpr int kPersistThreads = sizeof(T) == 4 ? 768 : 512;
constexpr int kPersistLevels = 12;
constexpr int kClusterBlocks = 16;
constexpr int kNormVBlocks = 444;           // the fixed grid of the norms: 444 blocks of 256 rows per stride
constexpr int kNormVWarps = kNormVBlocks * 8;
constexpr int kBarrierPolls = 1 << 22;      // seconds; a step takes microseconds
constexpr int kDenseTailRows = 128;         // coarse systems up to this size are solved by the tail's block

enum PersistSync { kSyncBlock = 0, kSyncCluster = 1, kSyncGrid = 2 };
enum PersistMode { kPersistMixed = 0, kPersistFp64 = 1, kPersistCycle = 2 };

// A level's operator for the kernel: the stencil, and its exception rows as
// coefficients on the stencil's taps where their columns allow it.
template <class T>
struct PersistStencil {
    StencilDev<T> s;
    int shape;              // tap count when the taps are one of the usual shapes, else 0
    const uint2* word;      // per 32 rows: exception mask, exceptions before
    const T* dense;         // per exception: shape coefficients
    const uint8_t* csr;     // per exception: 1 = only the column list gives its order (null: none)
};

// One axis factor of the transfers at one index: up to three fine indices
// with weights, up to two coarse ones (absent terms: weight zero).
template <class T>
struct alignas(sizeof(T) * 2) RestrictEntry {
    int f[3];
    T w[3];
};
template <class T>
struct alignas(sizeof(T) * 2) ProlongEntry {
    int c[2];
    T w[2];
};

template <class T>
struct PersistLevel {
    PersistStencil<T> A;
    XferDev<T> X;        // to the next coarser level
    const RestrictEntry<T>* rest[3];
    const ProlongEntry<T>* prol[3];
    int dim;             // axes of more than one node
    T* x[2];
    T* b;
    const T* dinv;
    int n;
    int smem;            // tail levels: element offset of (x0, x1, b) in shared memory
};

template <class T>
struct PersistArgs {
    PersistLevel<T> lv[kPersistLevels];
    PersistStencil<double> a0;    // unscaled fine operator (FP64 residual)
    const double* dinv0;
    const double* coarse_inv;
    double* b;                    // right-hand side (sources are applied in place)
    double* x;                    // initial guess and solution
    const unsigned long long* add_idx;
    const double* add_val;
    const unsigned long long* rep_idx;
    const double* rep_val;
    long long n_add, n_rep;
    double* partials;             // kNormVWarps warp sums
    MGState* st;
    unsigned* counter;            // grid barrier
    int polls;                    // its wait limit
    double tol;
    int mode;
    int first, tail, last;        // first level of this kernel, first tail level, coarsest level
    int dense_all;                // the coarse system is solved by every block
    int pre, post, max_cycles, interval;
    int null_space;
    int gated;                    // kPersistCycle: skip when the solve is done
};

// Barrier over the kernel's blocks; every thread calls it.
template <int SYNC, class T>
struct Barrier {
    const PersistArgs<T>& p;
    unsigned& target;       // thread 0's, in shared memory: every thread would hold a register for it
    bool& broken;

    __device__ __forceinline__ void operator()() {
        if constexpr (SYNC == kSyncBlock) {
            __syncthreads();
        } else if constexpr (SYNC == kSyncCluster) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
            if (threadIdx.x == 0) {
                const unsigned want = target += gridDim.x;
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.counter) : "memory");
                if (!broken) {
                    unsigned v = 0;
                    int it = 0;
                    for (;;) {
                        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.counter) : "memory");
                        if ((int)(v - want) >= 0) break;
                        if (++it >= p.polls) {
                            broken = true;
                            record_stall(&p.st->stall);
                            break;
                        }
                    }
                }
            }
            __syncthreads();
        }
    }
};

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// What a sweep reads as its iterate: the level's vector, or (scale = w on the
// right-hand side) the first sweep from zero, w b, rounded before it is used
// as when it is stored.  One code path for both: x * 1 is x.
template <class T>
struct Iterate {
    const T* x;
    T scale;
    __device__ __forceinline__ T get(int q) const { return mul_rn(scale, x[q]); }
};

// Taps of the usual stencil shapes, in the order the host's stencil
// extraction sorts them: 3 (1-D), 5 and 9 (2-D), 7 and 27 (3-D).
__host__ __device__ constexpr int shape_tap(int ns, int t, int axis) {
    return ns == 3 ? (axis == 0 ? t - 1 : 0)
         : ns == 5 ? (axis == 0 ? (t == 0 ? -1 : (t == 4 ? 1 : 0)) : (axis == 1 ? (t == 1 ? -1 : (t == 3 ? 1 : 0)) : 0))
         : ns == 9 ? (axis == 0 ? t / 3 - 1 : (axis == 1 ? t % 3 - 1 : 0))
                   : tma_tap_d(ns, t, axis);
}

// (A x)_r of an exception row: coefficients of its own on the shape's taps,
// or a column list where only that gives the order of its terms.
template <class T, int NS>
__device__ __forceinline__ T exception_row(const PersistStencil<T>& P, const Iterate<T>& val, const T (&v)[NS], int q) {
    T s = T(0);
    if (!P.csr || !__ldg(P.csr + q)) {
        const T* c = P.dense + (long long)q * NS;
#pragma unroll
        for (int t = 0; t < NS; ++t) s += __ldg(c + t) * v[t];
        if (s == s) return s;   // else the row may not have a tap whose value is infinite (0 times that is NaN)
        s = T(0);
    }
    const int b = __ldg(P.s.exc_ptr + q), e = __ldg(P.s.exc_ptr + q + 1);
#pragma unroll 1
    for (int t = b; t < e; ++t) s += __ldg(P.s.exc_val + t) * val.get(__ldg(P.s.exc_col + t));
    return s;
}

// Row r's neighbours: three offsets per axis, the wrapped one selected
// instead of branched to, so the rows beside a face (every warp has one on
// the small levels) cost the others nothing.
struct RowOffsets {
    int im, ip, jm, jp, km, kp;
    __device__ __forceinline__ int operator()(int di, int dj, int dk) const {
        return (di < 0 ? im : (di > 0 ? ip : 0)) + (dj < 0 ? jm : (dj > 0 ? jp : 0)) + (dk < 0 ? km : (dk > 0 ? kp : 0));
    }
};
template <int D, class T>
__device__ __forceinline__ RowOffsets row_offsets(const StencilDev<T>& A, int r) {
    int i = r, j = 0, k = 0;
    if (D > 1) {
        i = (int)fastdiv((unsigned)r, A.div12);
        j = r - i * (int)A.div12.d;
        if (D > 2) {
            const int rem = j;
            j = (int)fastdiv((unsigned)rem, A.div2);
            k = rem - j * A.n2;
        }
    }
    const int s1 = D == 3 ? A.n2 : 1, s0 = D == 1 ? 1 : (int)A.div12.d;
    return {i == 0 ? (A.n0 - 1) * s0 : -s0, i == A.n0 - 1 ? (1 - A.n0) * s0 : s0,
            j == 0 ? (A.n1 - 1) * s1 : -s1, j == A.n1 - 1 ? (1 - A.n1) * s1 : s1,
            k == 0 ? A.n2 - 1 : -1,         k == A.n2 - 1 ? 1 - A.n2 : 1};
}

// (A x)_r from a row's values: the stencil, or the row's own coefficients.
template <class T, int NS>
__device__ __forceinline__ T apply_row(const PersistStencil<T>& P, const Iterate<T>& val, const T (&v)[NS], uint2 word, int r) {
    const uint32_t bit = 1u << (r & 31);
    if (word.x & bit) return exception_row<T, NS>(P, val, v, (int)word.y + __popc(word.x & (bit - 1u)));
    T s = T(0);
#pragma unroll
    for (int t = 0; t < NS; ++t) s += P.s.c[t] * v[t];
    return s;
}

template <int NS>
constexpr int kShapeDim = NS == 3 ? 1 : (NS == 5 || NS == 9 ? 2 : 3);

// Rows spread over all blocks' threads: consecutive rows in consecutive
// threads, two in flight per thread.  The level is in L2 and its rows'
// neighbours in L1; what counts is how many loads are under way.
template <class T, int NS, class F>
__device__ __forceinline__ void spread_rows(const PersistStencil<T>& P, const Iterate<T>& val, const T* b, int tid, int nthr,
                                            F&& row) {
    constexpr int U = NS <= 9 ? 2 : 1;
    const int n = (int)P.s.n;
    const bool exc = P.s.any_exc;
    for (int r0 = tid; r0 < n; r0 += U * nthr) {
        T ax[U], xr[U], bv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = min(r0 + u * nthr, n - 1);   // past the end: computed, not stored
            const uint2 word = exc ? __ldg(P.word + (r >> 5)) : make_uint2(0u, 0u);
            const RowOffsets o = row_offsets<kShapeDim<NS>>(P.s, r);
            bv[u] = b[r];
            T v[NS];
#pragma unroll
            for (int t = 0; t < NS; ++t) v[t] = val.get(r + o(shape_tap(NS, t, 0), shape_tap(NS, t, 1), shape_tap(NS, t, 2)));
            ax[u] = apply_row<T, NS>(P, val, v, word, r);
            xr[u] = v[NS / 2];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (r0 + u * nthr < n) row(r0 + u * nthr, xr[u], ax[u], bv[u]);
    }
}

// Rows of a tail level, in shared memory and one block: instructions count,
// not latency.  A thread takes a column of the level (fixed indices on all
// axes but the first) over a strip of planes as long as the level has rows
// per thread: the values of planes i - 1 and i stay in registers and one
// index division serves the strip.  64 x 64 rows in FP64: 2.4 -> 1.7 us a
// sweep; spread over blocks the strip's serial loads make it slower
// (1025 x 1025: 6.3 -> 9.0 us).
template <class T, int NS, class F>
__device__ __forceinline__ void march_rows(const PersistStencil<T>& P, const Iterate<T>& val, const T* b, int tid, int nthr,
                                           F&& row) {
    const StencilDev<T>& A = P.s;
    constexpr int D = kShapeDim<NS>;
    constexpr bool STAR = NS == 3 || NS == 5 || NS == 7;
    constexpr int PT = STAR ? 1 : NS / 3;        // values kept per plane: a star needs its sides in the middle plane only
    const int n0 = A.n0, cols = D == 1 ? 1 : (D == 2 ? A.n1 : A.n1 * A.n2);
    const int R = D == 1 ? 1 : ((int)A.n + nthr - 1) / nthr;
    const int tasks = D == 1 ? n0 : (n0 + R - 1) / R * cols;
    const bool exc = A.any_exc;
    T c[NS];
#pragma unroll
    for (int t = 0; t < NS; ++t) c[t] = A.c[t];
    for (int task = tid; task < tasks; task += nthr) {
        const int strip = D == 1 ? task : (int)fastdiv((unsigned)task, A.div12);
        const int q = task - strip * cols, i0 = strip * R, i1 = min(i0 + R, n0);
        const RowOffsets o = row_offsets<D>(A, i0 * cols + q);   // in-plane offsets hold for the whole column
        auto tap = [&](int t, int p) {
            return val.get(p + o(0, D == 1 ? 0 : shape_tap(NS, t, 1), D < 3 ? 0 : shape_tap(NS, t, 2)));
        };
        auto load_plane = [&](T (&v)[PT], int i) {
            const int p = i * cols + q;
#pragma unroll
            for (int t = 0; t < PT; ++t) v[t] = STAR ? val.get(p) : tap(t, p);
        };
        T wm[PT], w0[PT], wp[PT];
        load_plane(wm, i0 == 0 ? n0 - 1 : i0 - 1);
        load_plane(w0, i0);
        for (int i = i0; i < i1; ++i) {
            const int r = i * cols + q;
            const uint2 word = exc ? __ldg(P.word + (r >> 5)) : make_uint2(0u, 0u);
            const T bv = b[r];
            load_plane(wp, i == n0 - 1 ? 0 : i + 1);
            T v[NS];
#pragma unroll
            for (int t = 0; t < NS; ++t) {
                const int di = shape_tap(NS, t, 0);
                if (!STAR) v[t] = di < 0 ? wm[t % PT] : (di > 0 ? wp[t % PT] : w0[t % PT]);
                else if (di != 0 || t == NS / 2) v[t] = di < 0 ? wm[0] : (di > 0 ? wp[0] : w0[0]);
                else v[t] = tap(t, r);
            }
            T ax = T(0);
            const uint32_t bit = 1u << (r & 31);
            if (word.x & bit) {
                ax = exception_row<T, NS>(P, val, v, (int)word.y + __popc(word.x & (bit - 1u)));
            } else {
#pragma unroll
                for (int t = 0; t < NS; ++t) ax += c[t] * v[t];
            }
            row(r, v[NS / 2], ax, bv);
#pragma unroll
            for (int t = 0; t < PT; ++t) {
                wm[t] = w0[t];
                w0[t] = wp[t];
            }
        }
    }
}

// (A x)_r of any stencil.
template <class T>
__device__ __forceinline__ T any_row(const StencilDev<T>& A, const Iterate<T>& val, int r) {
    const uint32_t word = A.any_exc ? __ldg(A.mask + (r >> 5)) : 0u;
    const int i = (int)fastdiv((unsigned)r, A.div12);
    const int rem = r - i * (int)A.div12.d;
    const int j = (int)fastdiv((unsigned)rem, A.div2);
    const int k = rem - j * A.n2;
    T s = T(0);
    const uint32_t bit = 1u << (r & 31);
    if (word & bit) {
        const int q = (int)__ldg(A.mask_prefix + (r >> 5)) + __popc(word & (bit - 1u));
        const int b = __ldg(A.exc_ptr + q), e = __ldg(A.exc_ptr + q + 1);
#pragma unroll 1
        for (int t = b; t < e; ++t) s += __ldg(A.exc_val + t) * val.get(__ldg(A.exc_col + t));
        return s;
    }
#pragma unroll 1
    for (int t = 0; t < A.ns; ++t) {
        const int ii = wrap_idx(i + A.di[t], A.n0);
        const int jj = wrap_idx(j + A.dj[t], A.n1);
        const int kk = wrap_idx(k + A.dk[t], A.n2);
        s += A.c[t] * val.get((ii * A.n1 + jj) * A.n2 + kk);
    }
    return s;
}

// One sweep (residual = false) or residual over the level's rows.
template <bool TAIL, class T, int NS>
__device__ __forceinline__ void sweep_ns(const PersistStencil<T>& P, const Iterate<T>& val, const T* b, T* __restrict__ out,
                                         bool residual, int tid, int nthr) {
    const T omega = T(2.0 / 3);
    auto row = [&](int r, T xr, T ax, T bv) { out[r] = residual ? bv - ax : xr + omega * (bv - ax); };
    if constexpr (NS == 0) {
        const int n = (int)P.s.n;
        for (int r = tid; r < n; r += nthr) row(r, val.get(r), any_row(P.s, val, r), b[r]);
    } else if constexpr (TAIL) {
        march_rows<T, NS>(P, val, b, tid, nthr, row);
    } else {
        spread_rows<T, NS>(P, val, b, tid, nthr, row);
    }
}

template <bool TAIL, class T>
__device__ __forceinline__ void sweep(const PersistStencil<T>& A, const Iterate<T>& val, const T* b, T* out, bool residual,
                                      int tid, int nthr) {
    if (A.shape == 5) sweep_ns<TAIL, T, 5>(A, val, b, out, residual, tid, nthr);
    else if (A.shape == 7) sweep_ns<TAIL, T, 7>(A, val, b, out, residual, tid, nthr);
    else if (A.shape == 9) sweep_ns<TAIL, T, 9>(A, val, b, out, residual, tid, nthr);
    else if (A.shape == 27) sweep_ns<TAIL, T, 27>(A, val, b, out, residual, tid, nthr);
    else if (A.shape == 3) sweep_ns<TAIL, T, 3>(A, val, b, out, residual, tid, nthr);
    else sweep_ns<TAIL, T, 0>(A, val, b, out, residual, tid, nthr);
}

// Transfers with the axis factors read as whole entries and absent terms as
// zero weights, so that a row's loads do not wait on one another; the terms
// are summed in restrict_value's and prolong_value's order, and a zero term
// changes no sum.
template <class T, int D>
__device__ __forceinline__ T restrict_at(const PersistLevel<T>& V, const T* rf, int c) {
    const XferDev<T>& X = V.X;
    int ci = c, cj = 0, ck = 0;
    if (D > 1) {
        ci = (int)fastdiv((unsigned)c, X.divc12);
        cj = c - ci * X.ax[1].nc * X.ax[2].nc;
        if (D > 2) {
            const int rem = cj;
            cj = (int)fastdiv((unsigned)rem, X.divc2);
            ck = rem - cj * X.ax[2].nc;
        }
    }
    const RestrictEntry<T> ei = V.rest[0][ci];
    const RestrictEntry<T> ej = D > 1 ? V.rest[1][cj] : RestrictEntry<T>{};
    const RestrictEntry<T> ek = D > 2 ? V.rest[2][ck] : RestrictEntry<T>{};
    const int nf1 = X.ax[1].nf, nf2 = X.ax[2].nf;
    T v[D == 1 ? 3 : (D == 2 ? 9 : 27)];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < (D > 1 ? 3 : 1); ++b)
#pragma unroll
            for (int q = 0; q < (D > 2 ? 3 : 1); ++q) {
                const int f = D == 1 ? ei.f[a] : (D == 2 ? ei.f[a] * nf1 + ej.f[b] : (ei.f[a] * nf1 + ej.f[b]) * nf2 + ek.f[q]);
                v[D == 1 ? a : (D == 2 ? a * 3 + b : (a * 3 + b) * 3 + q)] = rf[f];
            }
    T s = T(0);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < (D > 1 ? 3 : 1); ++b)
#pragma unroll
            for (int q = 0; q < (D > 2 ? 3 : 1); ++q) {
                T w = ei.w[a];
                if (D > 1) w = w * ej.w[b];
                if (D > 2) w = w * ek.w[q];
                s += w * v[D == 1 ? a : (D == 2 ? a * 3 + b : (a * 3 + b) * 3 + q)];
            }
    return s;
}

template <class T, int D>
__device__ __forceinline__ T prolong_at(const PersistLevel<T>& V, const T* xc, int f) {
    const XferDev<T>& X = V.X;
    int fi = f, fj = 0, fk = 0;
    if (D > 1) {
        fi = (int)fastdiv((unsigned)f, X.divf12);
        fj = f - fi * X.ax[1].nf * X.ax[2].nf;
        if (D > 2) {
            const int rem = fj;
            fj = (int)fastdiv((unsigned)rem, X.divf2);
            fk = rem - fj * X.ax[2].nf;
        }
    }
    const ProlongEntry<T> ei = V.prol[0][fi];
    const ProlongEntry<T> ej = D > 1 ? V.prol[1][fj] : ProlongEntry<T>{};
    const ProlongEntry<T> ek = D > 2 ? V.prol[2][fk] : ProlongEntry<T>{};
    const int nc1 = X.ax[1].nc, nc2 = X.ax[2].nc;
    T s = T(0);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < (D > 1 ? 2 : 1); ++b)
#pragma unroll
            for (int q = 0; q < (D > 2 ? 2 : 1); ++q) {
                const int c = D == 1 ? ei.c[a] : (D == 2 ? ei.c[a] * nc1 + ej.c[b] : (ei.c[a] * nc1 + ej.c[b]) * nc2 + ek.c[q]);
                T w = ei.w[a];
                if (D > 1) w = w * ej.w[b];
                if (D > 2) w = w * ek.w[q];
                s += w * xc[c];
            }
    return s;
}

template <class T, int D>
__device__ __forceinline__ void restrict_dim(const PersistLevel<T>& V, const T* res, T* __restrict__ bc, const T* dinv,
                                          int nc, int tid, int nthr) {
    for (int c = tid; c < nc; c += nthr) bc[c] = restrict_at<T, D>(V, res, c) * __ldg(dinv + c);
}
template <class T>
__device__ __forceinline__ void restrict_level(const PersistLevel<T>& V, const T* res, T* bc, const T* dinv, int nc,
                                               int tid, int nthr) {
    if (V.dim == 2) restrict_dim<T, 2>(V, res, bc, dinv, nc, tid, nthr);
    else if (V.dim == 3) restrict_dim<T, 3>(V, res, bc, dinv, nc, tid, nthr);
    else restrict_dim<T, 1>(V, res, bc, dinv, nc, tid, nthr);
}

template <class T, int D>
__device__ __forceinline__ void prolong_dim(const PersistLevel<T>& V, const T* e, T* x, bool unwritten, int tid, int nthr) {
    constexpr int U = 2;
    for (int f0 = tid; f0 < V.n; f0 += U * nthr) {
        T v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int f = min(f0 + u * nthr, V.n - 1);
            v[u] = prolong_at<T, D>(V, e, f) + (unwritten ? T(0) : x[f]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (f0 + u * nthr < V.n) x[f0 + u * nthr] = v[u];
    }
}
template <class T>
__device__ __forceinline__ void prolong_level(const PersistLevel<T>& V, const T* e, T* x, bool unwritten, int tid,
                                              int nthr) {
    if (V.dim == 2) prolong_dim<T, 2>(V, e, x, unwritten, tid, nthr);
    else if (V.dim == 3) prolong_dim<T, 3>(V, e, x, unwritten, tid, nthr);
    else prolong_dim<T, 1>(V, e, x, unwritten, tid, nthr);
}

// Where a level's vectors live: the global buffers, or the tail's shared
// memory (x0, x1, b one after another).
template <class T>
struct GlobalLevels {
    static constexpr bool kTail = false;
    const PersistLevel<T>* lv;
    __device__ __forceinline__ T* x(int l, int which) const { return lv[l].x[which]; }
    __device__ __forceinline__ T* b(int l) const { return lv[l].b; }
};
template <class T>
struct SharedLevels {
    static constexpr bool kTail = true;
    const PersistLevel<T>* lv;
    T* base;
    __device__ __forceinline__ T* x(int l, int which) const { return base + lv[l].smem + which * lv[l].n; }
    __device__ __forceinline__ T* b(int l) const { return base + lv[l].smem + 2 * lv[l].n; }
};

// Down the levels [first, last): pre-smoothing, residual, restriction into
// the right-hand side of the next level.  `par` bit l names the current
// buffer of level l; x of `first` starts at zero when zero_first, of the
// others always.  `rhs_out`: where the last restriction writes.
template <class T, class Mem, class Sync>
__device__ __forceinline__ void cycle_down(const PersistArgs<T>& p, const PersistLevel<T>* lv, const Mem& m, Sync& sync, int first, int last,
                                           bool zero_first, T* rhs_out, unsigned& par, int tid, int nthr) {
    const T omega = T(2.0 / 3);
    for (int l = first; l < last; ++l) {
        const PersistLevel<T>& V = lv[l];
        const bool zero = l > first || zero_first;
        const T* b = m.b(l);
        const T* res = b;   // from zero without a sweep the residual is b
        int k = 0;
        if (zero && p.pre >= 2) {
            par &= ~(1u << l);
            sweep<Mem::kTail>(V.A, Iterate<T>{b, omega}, b, m.x(l, 0), false, tid, nthr);   // the first two sweeps
            sync();
            k = 2;
        } else if (zero) {
            par &= ~(1u << l);
            if (p.pre == 1) {
                T* x = m.x(l, 0);
                for (int r = tid; r < V.n; r += nthr) x[r] = omega * b[r];
                sync();
            }
            k = p.pre;
        }
        for (; k < p.pre; ++k) {
            const int c = (par >> l) & 1;
            sweep<Mem::kTail>(V.A, Iterate<T>{m.x(l, c), T(1)}, b, m.x(l, 1 - c), false, tid, nthr);
            par ^= 1u << l;
            sync();
        }
        if (!zero || p.pre > 0) {
            const int c = (par >> l) & 1;
            sweep<Mem::kTail>(V.A, Iterate<T>{m.x(l, c), T(1)}, b, m.x(l, 1 - c), true, tid, nthr);
            res = m.x(l, 1 - c);
            sync();
        }
        restrict_level(V, res, l + 1 < last ? m.b(l + 1) : rhs_out, lv[l + 1].dinv, lv[l + 1].n, tid, nthr);
        sync();
    }
}

// Up the levels [first, last): prolongation-add (from `xc` at the top) and post-smoothing.
template <class T, class Mem, class Sync>
__device__ __forceinline__ void cycle_up(const PersistArgs<T>& p, const PersistLevel<T>* lv, const Mem& m, Sync& sync, int first, int last,
                                         bool zero_first, const T* xc, unsigned& par, int tid, int nthr) {
    for (int l = last - 1; l >= first; --l) {
        const PersistLevel<T>& V = lv[l];
        const bool unwritten = (l > first || zero_first) && p.pre == 0;   // x was never swept: zero
        const T* e = l + 1 < last ? m.x(l + 1, (par >> (l + 1)) & 1) : xc;
        T* x = m.x(l, (par >> l) & 1);
        prolong_level(V, e, x, unwritten, tid, nthr);
        sync();
        const T* b = m.b(l);
        for (int k = 0; k < p.post; ++k) {
            const int c = (par >> l) & 1;
            sweep<Mem::kTail>(V.A, Iterate<T>{m.x(l, c), T(1)}, b, m.x(l, 1 - c), false, tid, nthr);
            par ^= 1u << l;
            sync();
        }
    }
}

// x = Ainv b by the warps [warp, warp + nwarps, ...], dense_row's order.
template <class T>
__device__ __forceinline__ void dense_solve(const double* __restrict__ Ainv, const T* b, T* x, int n, int warp,
                                            int nwarps) {
    const int lane = threadIdx.x & 31;
    for (int row = warp; row < n; row += nwarps) {
        const double* a = Ainv + (long long)row * n;
        double s = 0.0;
#pragma unroll 8
        for (int c = lane; c < n; c += 32) s += __ldg(a + c) * (double)b[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) x[row] = (T)s;
    }
}

// Warp sums of a norm: warp q of the fixed 444 x 8 grid adds the rows that
// warp q % 8 of block q / 8 of k_residual64 / k_norm2 / k_sum adds, in order.
template <bool SQUARE, class F>
__device__ __forceinline__ void norm_partials(double* partials, int n, int warp, int nwarps, F&& value) {
    const int lane = threadIdx.x & 31;
    constexpr int S = kNormVBlocks * 256;
    const int used = min(kNormVWarps, (n + 31) / 32);   // further warps hold no rows: their sums are zero
    auto add = [](double acc, double v) { return SQUARE ? __fma_rn(v, v, acc) : acc + v; };
    if (n <= S) {
        // one row per thread of the fixed grid: four of its warps at a time
        constexpr int U = 4;
        for (int q0 = warp; q0 < used; q0 += U * nwarps) {
            double acc[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = (q0 + u * nwarps) * 32 + lane;
                acc[u] = r < n ? add(0.0, value(r)) : 0.0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (lane == 0 && q0 + u * nwarps < used) partials[q0 + u * nwarps] = acc[u];
        }
        return;
    }
    for (int q = warp; q < used; q += nwarps) {
        double acc = 0.0;
        int r = q * 32 + lane;
        for (; r + S < n; r += 2 * S) {   // two rows in flight, added in order
            const double v0 = value(r), v1 = value(r + S);
            acc = add(acc, v0);
            acc = add(acc, v1);
        }
        if (r < n) acc = add(acc, value(r));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) partials[q] = acc;
    }
}

// Their sum in the order of block_sum and k_check (lane_order) or k_sub_mean
// (shuffle tree); the same in every block.  Contains block barriers.
__device__ __forceinline__ double norm_total(const double* partials, int n, bool tree) {
    __shared__ double vb[kNormVBlocks];
    __shared__ double total;
    const int used = min(kNormVWarps, (n + 31) / 32);
    __syncthreads();
    for (int t = threadIdx.x; t < kNormVBlocks; t += blockDim.x) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += t * 8 + q < used ? partials[t * 8 + q] : 0.0;
        vb[t] = s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = 0.0;
        for (int q = threadIdx.x; q < kNormVBlocks; q += 32) v += vb[q];
        if (tree) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (threadIdx.x == 0) total = v;
        } else {
            __syncwarp();
            vb[threadIdx.x] = v;
            __syncwarp();
            if (threadIdx.x == 0) {
                double s = 0.0;
                for (int q = 0; q < 32; ++q) s += vb[q];
                total = s;
            }
        }
    }
    __syncthreads();
    return total;
}

// (A x)_r of a usual shape, row by row: the fixed order of the norm's rows
// does not follow the columns.
template <int NS>
__device__ __forceinline__ double residual_row(const PersistStencil<double>& P, const double* x, int r) {
    const StencilDev<double>& A = P.s;
    if constexpr (NS == 0) {
        return any_row(A, Iterate<double>{x, 1.0}, r);
    } else {
        const uint2 word = A.any_exc ? __ldg(P.word + (r >> 5)) : make_uint2(0u, 0u);
        const RowOffsets o = row_offsets<kShapeDim<NS>>(A, r);
        const Iterate<double> val{x, 1.0};
        double v[NS];
#pragma unroll
        for (int t = 0; t < NS; ++t) v[t] = x[r + o(shape_tap(NS, t, 0), shape_tap(NS, t, 1), shape_tap(NS, t, 2))];
        return apply_row<double, NS>(P, val, v, word, r);
    }
}

// FP64 residual of the fine operator, optionally bhat = T(dinv * r); the warp
// sums of r^2 go to partials.
template <class T, int NS>
__device__ __forceinline__ void residual64_ns(const PersistArgs<T>& p, const double* x, T* bhat, int warp, int nwarps) {
    norm_partials<true>(p.partials, (int)p.a0.s.n, warp, nwarps, [&](int r) {
        const double bv = p.b[r], dv = bhat ? __ldg(p.dinv0 + r) : 0.0;
        const double res = bv - residual_row<NS>(p.a0, x, r);
        if (bhat) bhat[r] = T(dv * res);
        return res;
    });
}
template <class T>
__device__ __forceinline__ void residual64(const PersistArgs<T>& p, const double* x, T* bhat, int warp, int nwarps) {
    if (p.a0.shape == 5) residual64_ns<T, 5>(p, x, bhat, warp, nwarps);
    else if (p.a0.shape == 7) residual64_ns<T, 7>(p, x, bhat, warp, nwarps);
    else residual64_ns<T, 0>(p, x, bhat, warp, nwarps);
}

// b of the level-by-level solve, or its residual, minus its mean.
template <class Sync>
__device__ __forceinline__ void project(double* v, int n, double* partials, Sync& sync, int tid, int nthr) {
    norm_partials<false>(partials, n, tid >> 5, nthr >> 5, [&](int r) { return v[r]; });
    sync();
    const double m = norm_total(partials, n, true) / (double)n;
    for (int r = tid; r < n; r += nthr) v[r] -= m;
    sync();
}

template <class T, int SYNC>
__global__ void __launch_bounds__(kPersistThreads<T>, 1) k_mg_persist(const __grid_constant__ PersistArgs<T> p) {
    const int NT = blockDim.x, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char persist_smem[];
    __shared__ __align__(16) unsigned char level_smem[sizeof(PersistLevel<T>) * kPersistLevels];
    if (p.mode == kPersistCycle && p.gated && p.st->done) return;
    __shared__ unsigned barrier_target;
    __shared__ bool barrier_broken;
    if (threadIdx.x == 0) {
        barrier_target = 0;
        barrier_broken = false;
    }
    Barrier<SYNC, T> sync{p, barrier_target, barrier_broken};
    Barrier<kSyncBlock, T> bsync{p, barrier_target, barrier_broken};
    const int tid = blockIdx.x * NT + threadIdx.x, nthr = gridDim.x * NT;
    const int warp = tid >> 5, nwarps = nthr >> 5;
    const int n = (int)p.a0.s.n;
    // the levels' descriptions in shared memory: indexed by a run-time level
    // they would be read through the constant cache, which they overflow
    PersistLevel<T>* const lv = reinterpret_cast<PersistLevel<T>*>(level_smem);
    static_assert(sizeof(PersistLevel<T>) % 4 == 0, "copied by words");
    for (int q = threadIdx.x; q < (int)(sizeof(PersistLevel<T>) / 4) * (p.last + 1); q += NT)
        reinterpret_cast<uint32_t*>(level_smem)[q] = reinterpret_cast<const uint32_t*>(p.lv)[q];
    __syncthreads();
    GlobalLevels<T> gm{lv};
    SharedLevels<T> sm{lv, reinterpret_cast<T*>(persist_smem)};
    unsigned par = 0;   // current buffer of every level
    const int L = p.last, tail = p.tail;
    const T* coarse_b = lv[L].b;

    // One V-cycle from level p.first; x of that level starts at zero when
    // `zero`, and its result is the buffer that `par` names.
    auto vcycle = [&](bool zero) __attribute__((always_inline)) {
        T* x_tail = lv[tail].x[0];
        cycle_down(p, lv, gm, sync, p.first, tail, zero, lv[tail].b, par, tid, nthr);
        if (blockIdx.x == 0 && tail < L) {
            // the tail's vectors in shared memory; with first == tail its x comes in too
            const int nt = lv[tail].n;
            const bool z = tail > p.first || zero;
            const T* xg = lv[tail].x[(par >> tail) & 1];
#pragma unroll 4
            for (int r = threadIdx.x; r < nt; r += NT) {
                sm.b(tail)[r] = lv[tail].b[r];
                if (!z) sm.x(tail, 0)[r] = xg[r];
            }
            par &= ~(1u << tail);
            __syncthreads();
            cycle_down(p, lv, sm, bsync, tail, L, z, p.dense_all ? lv[L].b : sm.b(L), par, (int)threadIdx.x, NT);
        }
        if (p.dense_all) {
            if (tail < L) sync();
            dense_solve(p.coarse_inv, coarse_b, lv[L].x[0], lv[L].n, warp, nwarps);
            sync();
        }
        if (blockIdx.x == 0 && tail < L) {
            T* xl = sm.x(L, 0);
            if (p.dense_all) {
                for (int r = threadIdx.x; r < lv[L].n; r += NT) xl[r] = lv[L].x[0][r];
            } else {
                dense_solve(p.coarse_inv, sm.b(L), xl, lv[L].n, (int)threadIdx.x >> 5, NW);
            }
            __syncthreads();
            const bool z = tail > p.first || zero;
            cycle_up(p, lv, sm, bsync, tail, L, z, xl, par, (int)threadIdx.x, NT);
            const T* xs = sm.x(tail, (par >> tail) & 1);
#pragma unroll 4
            for (int r = threadIdx.x; r < lv[tail].n; r += NT) x_tail[r] = xs[r];
        } else if (tail == L && !p.dense_all && blockIdx.x == 0) {
            dense_solve(p.coarse_inv, coarse_b, x_tail, lv[L].n, (int)threadIdx.x >> 5, NW);
        }
        par &= ~(1u << tail);
        sync();
        cycle_up(p, lv, gm, sync, p.first, tail, zero, x_tail, par, tid, nthr);
    };

    const bool cycle_only = p.mode == kPersistCycle;
    // sources, then the norm of the right-hand side
    if (p.n_add > 0) {
        for (long long i = tid; i < p.n_add; i += nthr) atomicAdd(p.b + p.add_idx[i], p.add_val[i]);
        sync();
    }
    if (p.n_rep > 0) {
        for (long long i = tid; i < p.n_rep; i += nthr) p.b[p.rep_idx[i]] = p.rep_val[i];
        sync();
    }
    if (p.null_space) project(p.b, n, p.partials, sync, tid, nthr);
    if (!cycle_only) norm_partials<true>(p.partials, n, warp, nwarps, [&](int r) { return p.b[r]; });
    T* const fx0 = lv[0].x[0];
    double* xfp = p.x;   // the FP64 iterate whose residual is tested
    if constexpr (sizeof(T) == 8) {
        for (int r = tid; r < n && !cycle_only; r += nthr) {
            fx0[r] = p.x[r];
            lv[0].b[r] = T(__ldg(p.dinv0 + r) * p.b[r]);
        }
    }
    double bnorm2 = 0.0;
    if (!cycle_only) {
        sync();
        bnorm2 = norm_total(p.partials, n, false);
        sync();   // partials are rewritten next
    }
    const double bn = bnorm2 > 0 ? bnorm2 : 1.0;
    double first = -1.0, last = -1.0;
    int cycles = 0, refinements = 0, status = 0;
    bool done = false;

    // Convergence test on ||r||^2 = s (check_update).  After the last cycle it
    // only records s, except in a mixed solve with a bound.
    auto check = [&](double s) {
        if (first < 0) first = s;
        last = s;
        if (cycles >= p.max_cycles && !(sizeof(T) == 4 && p.tol > 0)) return;
        if (!(s == s) || s > 1e300 || (first > 0 && s > 1e12 * first)) {
            status = PSUM_ERR_DIVERGED;
            done = true;
        } else if (p.tol > 0 && s <= p.tol * p.tol * bn) {
            done = true;
        }
    };
    bool tested = false;   // `last` is the residual of the final iterate
    for (;;) {
        if (cycle_only) {
        } else if constexpr (sizeof(T) == 4) {
            residual64<T>(p, p.x, lv[0].b, warp, nwarps);
            sync();
            check(norm_total(p.partials, n, false));
            tested = true;
            if (p.null_space) sync();   // the projection rewrites the partials
        } else if (p.tol > 0) {
            xfp = reinterpret_cast<double*>(lv[0].x[par & 1]);
            residual64<T>(p, xfp, nullptr, warp, nwarps);
            sync();
            check(norm_total(p.partials, n, false));
            tested = true;
            sync();   // a late block may still read the partials
        }
        if (done || cycles >= p.max_cycles) break;
        const int batch = cycle_only ? 1
                                     : (sizeof(T) == 8 && p.tol <= 0 ? p.max_cycles
                                                                     : min(p.interval, p.max_cycles - cycles));
        for (int c = 0; c < batch; ++c) vcycle(cycle_only || (sizeof(T) == 4 && c == 0));
        if (cycle_only) return;
        if constexpr (sizeof(T) == 4) {
            const T* e = lv[0].x[par & 1];
            for (int r = tid; r < n; r += nthr) p.x[r] += (double)e[r];
            ++refinements;
            sync();
        }
        cycles += batch;
        tested = false;
    }
    if constexpr (sizeof(T) == 8) {
        const T* xc = lv[0].x[par & 1];
        for (int r = tid; r < n; r += nthr) p.x[r] = (double)xc[r];
        sync();
    }
    if (p.null_space) {
        project(p.x, n, p.partials, sync, tid, nthr);
        tested = false;
    }
    if (!tested) {
        residual64<T>(p, p.x, (T*)nullptr, warp, nwarps);
        sync();
        const double s = norm_total(p.partials, n, false);
        if (first < 0) first = s;
        last = s;
    }
    if (tid == 0) {
        MGState* st = p.st;
        if (!(last == last) || last > 1e300) status = PSUM_ERR_DIVERGED;
        else if (status == 0 && p.tol > 0 && last > p.tol * p.tol * bn) status = PSUM_ERR_NOT_CONVERGED;
        st->bnorm2 = bnorm2;
        st->rnorm2_first = first;
        st->rnorm2_last = last;
        st->done = done;
        st->cycles = cycles;
        st->refinements = refinements;
        st->status = status;
        st->cycles_run = cycles;
        st->refinements_run = refinements;
    }
}

}  // namespace psum_b200
