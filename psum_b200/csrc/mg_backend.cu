// mg_backend.cu -- the B200 multigrid solver backends behind PSuM's func_table.
//
//   cuda_multigrid32f_gpu : FP32 V-cycles inside FP64 iterative refinement,
//                           restating sycl_multigrid32f_gpu::solve
//                           (src/field_solver/implements/sycl_multigrid32f_gpu.cpp:106-160)
//   cuda_multigrid64_gpu  : FP64 V-cycles with the caller's x as initial guess,
//                           restating cuda_multigrid_gpu::solve
//                           (src/field_solver/implements/cuda_multigrid_gpu.cu:140-180)
//
// Both accept PSuM's option grammar (sycl_multigrid32f_gpu.cpp:162-196) and
// add `tol` (stop once ||b - A x||_2 <= tol ||b||_2, checked on the device
// every correction_interval cycles; 0 = run exactly max_cycles like PSuM),
// `max_coarse`, and `periodic_I/J/K 1` (wrap-around transfers on that axis
// for operators whose node lattice wraps, where PSuM's open-interval
// transfers make the V-cycle diverge), and `null_space 1` (a periodic
// operator assembled without a pinned node, singular with the constants as
// its null space: the coarse solve inverts Ahat_L + 1 1^T / n and the solve
// returns the mean-zero solution of b minus its mean).  The whole solve is enqueued on one stream without host
// synchronisation; func_table.solve synchronises at the end, like PSuM.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

#include <cudaTypedefs.h>

#include "common.hpp"
#include "mg_backend.hpp"
#include "mg_host.hpp"
#include "mg_kernels.cuh"
#include "mg_persist.cuh"

namespace psum_b200 {

namespace mgdetail {

inline unsigned grid_for(long long n, int threads = kThreads) {
    return (unsigned)std::max<long long>(1, (n + threads - 1) / threads);
}

constexpr int kNormBlocks = 444;   // 3 x 148 SMs: fixed grid -> fixed reduction order

template <class T>
struct DevStencil {
    StencilDev<T> view{};
    PersistStencil<T> persist{};   // the operator as the one-kernel solve reads it
    DevBuf<unsigned char> rows;    // its exception words, coefficients and flags, one buffer
    DevBuf<uint32_t> mask, mask_prefix;
    DevBuf<int> exc_ptr, exc_col;
    DevBuf<T> exc_val;
    long long exceptions = 0;

    void upload(const StencilOp& op, cudaStream_t s) {
        mask.upload(op.mask.data(), op.mask.size(), s);
        mask_prefix.upload(op.mask_prefix.data(), op.mask_prefix.size(), s);
        exc_ptr.upload(op.exc_ptr.data(), op.exc_ptr.size(), s);
        exc_col.upload(op.exc_col.data(), op.exc_col.size(), s);
        std::vector<T> v(op.exc_val.begin(), op.exc_val.end());
        exc_val.upload(v.data(), v.size(), s);
        cuda_check(cudaStreamSynchronize(s), "upload stencil");
        exceptions = (long long)op.exc_rows.size();
        if (op.n >= (1LL << 31)) throw std::invalid_argument("multigrid: more than 2^31 - 1 rows per level");
        view.n0 = op.dims[0];
        view.n1 = op.dims[1];
        view.n2 = op.dims[2];
        view.n = op.n;
        view.ns = op.ns;
        view.any_exc = exceptions > 0;
        view.div12 = make_fastdiv((unsigned)(op.dims[1] * op.dims[2]));
        view.div2 = make_fastdiv((unsigned)op.dims[2]);
        for (int t = 0; t < op.ns && t < kMaxTaps; ++t) {
            view.di[t] = (signed char)op.delta[t][0];
            view.dj[t] = (signed char)op.delta[t][1];
            view.dk[t] = (signed char)op.delta[t][2];
            view.off[t] = (op.delta[t][0] * op.dims[1] + op.delta[t][1]) * op.dims[2] + op.delta[t][2];
            view.c[t] = T(op.coef[t]);
        }
        view.mask = mask.p;
        view.mask_prefix = mask_prefix.p;
        view.exc_ptr = exc_ptr.p;
        view.exc_col = exc_col.p;
        view.exc_val = exc_val.p;
    }

    // The stencil's shape, and every exception row as coefficients on the
    // shape's taps.  A row whose columns do not ascend with the taps (it
    // wraps around a face) would be summed in another order there: it keeps
    // its column list.
    void upload_persist(const StencilOp& op, cudaStream_t s) {
        persist = PersistStencil<T>{};
        persist.s = view;
        for (int ns : {3, 5, 7, 9, 27}) {
            bool same = ns == op.ns;
            for (int t = 0; t < ns && same; ++t)
                for (int a = 0; a < 3; ++a) same = same && op.delta[t][a] == shape_tap(ns, t, a);
            for (int a = 0; a < 3; ++a) same = same && op.dims[a] != 2;   // -1 and +1 would be the same neighbour
            if (ns == 3 || ns == 5 || ns == 9) same = same && op.dims[2] == 1 && (ns != 3 || op.dims[1] == 1);
            if (same) persist.shape = ns;
        }
        if (!persist.shape || !exceptions) return;
        std::vector<uint2> w(op.mask.size());
        for (size_t q = 0; q < w.size(); ++q) w[q] = make_uint2(op.mask[q], op.mask_prefix[q]);
        std::vector<T> c((size_t)exceptions * persist.shape, T(0));
        std::vector<uint8_t> list((size_t)exceptions, 0);
        bool any_list = false;
        for (long long q = 0; q < exceptions; ++q) {
            const int r = op.exc_rows[q];
            const int rc[3] = {r / (op.dims[1] * op.dims[2]), r / op.dims[2] % op.dims[1], r % op.dims[2]};
            int t = -1;
            bool ok = true;
            for (int e = op.exc_ptr[q]; e < op.exc_ptr[q + 1] && ok; ++e) {
                int found = -1;
                for (int u = t + 1; u < persist.shape && found < 0; ++u) {
                    long long col = 0;
                    for (int a = 0; a < 3; ++a) {
                        const int i = (rc[a] + op.delta[u][a] + op.dims[a]) % op.dims[a];
                        col = col * op.dims[a] + i;
                    }
                    if (col == op.exc_col[e]) found = u;
                }
                ok = found >= 0;
                if (ok) c[(size_t)q * persist.shape + found] = T(op.exc_val[e]);
                t = found;
            }
            list[q] = !ok;
            any_list |= !ok;
        }
        const size_t wb = w.size() * sizeof(uint2), cb = c.size() * sizeof(T);
        std::vector<unsigned char> h(wb + cb + list.size());
        std::memcpy(h.data(), w.data(), wb);
        std::memcpy(h.data() + wb, c.data(), cb);
        std::memcpy(h.data() + wb + cb, list.data(), list.size());
        rows.upload(h.data(), h.size(), s);
        cuda_check(cudaStreamSynchronize(s), "upload stencil");
        persist.word = reinterpret_cast<const uint2*>(rows.p);
        persist.dense = reinterpret_cast<const T*>(rows.p + wb);
        persist.csr = any_list ? rows.p + wb + cb : nullptr;
    }
};

template <class T>
struct DevAxis {
    DevBuf<int> p_c0, p_c1, r_f;
    DevBuf<T> p_w0, p_w1, r_w;
    // The same factors as whole entries (one-kernel solve).
    static void entries(const Axis1D& a, RestrictEntry<T>* re, ProlongEntry<T>* pe) {
        for (int c = 0; c < a.nc; ++c)
            for (int q = 0; q < 3; ++q) {
                re[c].f[q] = std::max(0, a.r_f[3 * c + q]);
                re[c].w[q] = a.r_f[3 * c + q] < 0 ? T(0) : T(a.r_w[3 * c + q]);
            }
        for (int f = 0; f < a.nf; ++f) {
            pe[f].c[0] = std::max(0, a.p_c0[f]);
            pe[f].c[1] = std::max(0, a.p_c1[f]);
            pe[f].w[0] = a.p_c0[f] < 0 ? T(0) : T(a.p_w0[f]);
            pe[f].w[1] = a.p_c1[f] < 0 ? T(0) : T(a.p_w1[f]);
        }
    }
    void upload(const Axis1D& a, cudaStream_t s, AxisDev<T>& view) {

        std::vector<T> w0(a.p_w0.begin(), a.p_w0.end()), w1(a.p_w1.begin(), a.p_w1.end()),
            rw(a.r_w.begin(), a.r_w.end());
        p_c0.upload(a.p_c0.data(), a.p_c0.size(), s);
        p_c1.upload(a.p_c1.data(), a.p_c1.size(), s);
        r_f.upload(a.r_f.data(), a.r_f.size(), s);
        p_w0.upload(w0.data(), w0.size(), s);
        p_w1.upload(w1.data(), w1.size(), s);
        r_w.upload(rw.data(), rw.size(), s);
        cuda_check(cudaStreamSynchronize(s), "upload transfer");
        view.nf = a.nf;
        view.nc = a.nc;
        view.p_c0 = p_c0.p;
        view.p_c1 = p_c1.p;
        view.p_w0 = p_w0.p;
        view.p_w1 = p_w1.p;
        view.r_f = r_f.p;
        view.r_w = r_w.p;
    }
};

// Launches of the stencil kernels with the operator's tap count as a
// compile-time constant where it is one of the common ones.
// 3-D levels of at least this many rows whose rows are a multiple of 16
// bytes long take the TMA-staged sweep (when the solver's option `tma` is on;
// option `tma_min_rows` overrides it).  Smaller levels stay in L2, where the
// per-row kernel's cached reads need no staging.
constexpr long long kTmaMinRows = 1LL << 20;

// Blocks of a TMA-staged sweep that fit on the GPU at once (SMs x resident
// blocks of the kernel); the kernel's shared memory is allowed on the way.
template <class T, int Mode, int NS>
int tma_resident_blocks() {
    static PerDevice<int> blocks;
    return blocks.get([](int dev) {
        int sms = 0, per_sm = 0;
        cuda_check(cudaFuncSetAttribute(k_level_op_tma<T, Mode, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)TmaShape<T, NS>::smem()),
                   "cudaFuncSetAttribute");
        cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_level_op_tma<T, Mode, NS>, kTmaThreads,
                                                                 TmaShape<T, NS>::smem()),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        return std::max(1, sms * std::max(1, per_sm));
    });
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
inline PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        cuda_check(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q),
                   "cudaGetDriverEntryPoint");
        if (q != cudaDriverEntryPointSuccess || !p) throw Error(PSUM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// The tensor map of a level vector viewed as (planes, rows, columns) with the
// sweep's box; the vector is one of the solver's own buffers on this GPU.
template <class T, int NS>
CUtensorMap make_level_map(const T* x, int P, int R, int C) {
    using S = TmaShape<T, NS>;
    CUtensorMap m;
    const cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)R, (cuuint64_t)P};
    const cuuint64_t strides[2] = {(cuuint64_t)C * sizeof(T), (cuuint64_t)R * C * sizeof(T)};
    const cuuint32_t box[3] = {(cuuint32_t)S::W, (cuuint32_t)S::H, 1u};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    const CUresult r = tmap_encoder()(&m, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                                      3, const_cast<T*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(PSUM_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    return m;
}

// Tensor maps of the level vectors the sweeps read, by pointer, view and
// stencil shape (the shape sets the box).
struct TmapCache {
    struct Entry {
        const void* p;
        int P, R, C, ns;
        CUtensorMap m;
    };
    std::vector<Entry> e;
    template <class T, int NS>
    CUtensorMap get(const T* x, int P, int R, int C) {   // by value: a later insertion may move the entries
        for (auto& q : e)
            if (q.p == x && q.P == P && q.R == R && q.C == C && q.ns == NS) return q.m;
        e.push_back({x, P, R, C, NS, make_level_map<T, NS>(x, P, R, C)});
        return e.back().m;
    }
};

// Launch over V's tiles; the planes are cut into as many chunks as keep one
// wave of resident blocks busy (each chunk re-reads two halo planes).
template <class T, int Mode, int NS>
void launch_tma_ns(TmapCache& cache, const StencilDev<T>& A, const T* x, const T* b, T* out, T omega,
                   const MGState* st, Stall* stall, cudaStream_t s) {
    using S = TmaShape<T, NS>;
    TmaTile V{};
    V.P = A.n0;
    V.R = A.n1;
    V.C = A.n2;
    V.tiles_c = (V.C + S::TC - 1) / S::TC;
    V.tiles_r = (V.R + S::TR - 1) / S::TR;
    const CUtensorMap map = cache.get<T, NS>(x, V.P, V.R, V.C);
    const long long tiles = (long long)V.tiles_c * V.tiles_r;
    const long long want = std::max(1LL, (long long)tma_resident_blocks<T, Mode, NS>() / tiles);
    V.chunk = (int)std::max(1LL, (V.P + want - 1) / want);
    V.chunks = (V.P + V.chunk - 1) / V.chunk;
    const unsigned blocks = (unsigned)(tiles * V.chunks);
    k_level_op_tma<T, Mode, NS><<<blocks, kTmaThreads, S::smem(), s>>>(map, A, V, x, b, out, omega, st, stall);
}

// Whether the TMA-staged sweep takes a level: not small, 3-D, rows a multiple
// of 16 bytes long, one of the kernel's two stencil shapes.
template <class T>
bool tma_level(const StencilDev<T>& A, long long min_rows) {
    if (A.n < min_rows) return false;
    if (!(A.n0 > 2 && A.n1 > 1 && A.n2 > 1)) return false;          // 3-D boxes only (2-D levels stay in L2)
    if ((A.n2 * (int)sizeof(T)) % 16 != 0) return false;             // tensor-map row pitch: 16-byte multiple
    if (A.ns != 7 && A.ns != 27) return false;                         // the kernel's two stencil shapes
    for (int t = 0; t < A.ns; ++t)
        if (A.di[t] != tma_tap_d(A.ns, t, 0) || A.dj[t] != tma_tap_d(A.ns, t, 1) || A.dk[t] != tma_tap_d(A.ns, t, 2))
            return false;
    return true;
}

// TMA-staged sweep of a level (k_level_op_tma); false when the level does not qualify.
template <class T, int Mode>
bool launch_level_op_tma(TmapCache& cache, long long min_rows, const StencilDev<T>& A, const T* x, const T* b, T* out,
                         T omega, const MGState* st, Stall* stall, cudaStream_t s) {
    if (Mode == kSmoothFromZero || !tma_level(A, min_rows)) return false;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return false;
    if (A.ns == 7) launch_tma_ns<T, Mode, 7>(cache, A, x, b, out, omega, st, stall, s);
    else launch_tma_ns<T, Mode, 27>(cache, A, x, b, out, omega, st, stall, s);
    count_launch();
    return true;
}

template <class T, int Mode>
void launch_level_op(const StencilDev<T>& A, const T* x, const T* b, T* out, T omega, const MGState* st,
                     cudaStream_t s, Stall* stall = nullptr, TmapCache* cache = nullptr,
                     long long tma_min_rows = kTmaMinRows) {
    if (stall && cache && launch_level_op_tma<T, Mode>(*cache, tma_min_rows, A, x, b, out, omega, st, stall, s)) return;
    const unsigned g = grid_for(A.n);
    if (Mode == kSmoothFromZero) k_level_op<T, Mode, 0><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    else if (A.ns == 5) k_level_op<T, Mode, 5><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    else if (A.ns == 7) k_level_op<T, Mode, 7><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    else if (A.ns == 9) k_level_op<T, Mode, 9><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    else if (A.ns == 27) k_level_op<T, Mode, 27><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    else k_level_op<T, Mode, 0><<<g, kThreads, 0, s>>>(A, x, b, out, omega, st);
    count_launch();
}

template <class TOut>
void launch_residual64(const StencilDev<double>& A, const double* x, const double* b, const double* dinv, TOut* bhat,
                       double* partials, const MGState* st, int gated, cudaStream_t s) {
    if (A.ns == 5) k_residual64<TOut, 5><<<kNormBlocks, kThreads, 0, s>>>(A, x, b, dinv, bhat, partials, st, gated);
    else if (A.ns == 7) k_residual64<TOut, 7><<<kNormBlocks, kThreads, 0, s>>>(A, x, b, dinv, bhat, partials, st, gated);
    else if (A.ns == 9) k_residual64<TOut, 9><<<kNormBlocks, kThreads, 0, s>>>(A, x, b, dinv, bhat, partials, st, gated);
    else if (A.ns == 27) k_residual64<TOut, 27><<<kNormBlocks, kThreads, 0, s>>>(A, x, b, dinv, bhat, partials, st, gated);
    else k_residual64<TOut, 0><<<kNormBlocks, kThreads, 0, s>>>(A, x, b, dinv, bhat, partials, st, gated);
    count_launch();
}

// ------------------------------------------------- one-kernel solves --
// Which levels one kernel takes, and how its blocks meet.  Solves on a B200,
// one launch per step against one kernel: 64^2 FP64 3.3 -> 0.43 ms, 256^2
// mixed 4.4 -> 0.63, 1025^2 mixed 6.0 -> 1.24, 33 x 41 x 29 FP64 4.3 -> 1.7,
// 128^3 mixed 7.2 -> 2.3 (14 cycles).  About the limit, to 1e-8: 1400^2 mixed
// 3.8 -> 2.1, 128^3 FP64 4.9 -> 4.1 (all levels); 1504 x 1600 mixed 3.9 -> 3.7,
// 2049^2 mixed 5.0 -> 4.1, 129^3 mixed 6.1 -> 4.4, 160^3 mixed 5.7 -> 5.0 and
// FP64 6.9 -> 6.5, 200^3 mixed 15.0 -> 12.5 (coarse levels only).  256^3 mixed
// takes 14.1 that way and 21.4 with all levels inside: its finest level
// streams from HBM, where the TMA-staged sweep is twice as fast.  Finest
// levels between 2^21 and 2^24 rows were not tried inside the kernel.
constexpr long long kPersistRows = 1LL << 21;     // largest level worked inside the kernel
// Up to here one cluster of 16 blocks, above one block per SM: a cluster
// barrier and its loads take about 1 us a step against 2.6, but 16 SMs sweep
// 65536 rows in 3.4 us, as long as 148 take for 512 x 512.
constexpr long long kClusterRows = 100000;
constexpr long long kTailBytes = 176 << 10;       // rows x taps x element size a tail level may have ...
constexpr long long kTailBytesGrid = 256 << 10;   // ... and under a grid barrier, which costs more than a slow sweep
constexpr size_t kTailSmem = 200 << 10;           // shared memory of the tail's vectors

inline int device_sms() {
    static PerDevice<int> sms;
    return sms.get([](int dev) {
        int n = 0;
        cuda_check(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
        return n;
    });
}

// Blocks of the whole-GPU kernel when `beside` particles are still being
// written (the fused step's second pass): a block takes its SM, so a pass
// that lasts as long as the solve goes on with the others.  By particles per
// row; a step with every SM against the share taken from there on:
//   128^3 rows: 0.01 4.05 / 4.66 ms, 1 6.49 / 7.03, 4 6.46 / 6.66,
//     16 6.35 / 6.36, 60 8.42 / 8.22 (two thirds; 32 and a quarter: 8.3);
//   64^3 rows: 8 2.11 / 2.08, 32 2.15 / 2.10, 120 3.14 / 3.03 (two thirds),
//     500 8.59 / 8.23 (a quarter);
//   351^2 rows: 64 1.44 / 1.41, 250 1.40 / 1.31 (two thirds),
//     500 1.89 / 1.71, 1000 3.36 / 2.97 (a quarter);
//   1025^2 rows: 512 9.15 / 8.78 (a quarter; 20 blocks: 9.38).
inline int persist_blocks(long long beside, long long rows) {
    const int sms = device_sms();
    if (beside < 8 * rows) return sms;
    return std::max(1, beside >= 256 * rows ? sms / 4 : sms * 2 / 3);
}

// Whole-GPU solves of one device in turn.  Their blocks wait for one another
// and take an SM each, so two of them (two handles on two streams, two
// threads) must not be placed side by side by halves: each waits for the
// event of the one before.  A solver's own graph is ordered where it is
// launched (solver_solve_async); a graph of the caller's holds no such kernel
// (SolverBase::callers_graph).
class Turn {
    struct Device {
        std::mutex m;
        cudaEvent_t last = nullptr;
    };
    Device* d = nullptr;
    cudaStream_t s;

public:
    Turn(cudaStream_t stream, bool needed) : s(stream) {
        if (!needed) return;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cuda_check(cudaStreamIsCapturing(s, &cs), "cudaStreamIsCapturing");
        if (cs != cudaStreamCaptureStatusNone) return;
        static Device devices[64];
        int dev = 0;
        cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
        if (dev < 0 || dev >= 64) throw Error(PSUM_ERR_INTERNAL, "device ordinal out of range");
        devices[dev].m.lock();
        d = &devices[dev];
        const cudaError_t e = d->last ? cudaStreamWaitEvent(s, d->last, 0)
                                      : cudaEventCreateWithFlags(&d->last, cudaEventDisableTiming);
        if (e != cudaSuccess) {
            d->m.unlock();
            d = nullptr;
            cuda_check(e, "order of whole-GPU solves");
        }
    }
    Turn(const Turn&) = delete;
    Turn& operator=(const Turn&) = delete;
    ~Turn() {
        if (!d) return;
        cudaEventRecord(d->last, s);
        d->m.unlock();
    }
};

// Whether the GPU places a cluster of 16 blocks of the kernel.
template <class T>
bool cluster_fits() {
    static PerDevice<bool> fits;
    return fits.get([](int) {
        if (cudaFuncSetAttribute(k_mg_persist<T, kSyncCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_mg_persist<T, kSyncCluster>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return false;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kClusterBlocks);
        cfg.blockDim = dim3(kPersistThreads<T>);
        cfg.dynamicSmemBytes = kTailSmem;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kClusterBlocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, k_mg_persist<T, kSyncCluster>, &cfg);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && n >= 1;
    });
}

// Whether the device takes the whole-GPU kernel: launched cooperatively, one
// block per SM.
template <class T>
bool whole_gpu_fits() {
    static PerDevice<bool> fits;
    return fits.get([](int dev) {
        int coop = 0, per_sm = 0;
        cuda_check(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev), "cudaDeviceGetAttribute");
        if (!coop) return false;
        if (cudaFuncSetAttribute(k_mg_persist<T, kSyncGrid>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mg_persist<T, kSyncGrid>, kPersistThreads<T>,
                                                          kTailSmem) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return per_sm >= 1;
    });
}

// False where the device refuses the cooperative launch (a share of its SMs
// only, whatever the attributes say).
template <class T, int SYNC>
bool launch_persist_sync(const PersistArgs<T>& a, size_t smem, long long beside, cudaStream_t s) {
    static PerDevice<bool> ready;
    ready.get([](int) {
        cuda_check(cudaFuncSetAttribute(k_mg_persist<T, SYNC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kTailSmem),
                   "cudaFuncSetAttribute");
        return true;
    });
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(SYNC == kSyncBlock ? 1 : (SYNC == kSyncCluster ? kClusterBlocks : persist_blocks(beside, (long long)a.lv[0].n)));
    cfg.blockDim = dim3(kPersistThreads<T>);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    if (SYNC == kSyncCluster) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kClusterBlocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    cfg.attrs = &at;
    cfg.numAttrs = SYNC == kSyncBlock ? 0 : 1;
    const Turn turn(s, SYNC == kSyncGrid);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_mg_persist<T, SYNC>, a);
    if (SYNC == kSyncGrid && (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported)) {
        cudaGetLastError();
        return false;
    }
    cuda_check(e, "multigrid kernel launch");
    count_launch();
    return true;
}

template <class T>
bool launch_persist(const PersistArgs<T>& a, int sync, size_t smem, long long beside, cudaStream_t s) {
    if (sync == kSyncBlock) return launch_persist_sync<T, kSyncBlock>(a, smem, beside, s);
    if (sync == kSyncCluster) return launch_persist_sync<T, kSyncCluster>(a, smem, beside, s);
    return launch_persist_sync<T, kSyncGrid>(a, smem, beside, s);
}

template <class T>
struct Level {
    long long n = 0;
    DevStencil<T> op;
    DevBuf<T> dinv;
    DevBuf<T> bufA, bufB, b;   // x ping-pong pair and right-hand side
    XferDev<T> xfer{};         // to the next coarser level
    DevAxis<T> axes[3];
    DevBuf<unsigned char> entries;   // RestrictEntry and ProlongEntry tables of the three axes, one buffer
    const RestrictEntry<T>* rest[3] = {};
    const ProlongEntry<T>* prol[3] = {};
    void upload_entries(const std::array<Axis1D, 3>& ax, cudaStream_t s) {
        size_t at[6], bytes = 0;
        for (int a = 0; a < 3; ++a) {
            at[a] = bytes;
            bytes += sizeof(RestrictEntry<T>) * ax[a].nc;
            at[3 + a] = bytes = (bytes + 31) / 32 * 32;
            bytes = (bytes + sizeof(ProlongEntry<T>) * ax[a].nf + 31) / 32 * 32;
        }
        std::vector<unsigned char> h(bytes);
        for (int a = 0; a < 3; ++a)
            DevAxis<T>::entries(ax[a], reinterpret_cast<RestrictEntry<T>*>(h.data() + at[a]),
                                reinterpret_cast<ProlongEntry<T>*>(h.data() + at[3 + a]));
        entries.upload(h.data(), bytes, s);
        cuda_check(cudaStreamSynchronize(s), "upload transfer");
        for (int a = 0; a < 3; ++a) {
            rest[a] = reinterpret_cast<const RestrictEntry<T>*>(entries.p + at[a]);
            prol[a] = reinterpret_cast<const ProlongEntry<T>*>(entries.p + at[3 + a]);
        }
    }
};

}  // namespace mgdetail

using namespace mgdetail;

// ------------------------------------------------------------------------
struct SolverBase {
    uint32_t magic = kSolverMagic;
    int precision = 32;   // 32: mixed refinement, 64: FP64 V-cycles
    // options (defaults of sycl_multigrid32f_gpu.cpp:28-38)
    int I = 0, J = 0, K = 0;
    int depth = 3, pre_relax = 2, post_relax = 1, max_cycles = 10, correction_interval = 4;
    int max_coarse = 8192;
    std::array<int, 3> periodic{0, 0, 0};   // wrap-around transfers per axis (option periodic_I/J/K)
    double tol = 0.0;
    int null_space = 0;                     // option `null_space 0|1` (read by set_matrix)
    bool ns_built = false;                  // the hierarchy was built for a singular operator
    int use_graph = 1;                      // option `graph 0|1`: replay the solve as one CUDA graph
    int use_persist = 1;                    // option `persist 0|1`: the solve, or its coarse levels, as one kernel
    int use_tma = 1;                        // option `tma 0|1`: TMA-staged sweeps on large levels
    int barrier_polls = kBarrierPolls;      // option `barrier_polls`: wait limit of a whole-GPU barrier
    long long tma_min_rows = 0;             // option `tma_min_rows`: smallest level (rows) swept that way (0: rule)
    unsigned long long n_row = 0;
    long long beside = 0;                   // particles being written meanwhile (solver_solve_async)
    bool callers_graph = false;             // recorded into a graph that the caller replays when it likes
    bool whole_gpu = true;                  // false once the device has refused a whole-GPU kernel: launched kernels instead
    bool ready = false;
    cudaStream_t own_stream = nullptr;
    // The solve's launch sequence depends only on the options, the operator,
    // the sources and the (b, x) pointers: it is captured once into a CUDA
    // graph and replayed while none of them changes (`version` counts the
    // changes of the first three).
    unsigned long long version = 0;
    struct {
        cudaGraphExec_t exec = nullptr;
        const double* b = nullptr;
        const double* x = nullptr;
        unsigned long long version = 0;
        unsigned long long kernels = 0;
    } graph;
    // sources (host copies kept, device copies uploaded at set time)
    std::vector<unsigned long long> rep_idx, add_idx;
    std::vector<double> rep_val, add_val;
    DevBuf<unsigned long long> d_rep_idx, d_add_idx;
    DevBuf<double> d_rep_val, d_add_val;
    // FP64 fine operator for the residual
    DevStencil<double> a0;
    DevBuf<double> dinv0;
    DevBuf<double> partials;
    DevBuf<MGState> state;
    int* stalled = nullptr;   // pinned, written by a kernel that gave up a wait (Stall::report)
    Hierarchy host;   // kept for introspection
    int levels = 0;
    unsigned long long coarse_rows = 0;

    virtual int tma_level_vectors() const { return 0; }   // level vectors swept by the TMA-staged kernel so far
    virtual ~SolverBase() {
        drop_graph();
        if (aux_stream) cudaStreamDestroy(aux_stream);
        if (own_stream) cudaStreamDestroy(own_stream);
        give_host_word(stalled);   // the solver's buffers are freed by now, which waits for its kernels
    }
    void drop_graph() {
        if (graph.exec) cudaGraphExecDestroy(graph.exec);
        graph.exec = nullptr;
    }
    cudaStream_t aux_stream = nullptr;      // captures the body of a conditional loop
    unsigned long long loop_kernels = 0;    // kernels captured into loop bodies (counted on the device)
    virtual bool one_kernel() const { return false; }   // the solve is a single kernel: no graph is captured
    virtual bool waits_on_gpu() const { return false; }   // holds a kernel whose blocks wait over the whole GPU
    virtual void build_device(cudaStream_t s) = 0;
    virtual void build_persist(cudaStream_t s) = 0;   // tables of the one-kernel solve, unless they are there
    virtual void enqueue_solve(double* b, double* x, cudaStream_t s) = 0;
};

namespace {

template <class T>
struct Solver : SolverBase {
    std::vector<std::unique_ptr<Level<T>>> lv;
    DevBuf<double> coarse_inv;   // FP64 in both backends (see k_dense_mv)
    DevBuf<double> x64;   // FP64 level-0 iterate for the FP64 backend
    void build_device(cudaStream_t s) override {
        tmaps.e.clear();
        a0.upload(host.a0, s);
        persist_tables = false;
        dinv0.upload(host.dinv[0].data(), host.dinv[0].size(), s);
        partials.alloc(std::max(kNormBlocks, kNormVWarps));
        MGState fresh{};
        fresh.stall.report = stalled;
        state.upload(&fresh, 1, s);
        cuda_check(cudaStreamSynchronize(s), "build_device");
        lv.clear();
        for (int l = 0; l <= host.L; ++l) {
            auto L = std::make_unique<Level<T>>();
            L->n = (long long)host.dims[l][0] * host.dims[l][1] * host.dims[l][2];
            if (l < host.L) L->op.upload(host.ahat[l], s);
            std::vector<T> d(host.dinv[l].begin(), host.dinv[l].end());
            L->dinv.upload(d.data(), d.size(), s);
            // +16 elements: the TMA-staged sweep's 16-byte-aligned copies may read past a vector's last element
            L->bufA.alloc(L->n + 16);
            L->bufB.alloc(L->n + 16);
            L->b.alloc(L->n + 16);
            if (l < host.L) {
                for (int a = 0; a < 3; ++a) L->axes[a].upload(host.xfer[l][a], s, L->xfer.ax[a]);
                const AxisDev<T>* ax = L->xfer.ax;
                L->xfer.divc12 = make_fastdiv((unsigned)(ax[1].nc * ax[2].nc));
                L->xfer.divc2 = make_fastdiv((unsigned)ax[2].nc);
                L->xfer.divf12 = make_fastdiv((unsigned)(ax[1].nf * ax[2].nf));
                L->xfer.divf2 = make_fastdiv((unsigned)ax[2].nf);
            }
            lv.push_back(std::move(L));
        }
        coarse_inv.upload(host.coarse_inv.data(), host.coarse_inv.size(), s);
        if (precision == 64) x64.alloc(n_row + 16);
        if (use_persist) build_persist(s);
        cuda_check(cudaStreamSynchronize(s), "build_device");
        levels = host.L + 1;
        coarse_rows = (unsigned long long)lv.back()->n;
    }

    // The operators and transfers as the one-kernel solve reads them, for the
    // levels that it can work (with varying coefficients many rows
    // are exception rows: 40 to 216 bytes more each).
    bool persist_tables = false;
    void build_persist(cudaStream_t s) override {
        if (persist_tables || host.L < 1 || host.L + 1 > kPersistLevels) return;
        for (int l = 0; l < host.L; ++l) {
            if (lv[l]->n > kPersistRows) continue;
            lv[l]->op.upload_persist(host.ahat[l], s);
            lv[l]->upload_entries(host.xfer[l], s);
        }
        if (lv[0]->n <= kPersistRows) a0.upload_persist(host.a0, s);
        persist_tables = true;
    }

    // where the TMA-staged sweeps record a stall, or null when option `tma` is off
    Stall* tma_stall() { return use_tma ? &state.p->stall : nullptr; }
    TmapCache tmaps;   // tensor maps of the level vectors (rebuilt with the hierarchy)
    int tma_level_vectors() const override { return (int)tmaps.e.size(); }

    // One-kernel plan: the first level the kernel takes (0: the whole solve;
    // L + 1: none), its tail and its barrier.
    struct Plan {
        int first = 0, tail = 0, sync = kSyncGrid;
        bool dense_all = false;
        size_t smem = 0;
    };
    Plan persist_plan() const {
        Plan P;
        const int L = host.L;
        P.first = L + 1;
        // mixed solves with graph 0 launch every kernel (profiling); the FP64 backend has the same launches either way
        if (!use_persist || !persist_tables || (precision == 32 && !use_graph)) return P;
        int first = 0;
        while (first < L && (lv[first]->n > kPersistRows || (use_tma && tma_level(lv[first]->op.view, tma_rows()))))
            ++first;
        if (first >= L) return P;
        size_t elems = 3 * (size_t)lv[L]->n;
        if (elems * sizeof(T) > kTailSmem) return P;
        const bool grid = lv[first]->n > kClusterRows || !cluster_fits<T>();
        int tail = L;
        while (tail > first) {
            const Level<T>& V = *lv[tail - 1];
            if (V.n * V.op.view.ns * (long long)sizeof(T) > (grid ? kTailBytesGrid : kTailBytes) ||
                (elems + 3 * (size_t)V.n) * sizeof(T) > kTailSmem)
                break;
            elems += 3 * (size_t)V.n;
            --tail;
        }
        if (tail > first && grid && !grid_ok()) return P;
        P.first = first;
        P.tail = tail;
        P.dense_all = lv[L]->n > kDenseTailRows;
        P.smem = tail < L ? elems * sizeof(T) : 0;
        P.sync = tail == first ? kSyncBlock : (grid ? kSyncGrid : kSyncCluster);
        return P;
    }
    bool grid_ok() const { return whole_gpu && !callers_graph && whole_gpu_fits<T>(); }
    // Smallest level of the TMA-staged sweep: the option, or by rule 2^20 rows
    // in a problem that is too large for one kernel.  A smaller problem is
    // worked whole by one (128^3 nodes, 14 mixed cycles: 2.3 ms against 3.8
    // with the finest level's sweeps TMA-staged and launched).
    long long tma_rows() const {
        if (tma_min_rows > 0) return tma_min_rows;
        const bool whole = use_persist && persist_tables && !(precision == 32 && !use_graph) && lv[0]->n <= kPersistRows && grid_ok();
        return whole ? kPersistRows + 1 : kTmaMinRows;
    }
    PersistArgs<T> persist_args(const Plan& P, double* b, double* x) {
        PersistArgs<T> a{};
        const int L = host.L;
        int at = 0;
        for (int l = L; l >= 0; --l) {
            PersistLevel<T>& q = a.lv[l];
            q.A = lv[l]->op.persist;
            q.X = lv[l]->xfer;
            for (int d = 0; d < 3; ++d) {
                q.rest[d] = lv[l]->rest[d];
                q.prol[d] = lv[l]->prol[d];
            }
            q.dim = q.A.s.n2 > 1 ? 3 : (q.A.s.n1 > 1 ? 2 : 1);
            q.x[0] = lv[l]->bufA.p;
            q.x[1] = lv[l]->bufB.p;
            q.b = lv[l]->b.p;
            q.dinv = lv[l]->dinv.p;
            q.n = (int)lv[l]->n;
            if (l >= P.tail) {
                q.smem = at;
                at += 3 * q.n;
            }
        }
        if (precision == 64) a.lv[0].x[0] = reinterpret_cast<T*>(x64.p);
        a.a0 = a0.persist;
        a.dinv0 = dinv0.p;
        a.coarse_inv = coarse_inv.p;
        a.b = b;
        a.x = x;
        a.add_idx = d_add_idx.p;
        a.add_val = d_add_val.p;
        a.rep_idx = d_rep_idx.p;
        a.rep_val = d_rep_val.p;
        a.n_add = (long long)add_idx.size();
        a.n_rep = (long long)rep_idx.size();
        a.partials = partials.p;
        a.st = state.p;
        a.counter = &state.p->arrivals;
        a.polls = barrier_polls;
        a.tol = tol;
        a.first = P.first;
        a.tail = P.tail;
        a.last = L;
        a.dense_all = P.dense_all;
        a.pre = pre_relax;
        a.post = post_relax;
        a.max_cycles = max_cycles;
        a.interval = correction_interval;
        a.null_space = ns_built;
        return a;
    }
    bool one_kernel() const override { return ready_levels() && persist_plan().first == 0; }
    bool waits_on_gpu() const override {
        const Plan P = persist_plan();
        return P.first <= host.L && P.sync == kSyncGrid;
    }
    bool ready_levels() const { return (int)lv.size() == host.L + 1; }

    // The whole solve as one kernel; false when the device refuses it.
    bool enqueue_persist(const Plan& P, double* b, double* x, cudaStream_t s) {
        PersistArgs<T> a = persist_args(P, b, x);
        a.mode = precision == 64 ? kPersistFp64 : kPersistMixed;
        cuda_check(cudaMemsetAsync(&state.p->arrivals, 0, sizeof(unsigned), s), "memset");
        const bool taken = launch_persist(a, P.sync, P.smem, beside, s);
        if (!taken) whole_gpu = false;
        return taken;
    }

    // One V-cycle from level P.first (its right-hand side restricted, its
    // iterate zero) as one kernel; returns the buffer of its result, null when
    // the device refuses the kernel.
    T* enqueue_persist_cycle(const Plan& P, bool gated, cudaStream_t s) {
        PersistArgs<T> a = persist_args(P, nullptr, nullptr);
        a.mode = kPersistCycle;
        a.n_add = a.n_rep = 0;
        a.null_space = 0;
        a.max_cycles = 1;
        a.gated = gated;
        if (P.sync == kSyncGrid)
            cuda_check(cudaMemsetAsync(&state.p->arrivals, 0, sizeof(unsigned), s), "memset");
        // on every SM: the graph that holds it is replayed whatever runs beside it
        if (!launch_persist(a, P.sync, P.smem, 0, s)) {
            whole_gpu = false;
            return nullptr;
        }
        if (P.tail == P.first) return lv[P.first]->bufA.p;
        const int sweeps = (pre_relax >= 2 ? pre_relax - 2 : 0) + post_relax;
        return sweeps % 2 ? lv[P.first]->bufB.p : lv[P.first]->bufA.p;
    }

    // Enqueue `cycles` V(pre,post) cycles on level-0 (x0 in/out, b0 = scaled rhs).
    // `x_is_zero`: the level-0 iterate starts at zero (first sweep simplified).
    // Returns the buffer holding the final level-0 iterate.
    T* enqueue_vcycles(T* x0, T* other0, T* b0, int cycles, bool x_is_zero, cudaStream_t s, bool gated = true) {
        const MGState* st = gated ? state.p : nullptr;
        const T omega = T(2.0 / 3);
        const Plan P = persist_plan();
        int L = std::min(host.L, P.first);   // levels below are launched one kernel per step
        std::vector<T*> xcur(host.L + 1), xoth(host.L + 1), bl(host.L + 1);
        xcur[0] = x0;
        xoth[0] = other0;
        bl[0] = b0;
        for (int l = 1; l <= host.L; ++l) {
            xcur[l] = lv[l]->bufA.p;
            xoth[l] = lv[l]->bufB.p;
            bl[l] = lv[l]->b.p;
        }
        std::vector<bool> zero(host.L + 1, false);
        zero[0] = x_is_zero;
        auto smooth = [&](int l) {
            Level<T>& V = *lv[l];
            if (zero[l]) {
                launch_level_op<T, kSmoothFromZero>(V.op.view, xcur[l], bl[l], xoth[l], omega, st, s);
                zero[l] = false;
            } else {
                launch_level_op<T, kSmooth>(V.op.view, xcur[l], bl[l], xoth[l], omega, st, s, tma_stall(), &tmaps, tma_rows());
            }
            std::swap(xcur[l], xoth[l]);
        };
        auto down = [&](int from) {
            for (int l = from; l < L; ++l) {
                for (int k = 0; k < pre_relax; ++k) smooth(l);
                Level<T>& V = *lv[l];
                if (zero[l]) {
                    // x is zero: residual = b; restrict b directly
                    { k_restrict<T><<<grid_for(lv[l + 1]->n), kThreads, 0, s>>>(V.xfer, bl[l], bl[l + 1], xcur[l + 1],
                                                                             lv[l + 1]->dinv.p, st); count_launch(); }
                } else {
                    launch_level_op<T, kResidual>(V.op.view, xcur[l], bl[l], xoth[l], omega, st, s, tma_stall(), &tmaps, tma_rows());
                    { k_restrict<T><<<grid_for(lv[l + 1]->n), kThreads, 0, s>>>(V.xfer, xoth[l], bl[l + 1],
                                                                             xcur[l + 1], lv[l + 1]->dinv.p, st); count_launch(); }
                }
                zero[l + 1] = true;
            }
        };
        for (int c = 0; c < cycles; ++c) {
            down(0);
            T* coarse = L < host.L ? enqueue_persist_cycle(P, gated, s) : nullptr;
            if (L < host.L && !coarse) {   // refused: these levels too are launched from here on
                L = host.L;
                down(P.first);
            }
            if (coarse) {
                xcur[L] = coarse;
                zero[L] = false;
            } else {
                const int n = (int)lv[L]->n;
                { k_dense_mv<T><<<grid_for((long long)n * 32), kThreads, 0, s>>>(coarse_inv.p, bl[L], xcur[L], n, st); count_launch(); }
                zero[L] = false;
            }
            for (int l = L - 1; l >= 0; --l) {
                if (zero[l]) {
                    // only possible with pre_relax == 0 on a level that started at zero:
                    // x_l was never written; the restriction kernel did not zero it.
                    cuda_check(cudaMemsetAsync(xcur[l], 0, sizeof(T) * lv[l]->n, s), "memset");
                    zero[l] = false;
                }
                if (lv[l]->xfer.ax[2].nf % 4 == 0) {
                    k_prolong_add_row4<T><<<grid_for(lv[l]->n / 4), kThreads, 0, s>>>(lv[l]->xfer, xcur[l + 1],
                                                                                       xcur[l], st);
                } else {
                    k_prolong_add<T><<<grid_for((lv[l]->n + kProlongPer - 1) / kProlongPer), kThreads, 0, s>>>(
                        lv[l]->xfer, xcur[l + 1], xcur[l], st);
                }
                count_launch();
                for (int k = 0; k < post_relax; ++k) smooth(l);
            }
        }
        cuda_check(cudaGetLastError(), "multigrid kernel launch");
        return xcur[0];
    }

    // [residual, check] then WHILE(check says continue) { V-cycles, correct,
    // residual, check } (sycl_multigrid32f_gpu.cpp:137-157 with the loop kept
    // on the device).  The body's check adds the body's kernel count to the
    // mapped launch counter each time the body runs.
    void enqueue_refinement_loop(double* b, double* x, cudaStream_t s) {
        MGState* st = state.p;
        Level<T>& F = *lv[0];
        const long long n = (long long)n_row;
        const int ci = correction_interval;
        if (!aux_stream) throw Error(PSUM_ERR_INTERNAL, "multigrid: loop stream missing");
        unsigned long long* counter = device_launch_counter();   // created by set_matrix
        cudaStreamCaptureStatus cs;
        cudaGraph_t g = nullptr;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        cuda_check(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, &nd), "cudaStreamGetCaptureInfo");
        cudaGraphConditionalHandle h;
        cuda_check(cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault), "conditional handle");
        launch_residual64<T>(a0.view, x, b, dinv0.p, F.b.p, partials.p, st, 1, s);
        { k_check_loop<<<1, 32, 0, s>>>(partials.p, kNormBlocks, st, 0, max_cycles, tol, h, 0ull, counter); count_launch(); }
        cuda_check(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, &nd), "cudaStreamGetCaptureInfo");
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = h;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        cudaGraphNode_t loop;
        cuda_check(cudaGraphAddNode(&loop, g, deps, nd, &np), "add conditional node");
        cudaGraph_t body = np.conditional.phGraph_out[0];
        cuda_check(cudaStreamUpdateCaptureDependencies(s, &loop, 1, cudaStreamSetCaptureDependencies),
                   "update capture dependencies");
        cuda_check(cudaStreamBeginCaptureToGraph(aux_stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal),
                   "capture loop body");
        const unsigned long long k0 = thread_launches();
        unsigned long long body_kernels = 0;
        try {
            // inside the loop the solve is never done: the kernels skip the flag
            T* e = enqueue_vcycles(F.bufA.p, F.bufB.p, F.b.p, ci, /*x_is_zero=*/true, aux_stream, /*gated=*/false);
            { k_correct<T><<<grid_for(n), kThreads, 0, aux_stream>>>(x, e, n, nullptr); count_launch(); }
            launch_residual64<T>(a0.view, x, b, dinv0.p, F.b.p, partials.p, nullptr, 0, aux_stream);
            body_kernels = thread_launches() - k0 + 1;
            { k_check_loop<<<1, 32, 0, aux_stream>>>(partials.p, kNormBlocks, st, ci, max_cycles, tol, h,
                                                     body_kernels, counter); count_launch(); }
            cuda_check(cudaGetLastError(), "loop body launch");
        } catch (...) {
            cudaGraph_t tmp = nullptr;
            cudaStreamEndCapture(aux_stream, &tmp);
            uncount_launches(thread_launches() - k0);
            throw;
        }
        cuda_check(cudaStreamEndCapture(aux_stream, &body), "end loop body capture");
        uncount_launches(body_kernels);   // counted by the body's check, once per iteration run
        loop_kernels += body_kernels;
    }

    void enqueue_sources(double* b, cudaStream_t s) {
        const long long na = (long long)add_idx.size(), nr = (long long)rep_idx.size();
        if (na > 0) { k_addback<<<grid_for(na), kThreads, 0, s>>>(b, d_add_idx.p, d_add_val.p, na); count_launch(); }
        if (nr > 0) { k_replace<<<grid_for(nr), kThreads, 0, s>>>(b, d_rep_idx.p, d_rep_val.p, nr); count_launch(); }
    }

    // v -= mean(v) (two launches; fixed reduction order)
    void enqueue_project(double* v, cudaStream_t s) {
        const long long n = (long long)n_row;
        { k_sum<<<kNormBlocks, kThreads, 0, s>>>(v, n, partials.p); count_launch(); }
        { k_sub_mean<<<kNormBlocks, kThreads, 0, s>>>(v, n, partials.p, kNormBlocks); count_launch(); }
    }

    void enqueue_solve(double* b, double* x, cudaStream_t s) override {
        const long long n = (long long)n_row;
        MGState* st = state.p;
        if (ns_built && !rep_idx.empty())
            throw std::invalid_argument("multigrid: null_space 1 with fixed (replaced) nodes");
        if (const Plan P = persist_plan(); P.first == 0 && enqueue_persist(P, b, x, s)) return;
        enqueue_sources(b, s);
        // singular operator: solve for the consistent part of b (the mean-zero
        // projection; b is the solve's scratch like PSuM's source vector)
        if (ns_built) enqueue_project(b, s);
        { k_norm2<<<kNormBlocks, kThreads, 0, s>>>(b, n, partials.p); count_launch(); }
        { k_check<<<1, 32, 0, s>>>(partials.p, kNormBlocks, st, 0, tol, 0, 0); count_launch(); }
        Level<T>& F = *lv[0];
        int cycles_done = 0, refinements = 0;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cuda_check(cudaStreamIsCapturing(s, &cs), "cudaStreamIsCapturing");
        if (precision == 32 && cs == cudaStreamCaptureStatusActive && tol > 0 && max_cycles > 0 &&
            max_cycles % correction_interval == 0) {
            // captured into a graph: the refinements run as a conditional loop
            // that ends on the device once the residual test passes, so no
            // kernel of the cycles after convergence is launched
            enqueue_refinement_loop(b, x, s);
            cycles_done = max_cycles;
            refinements = max_cycles / correction_interval;
        } else if (precision == 32) {
            // FP64 refinement around FP32 V-cycles (sycl_multigrid32f_gpu.cpp:137-157)
            while (cycles_done < max_cycles) {
                const int batch = std::min(correction_interval, max_cycles - cycles_done);
                launch_residual64<T>(a0.view, x, b, dinv0.p, F.b.p, partials.p, st, 1, s);
                { k_check<<<1, 32, 0, s>>>(partials.p, kNormBlocks, st, 1, tol, cycles_done, refinements); count_launch(); }
                T* e = enqueue_vcycles(F.bufA.p, F.bufB.p, F.b.p, batch, /*x_is_zero=*/true, s);
                { k_correct<T><<<grid_for(n), kThreads, 0, s>>>(x, e, n, st); count_launch(); }
                cycles_done += batch;
                ++refinements;
            }
        } else {
            cuda_check(cudaMemcpyAsync(x64.p, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s), "copy x");
            { k_scale<T><<<grid_for(n), kThreads, 0, s>>>(b, dinv0.p, F.b.p, n); count_launch(); }
            double* xc = x64.p;
            double* xo = reinterpret_cast<double*>(F.bufB.p);
            while (cycles_done < max_cycles) {
                const int batch = tol > 0 ? std::min(correction_interval, max_cycles - cycles_done) : max_cycles;
                if (tol > 0) {
                    launch_residual64<double>(a0.view, xc, b, nullptr, (double*)nullptr, partials.p, st, 1, s);
                    { k_check<<<1, 32, 0, s>>>(partials.p, kNormBlocks, st, 1, tol, cycles_done, refinements); count_launch(); }
                }
                T* r = enqueue_vcycles(reinterpret_cast<T*>(xc), reinterpret_cast<T*>(xo), F.b.p, batch, false, s);
                if ((double*)r != xc) std::swap(xc, xo);
                cycles_done += batch;
            }
            cuda_check(cudaMemcpyAsync(x, xc, sizeof(double) * n, cudaMemcpyDeviceToDevice, s), "copy x");
        }
        if (ns_built) enqueue_project(x, s);   // the mean-zero representative
        launch_residual64<double>(a0.view, x, b, nullptr, (double*)nullptr, partials.p, st, 0, s);
        { k_check<<<1, 32, 0, s>>>(partials.p, kNormBlocks, st, 2, tol, cycles_done, refinements); count_launch(); }
        cuda_check(cudaGetLastError(), "solve launch");
    }
};

int parse_int(std::istringstream& iss, const std::string& key) {
    int v;
    if (!(iss >> v)) throw std::invalid_argument("set_options: option '" + key + "' needs an integer value");
    return v;
}

}  // namespace

SolverBase* solver_from_handle(void* h) {
    SolverBase* s = static_cast<SolverBase*>(h);
    if (!s || s->magic != kSolverMagic) throw Error(PSUM_ERR_INVALID_ARGUMENT, "not a handle of this library");
    return s;
}

cudaStream_t solver_stream(SolverBase* s) { return s->own_stream; }

SolverBase* create_solver(int precision) {
    SolverBase* s = precision == 64 ? static_cast<SolverBase*>(new Solver<double>())
                                    : static_cast<SolverBase*>(new Solver<float>());
    s->precision = precision;
    return s;   // the CUDA stream is created on first device use (set_matrix)
}

static void ensure_stream(SolverBase* s) {
    if (!s->own_stream)
        cuda_check(cudaStreamCreateWithFlags(&s->own_stream, cudaStreamNonBlocking), "cudaStreamCreate");
}

void solver_set_options(SolverBase* s, const char* options) {
    if (!options) throw std::invalid_argument("set_options: null option string");
    std::istringstream iss(options);
    std::string key;
    bool k_provided = false;
    while (iss >> key) {
        if (key == "I") s->I = parse_int(iss, key);
        else if (key == "J") s->J = parse_int(iss, key);
        else if (key == "K") {
            s->K = parse_int(iss, key);
            k_provided = true;
        } else if (key == "depth") s->depth = parse_int(iss, key);
        else if (key == "pre_relax") s->pre_relax = parse_int(iss, key);
        else if (key == "post_relax") s->post_relax = parse_int(iss, key);
        else if (key == "max_cycles") s->max_cycles = parse_int(iss, key);
        else if (key == "max_coarse") s->max_coarse = parse_int(iss, key);
        else if (key == "periodic_I") s->periodic[0] = parse_int(iss, key) != 0;
        else if (key == "periodic_J") s->periodic[1] = parse_int(iss, key) != 0;
        else if (key == "periodic_K") s->periodic[2] = parse_int(iss, key) != 0;
        else if (key == "graph") s->use_graph = parse_int(iss, key) != 0;
        else if (key == "persist") s->use_persist = parse_int(iss, key) != 0;
        else if (key == "tma") s->use_tma = parse_int(iss, key) != 0;
        else if (key == "tma_min_rows") {
            long long v = 0;
            if (!(iss >> v) || v < 1) throw std::invalid_argument("tma_min_rows must be positive");
            s->tma_min_rows = v;
        }
        else if (key == "barrier_polls") {
            int v = 0;
            if (!(iss >> v) || v < 1) throw std::invalid_argument("barrier_polls must be positive");
            s->barrier_polls = v;
        }
        else if (key == "null_space") s->null_space = parse_int(iss, key) != 0;
        else if (key == "correction_interval") {
            int v = 0;
            if (!(iss >> v) || v < 1) throw std::invalid_argument("correction_interval must be positive");
            s->correction_interval = v;
        } else if (key == "tol") {
            double v;
            if (!(iss >> v) || !(v >= 0)) throw std::invalid_argument("tol must be a non-negative number");
            s->tol = v;
        } else if (key.rfind("num_conv", 0) == 0 || key == "num_threads") {
            parse_int(iss, key);   // PSuM tuning keys: accepted and ignored
        }
        // other unknown keys are skipped like PSuM's parser does
    }
    if (!k_provided) s->K = 1;
    if (s->pre_relax < 0 || s->post_relax < 0 || s->max_cycles < 0 || s->depth < 1)
        throw std::invalid_argument("set_options: negative relax/cycle counts or depth < 1");
    s->version++;
    if (s->ready && s->use_persist) s->build_persist(s->own_stream);
}

void solver_set_matrix(SolverBase* s, unsigned long long n_row, unsigned long long n_col, unsigned long long nnz,
                       const unsigned long long* rows, const unsigned long long* cols, const double* vals) {
    if (n_row != n_col) throw std::invalid_argument("set_matrix: matrix must be square");
    HostCSR A = csr_from_coo((long long)n_row, (long long)n_col, (long long)nnz, rows, cols, vals);
    s->host = build_hierarchy(A, s->I, s->J, s->K, s->depth, s->max_coarse, s->periodic, s->null_space != 0);
    s->ns_built = s->null_space != 0;
    s->n_row = n_row;
    ensure_stream(s);
    // created here, outside any stream capture: the stream that captures the
    // body of the conditional refinement loop, and the mapped launch counter
    if (!s->aux_stream) cuda_check(cudaStreamCreateWithFlags(&s->aux_stream, cudaStreamNonBlocking), "cudaStreamCreate");
    device_launch_counter();
    if (!s->stalled) s->stalled = take_host_word();
    s->version++;
    s->drop_graph();
    s->build_device(s->own_stream);
    s->ready = true;
}

static void upload_sources(SolverBase* s) {
    ensure_stream(s);
    s->d_rep_idx.upload(s->rep_idx.data(), s->rep_idx.size(), s->own_stream);
    s->d_rep_val.upload(s->rep_val.data(), s->rep_val.size(), s->own_stream);
    s->d_add_idx.upload(s->add_idx.data(), s->add_idx.size(), s->own_stream);
    s->d_add_val.upload(s->add_val.data(), s->add_val.size(), s->own_stream);
    cuda_check(cudaStreamSynchronize(s->own_stream), "upload sources");
    s->version++;
}

// Graph capture needs a stream that is not the legacy/per-thread default
// stream and is not already being captured by the caller (then the caller's
// capture records the launches directly).
static bool being_captured(cudaStream_t st) {
    if (st == cudaStreamLegacy) return false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cuda_check(cudaStreamIsCapturing(st, &cs), "cudaStreamIsCapturing");
    return cs != cudaStreamCaptureStatusNone;
}
static bool capturable(cudaStream_t st) {
    return st != nullptr && st != cudaStreamLegacy && st != cudaStreamPerThread && !being_captured(st);
}

static void capture_solve(SolverBase* s, double* b, double* x, cudaStream_t st) {
    s->drop_graph();
    const unsigned long long k0 = thread_launches();
    s->loop_kernels = 0;
    cuda_check(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    cudaGraph_t g = nullptr;
    try {
        s->enqueue_solve(b, x, st);
    } catch (...) {
        cudaStreamEndCapture(st, &g);
        if (g) cudaGraphDestroy(g);
        uncount_launches(thread_launches() - k0 - s->loop_kernels);
        throw;
    }
    cuda_check(cudaStreamEndCapture(st, &g), "cudaStreamEndCapture");
    const unsigned long long kernels = thread_launches() - k0 - s->loop_kernels;   // outside loop bodies
    uncount_launches(kernels);   // counted again at every replay
    const cudaError_t e = cudaGraphInstantiate(&s->graph.exec, g, 0);
    cudaGraphDestroy(g);
    cuda_check(e, "cudaGraphInstantiate");
    s->graph.b = b;
    s->graph.x = x;
    s->graph.version = s->version;
    s->graph.kernels = kernels;
}

void solver_set_source(SolverBase* s, bool replace, unsigned long long n, const unsigned long long* idx,
                       const double* v) {
    if (n > 0 && (!idx || !v)) throw std::invalid_argument("set_source: null array");
    if (s->ready)
        for (unsigned long long i = 0; i < n; ++i)
            if (idx[i] >= s->n_row) throw std::invalid_argument("set_source: index out of range");
    if (replace) {
        s->rep_idx.assign(idx, idx + n);
        s->rep_val.assign(v, v + n);
    } else {
        s->add_idx.assign(idx, idx + n);
        s->add_val.assign(v, v + n);
    }
    upload_sources(s);
}

void solver_check_stall(SolverBase* s) {
    if (s->stalled && __atomic_exchange_n(s->stalled, 0, __ATOMIC_ACQ_REL))
        throw Error(PSUM_ERR_INTERNAL, "multigrid: a kernel of this or an earlier solve of the handle stopped waiting "
                                       "(copy or barrier); its result is not a solution");
}

void solver_solve_async(SolverBase* s, double* b, double* x, cudaStream_t stream, long long beside) {
    if (!s->ready) throw Error(PSUM_ERR_NOT_READY, "solve called before set_matrix");
    solver_check_stall(s);
    if (!b || !x) throw std::invalid_argument("solve: null device pointer");
    for (auto i : s->rep_idx)
        if (i >= s->n_row) throw std::invalid_argument("set_source_replace: index out of range");
    for (auto i : s->add_idx)
        if (i >= s->n_row) throw std::invalid_argument("set_source_addback: index out of range");
    cudaStream_t st = stream ? stream : s->own_stream;
    s->beside = beside;
    s->callers_graph = being_captured(st);
    if (s->use_graph && !s->one_kernel() && capturable(st)) {
        if (!(s->graph.exec && s->graph.b == b && s->graph.x == x && s->graph.version == s->version)) {
            const bool whole = s->whole_gpu;
            try {
                capture_solve(s, b, x, st);
            } catch (const Error&) {
                // a graph (or the body of its loop) that may not hold the cooperative kernel: capture without it
                if (!whole || (s->whole_gpu && !s->waits_on_gpu())) throw;
                cudaGetLastError();
                s->whole_gpu = false;
                try {
                    capture_solve(s, b, x, st);
                } catch (...) {   // it failed for another reason
                    s->whole_gpu = whole;
                    throw;
                }
            }
        }
        const Turn turn(st, s->waits_on_gpu());
        cuda_check(cudaGraphLaunch(s->graph.exec, st), "cudaGraphLaunch");
        add_launches(s->graph.kernels);
        return;
    }
    s->enqueue_solve(b, x, st);
}

MGState solver_read_state(SolverBase* s, cudaStream_t stream) {
    MGState st{};
    cuda_check(cudaMemcpyAsync(&st, s->state.p, sizeof(MGState), cudaMemcpyDeviceToHost,
                               stream ? stream : s->own_stream),
               "read state");
    cuda_check(cudaStreamSynchronize(stream ? stream : s->own_stream), "read state sync");
    return st;
}

void solver_destroy(SolverBase* s) {
    if (s->own_stream) cudaStreamSynchronize(s->own_stream);
    s->magic = 0;
    delete s;
}

}  // namespace psum_b200

// ===================================================================== ABI ==
using namespace psum_b200;

namespace {

template <int P>
psum_field_solver_handle ft_init() {
    return create_solver(P);
}

void ft_set_matrix(psum_field_solver_handle h, unsigned long long n_row, unsigned long long n_col,
                   unsigned long long nnz, unsigned long long* rows, unsigned long long* cols, double* vals) {
    solver_set_matrix(solver_from_handle(h), n_row, n_col, nnz, rows, cols, vals);
}

void ft_solve(psum_field_solver_handle h, double* b, double* x) {
    SolverBase* s = solver_from_handle(h);
    solver_solve_async(s, b, x, s->own_stream);
    cuda_check(cudaStreamSynchronize(s->own_stream), "solve sync");
    MGState st = solver_read_state(s, s->own_stream);
    solver_check_stall(s);
    if (st.status == PSUM_ERR_DIVERGED) throw Error(PSUM_ERR_DIVERGED, "multigrid: residual diverged");
}

void ft_set_options(psum_field_solver_handle h, const char* o) { solver_set_options(solver_from_handle(h), o); }

void ft_set_source_replace(psum_field_solver_handle h, unsigned long long n, unsigned long long* idx, double* v) {
    solver_set_source(solver_from_handle(h), true, n, idx, v);
}

void ft_set_source_addback(psum_field_solver_handle h, unsigned long long n, unsigned long long* idx, double* v) {
    solver_set_source(solver_from_handle(h), false, n, idx, v);
}

void ft_free(psum_field_solver_handle h) {
    if (h) solver_destroy(solver_from_handle(h));
}

// Static registration, as the reference backends do (sycl_multigrid32f_gpu.cpp:255-266).
int register_backends() {
    func_table t32{ft_init<32>, ft_set_matrix, ft_solve, ft_set_options, ft_set_source_replace, ft_set_source_addback,
                   ft_free};
    func_table t64{ft_init<64>, ft_set_matrix, ft_solve, ft_set_options, ft_set_source_replace, ft_set_source_addback,
                   ft_free};
    register_solver("cuda_multigrid32f_gpu", t32);
    register_solver("cuda_multigrid64_gpu", t64);
    return 0;
}
const int g_registered = register_backends();

}  // namespace

extern "C" {

EXPORT int psum_mg_create(const char* kind, psum_field_solver_handle* out) {
    return guarded([&] {
        if (!out) throw std::invalid_argument("psum_mg_create: null output");
        *out = nullptr;
        func_table t = get_solver_funcs(kind ? kind : "");
        if (!t.init) throw std::invalid_argument(std::string("unknown solver backend: ") + (kind ? kind : "(null)"));
        *out = t.init();
        if (!*out) throw Error(PSUM_ERR_INTERNAL, "failed to create solver.");
    });
}

EXPORT int psum_mg_set_options(psum_field_solver_handle h, const char* options) {
    return guarded([&] { solver_set_options(solver_from_handle(h), options); });
}

EXPORT int psum_mg_set_matrix(psum_field_solver_handle h, unsigned long long n_row, unsigned long long n_col,
                              unsigned long long nnz, const unsigned long long* rows, const unsigned long long* cols,
                              const double* vals) {
    return guarded([&] { solver_set_matrix(solver_from_handle(h), n_row, n_col, nnz, rows, cols, vals); });
}

EXPORT int psum_mg_set_source_replace(psum_field_solver_handle h, unsigned long long n, const unsigned long long* idx,
                                      const double* values) {
    return guarded([&] { solver_set_source(solver_from_handle(h), true, n, idx, values); });
}

EXPORT int psum_mg_set_source_addback(psum_field_solver_handle h, unsigned long long n, const unsigned long long* idx,
                                      const double* values) {
    return guarded([&] { solver_set_source(solver_from_handle(h), false, n, idx, values); });
}

EXPORT int psum_mg_solve(psum_field_solver_handle h, double* b_dev, double* x_dev) {
    int status = PSUM_OK;
    int rc = guarded([&] {
        SolverBase* s = solver_from_handle(h);
        solver_solve_async(s, b_dev, x_dev, s->own_stream);
        MGState st = solver_read_state(s, s->own_stream);
        solver_check_stall(s);
        status = st.status;
    });
    if (rc != PSUM_OK) return rc;
    if (status == PSUM_ERR_NOT_CONVERGED) set_last_error("multigrid: tol not reached within max_cycles");
    if (status == PSUM_ERR_DIVERGED) set_last_error("multigrid: residual diverged");
    return status;
}

EXPORT int psum_mg_solve_async(psum_field_solver_handle h, double* b_dev, double* x_dev, void* stream) {
    return guarded([&] {
        SolverBase* s = solver_from_handle(h);
        solver_solve_async(s, b_dev, x_dev, static_cast<cudaStream_t>(stream));
    });
}

EXPORT int psum_mg_last_stats(psum_field_solver_handle h, int* cycles, int* refinements, double* rel_residual,
                              double* initial_rel_residual) {
    return guarded([&] {
        SolverBase* s = solver_from_handle(h);
        if (!s->ready) throw Error(PSUM_ERR_NOT_READY, "no solve has run");
        cuda_check(cudaDeviceSynchronize(), "stats sync");
        MGState st = solver_read_state(s, s->own_stream);
        solver_check_stall(s);
        const double bn = st.bnorm2 > 0 ? std::sqrt(st.bnorm2) : 1.0;
        if (cycles) *cycles = st.cycles;
        if (refinements) *refinements = st.refinements;
        auto rel = [&](double r2) { return r2 < 0 ? 0.0 : std::sqrt(r2) / bn; };   // -1: none was taken; NaN stays NaN
        if (rel_residual) *rel_residual = rel(st.rnorm2_last);
        if (initial_rel_residual) *initial_rel_residual = rel(st.rnorm2_first);
    });
}

EXPORT int psum_mg_hierarchy_info(psum_field_solver_handle h, int* levels, unsigned long long* coarse_rows,
                                  unsigned long long* exception_rows_level0) {
    return guarded([&] {
        SolverBase* s = solver_from_handle(h);
        if (!s->ready) throw Error(PSUM_ERR_NOT_READY, "set_matrix has not been called");
        if (levels) *levels = s->levels;
        if (coarse_rows) *coarse_rows = s->coarse_rows;
        if (exception_rows_level0) *exception_rows_level0 = s->host.ahat[0].exc_rows.size();
    });
}

EXPORT int psum_mg_tma_sweeps(psum_field_solver_handle h, int* level_vectors) {
    return guarded([&] {
        SolverBase* s = solver_from_handle(h);
        if (level_vectors) *level_vectors = s->tma_level_vectors();
    });
}

EXPORT int psum_mg_destroy(psum_field_solver_handle h) {
    return guarded([&] {
        if (h) solver_destroy(solver_from_handle(h));
    });
}

}  // extern "C"
