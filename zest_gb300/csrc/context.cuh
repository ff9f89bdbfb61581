// Context and per-order plan structures of the GLQ path, shared by the FP64
// host code (zest_gpu.cu) and the split-precision host code (split.cu).
#pragma once

#include <atomic>

#include <map>
#include <memory>
#include <string>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "split.cuh"
#include "lsq.cuh"

namespace zgpu {

// ---------------------------------------------------------------------------
// Number of device buffers freed so far (process-wide).  A captured CUDA
// graph holds raw device pointers: it may be replayed only while this count is
// what it was at capture, i.e. while no buffer it might use has been freed or
// moved by a reallocation.
inline std::atomic<unsigned long long>& alloc_epoch() {
    static std::atomic<unsigned long long> epoch{0};
    return epoch;
}

struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) {
            cudaFree(p);
            alloc_epoch().fetch_add(1, std::memory_order_relaxed);
        }
        p = nullptr;
        bytes = 0;
    }
    int ensure(size_t n) {
        if (n <= bytes && p) return ZEST_GPU_OK;
        release();
        if (n == 0) n = 16;
        if (cudaMalloc(&p, n) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            return fail(ZEST_GPU_ERR_OOM, "device allocation of " + std::to_string(n) + " bytes failed");
        }
        bytes = n;
        return ZEST_GPU_OK;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

template <class T>
inline int upload(DevBuf& buf, const std::vector<T>& v, cudaStream_t s) {
    ZG_TRY(buf.ensure(v.size() * sizeof(T)));
    if (!v.empty()) ZG_CUDA_TRY(cudaMemcpyAsync(buf.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    ZG_CUDA_TRY(cudaStreamSynchronize(s));  // host vector may die after return
    return ZEST_GPU_OK;
}

// Device buffers of the evaluation at arbitrary points (evaluate.cu).
struct EvalBufs {
    DevBuf z, r, cs, trig;            // points: cos(colat), radii, (cos, sin)(lon), trig table
    DevBuf P, offP, cntP;             // Legendre table at the colatitudes, groups (m, parity)
    DevBuf R, offR, cntR;             // radial table at the radii, groups l
    DevBuf flm, G;                    // radial and Legendre sums
    DevBuf tiles[3];                  // tile lists of the three sums
};

struct FftEntry {
    FftPlan plan;
    DevBuf tab, itab, rows;
};

// Folded Legendre tables (forward: weights * quadrature prefactor folded in;
// backward: 1/2 for m > 0) with their group offsets.
struct LegTables {
    int L = 0, nnodes = 0;  // nnodes = folded node count (ld)
    int j0u = 0, j0d = 0;
    DevBuf Pf, Pb, off;
    std::vector<long long> off_h;
    std::map<int, std::unique_ptr<DevBuf>> cnt;  // per truncation order Lm
};

struct RadTables {
    int L = 0, nr = 0;
    DevBuf Rf, Rb, off;
    std::vector<long long> off_h;
    std::map<int, std::unique_ptr<DevBuf>> cnt;
};

struct ZtPlan {
    ZtShape sh{};
    LegTables leg;
    RadTables rad;
    std::vector<double> lat_nodes, lat_w, rad_nodes, rad_w;  // host copies (r = (1+x)/2)
};

struct StPlan {
    StShape sh{};
    LegTables leg;
};

// The buffers and conventions of a call on a batch of uneven order.
struct RaggedCall {
    double* coeffs = nullptr;
    const double* euler = nullptr;
    double* grids = nullptr;
    int zn = 0, sn = 0, sp = 0, type = 0, precision = 0, slices = 0;
    bool operator==(const RaggedCall& o) const {
        return coeffs == o.coeffs && euler == o.euler && grids == o.grids && zn == o.zn && sn == o.sn && sp == o.sp &&
               type == o.type && precision == o.precision && slices == o.slices;
    }
};

// A recorded CUDA graph, ready to launch.
struct RecordedGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bool launched = false;
    RecordedGraph() = default;
    RecordedGraph(const RecordedGraph&) = delete;
    RecordedGraph& operator=(const RecordedGraph&) = delete;
    ~RecordedGraph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

// A batch of expansions of different orders (rotate, then backward
// transform): its device work lists, the last call, and the CUDA graph that
// replays that call.
struct RaggedPlan {
    std::vector<int> orders;
    RaggedCall call;
    int Lmax = 0;
    DevBuf coff;                                               // per-item coefficient offsets
    DevBuf vecl;                                               // the {item, n, l, first pair} vectors sorted by l
    std::vector<long long> voff;                               // vecl rows of order l: [voff[l], voff[l+1])
    DevBuf voff_dev;
    std::vector<long long> coff_h, goff_h;
    std::vector<std::tuple<int, int, int>> buckets;            // {order, first item, count}
    std::unique_ptr<RecordedGraph> recorded;                   // null where the last call failed
    unsigned long long epoch = 0;                              // alloc_epoch() when it was recorded
};

struct TileEntry {
    DevBuf buf;
    int count = 0;
};

// CUDA-event timing of pipeline stages on the context stream.
struct Profiler {
    bool on = false;
    std::vector<cudaEvent_t> pool;
    std::vector<std::tuple<int, cudaEvent_t, cudaEvent_t>> pending;
    double ms[ST_COUNT] = {};
    long long count[ST_COUNT] = {};
    cudaEvent_t get() {
        if (!pool.empty()) {
            cudaEvent_t e = pool.back();
            pool.pop_back();
            return e;
        }
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        return e;
    }
    ~Profiler() {
        for (auto& t : pending) {
            cudaEventDestroy(std::get<1>(t));
            cudaEventDestroy(std::get<2>(t));
        }
        for (auto e : pool) cudaEventDestroy(e);
    }
};

}  // namespace zgpu

using namespace zgpu;

struct zest_gpu_context {
    int device = 0;
    cudaStream_t stream = nullptr;
    int precision = ZEST_PRECISION_FP64;
    int slices = 6;
    std::map<std::tuple<int, int, int, int>, std::unique_ptr<ZtPlan>> zt_plans;
    std::map<std::tuple<int, int, int, int>, std::unique_ptr<StPlan>> st_plans;
    std::map<int, std::unique_ptr<FftEntry>> ffts;
    std::map<int, std::unique_ptr<DevBuf>> wigner;
    std::map<int, std::unique_ptr<DevBuf>> wigner_fixed;      // the same as limbs (split rotations)
    std::map<std::tuple<int, int>, std::pair<std::unique_ptr<DevBuf>, int>> vec_lists;
    std::map<std::tuple<int, int, int, int, int, int>, std::unique_ptr<TileEntry>> tiles;
    bool autotune = true;                                     // time the tile shapes on first use
    bool defer_finish = false;                                // split calls leave the wait flag to their caller
    size_t host_chunk_bytes = size_t(1) << 28;                // pipelined host calls: input bytes per chunk
    std::unique_ptr<RaggedPlan> ragged;                       // last batch of uneven orders, with its graph
    cudaStream_t graph_stream = nullptr;                      // own stream for graph capture and replay
    cudaStream_t copy_stream[2] = {nullptr, nullptr};         // host->device, device->host of pipelined calls
    cudaEvent_t pipe_ev[3][2] = {};                           // uploaded, computed, downloaded per slot
    cudaEvent_t graph_ev[2] = {nullptr, nullptr};             // ordering with the context stream
    std::map<std::tuple<int, int, int, int>, int> tuned;      // chosen shape per (stage, L, Lm, batch)
    DevBuf s0, s1;          // transform scratch (spectra, flm)
    DevBuf in_stage, out_stage, aux_stage;  // host <-> device staging
    DevBuf phase;           // rotation phases
    DevBuf adj0, adj1, adj2;  // adjoint scratch (scaled operands, inverse angles, angle partials)
    std::map<std::tuple<int, int, int>, std::unique_ptr<DevBuf>> adj_w;  // quadrature weight slabs
    std::unique_ptr<SplitState, SplitDeleter> split;
    EvalBufs eval;          // evaluation at arbitrary points
    std::unique_ptr<LsqState, LsqDeleter> lsq;  // least-squares fits
    Profiler prof;
};

namespace zgpu {
// The plan of the longitude transforms of length N, cached (zest_gpu.cu).
int get_fft(zest_gpu_context* ctx, int N, const FftPlan** out);

// Gives a variable another value for the lifetime of the object, also where an
// exception ends it.
template <class T>
struct ScopedValue {
    T& ref;
    const T before;
    ScopedValue(T& r, T v) : ref(r), before(r) { ref = v; }
    ScopedValue(const ScopedValue&) = delete;
    ScopedValue& operator=(const ScopedValue&) = delete;
    ~ScopedValue() { ref = before; }
};

// Brackets one pipeline stage with events when profiling is on.
struct StageScope {
    zest_gpu_context* ctx;
    int stage;
    cudaStream_t stream;
    cudaEvent_t e0 = nullptr;
    StageScope(zest_gpu_context* c, int st, cudaStream_t s = nullptr) : ctx(c), stage(st), stream(s ? s : c->stream) {
        if (ctx->prof.on) {
            e0 = ctx->prof.get();
            cudaEventRecord(e0, stream);
        }
    }
    ~StageScope() {
        if (e0) {
            cudaEvent_t e1 = ctx->prof.get();
            cudaEventRecord(e1, stream);
            ctx->prof.pending.emplace_back(stage, e0, e1);
        }
    }
};
}  // namespace zgpu


