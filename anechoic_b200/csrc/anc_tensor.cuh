// Batched SCA engine for replicas sharing J (tcgen05 int8 J * dS update); host-facing interface.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "anc_common.cuh"

namespace anc {

// Whether work submitted to the stream is being recorded into a CUDA graph.
inline bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return s != cudaStreamCaptureStatusNone;
}

// What a kernel's set-up returns when it lacks device memory, or would have to allocate during a capture: nothing has been
// enqueued, and an engine that needs no memory of its own can run the call instead.
constexpr int kNoRoom = -4;
inline int setup_code(cudaError_t e) {
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation || e == cudaErrorStreamCaptureUnsupported ? kNoRoom : -2;
}

// A handle's device workspace, which grows with its largest call. A block that a captured launch uses is kept until the handle
// goes, because the graph may be replayed after the workspace has grown; other blocks are freed when they are replaced.
struct Workspace {
    uint8_t* p = nullptr;
    size_t bytes = 0;
    // At least `need` bytes for a launch on st. While st is being captured nothing can be allocated: a call that needs more is
    // refused without ending the capture.
    cudaError_t ensure(size_t need, cudaStream_t st) {
        const bool cap = capturing(st);
        if (bytes < need) {
            if (cap) return cudaErrorStreamCaptureUnsupported;
            if (p && captured) kept.push_back(p);
            else if (p) cudaFree(p);
            p = nullptr;
            bytes = 0;
            captured = false;
            void* q = nullptr;
            const cudaError_t e = cudaMalloc(&q, need);
            if (e != cudaSuccess) return e;
            p = static_cast<uint8_t*>(q);
            bytes = need;
        }
        captured = captured || cap;
        return cudaSuccess;
    }
    void free() {
        if (p) cudaFree(p);
        for (uint8_t* k : kept) cudaFree(k);
        *this = Workspace{};
    }

private:
    bool captured = false;
    std::vector<uint8_t*> kept;
};

struct TensorInstance {
    int n = 0, np = 0;
    int npp = 0;                 // permuted width of J_perm (np, or 256 x the padded rounds for the streaming kernel)
    bool stream = false;         // 32 < NP/256 <= 64: J streamed from HBM (tensor_stream.cu)
    std::vector<int> perm;       // slot i -> permuted index (CTA-contiguous slot slices)
    int8_t* d_J = nullptr;       // J_perm [np][np] int8 (row = y, contiguous x)
    size_t bytes = 0;
    Workspace ws;                // exchange buffers + error word
    int32_t* d_bias_perm = nullptr;
    int* last_err = nullptr;     // error word of the last launch
    int last_ctas = 0, last_cluster = 0;
};

// Slots per CTA of the opt-in phase profile (clock64 totals, see tensor_engine.cu).
constexpr int kTensorProfSlots = 56;

struct TensorRun {
    DevTables tab;
    uint64_t seed;
    uint32_t trial_offset;
    int nchains;
    int32_t hclamp;
    const int32_t* bias;
    uint32_t* out_spins;
    int64_t* out_sum_sh;
    int64_t* out_sum_bs;
    int64_t* out_flips;
    int32_t* out_trace;
    int32_t* out_h;
    long long* prof;          // device [grid][16] phase cycle totals, or null (profiling off)
    uint64_t wait_ns;         // limit of each device wait of the launch (0: give up at the first unsatisfied poll)
    int variant;              // planes kernel at NP = 2048, one plane: its geometry (kF4Variants; 0 = by rule)
};

// Variants of the fp4 kernel (the planes kernel at NP = 2048 with one plane): lanes per decision thread -- variant 0 by the
// number of replica groups, 1 .. 3: 8, 4 or 2.
constexpr int kF4Variants = 4;

// Launch geometry of a run: CTAs in the grid, CTAs per cluster, and how many clusters can be co-resident.
struct TensorGeometry {
    int ctas = 0, cluster = 0, max_active_clusters = 0;
};
int tensor_geometry(int n, int nchains, TensorGeometry* g);

bool tensor_supported(int n, int K, int nchains);
// Anneals one launch of the tensor kernel that runs this instance advances together (more anneals take further waves
// of replica groups inside the launch).
int tensor_wave_chains(int n, int* out);
int tensor_build_instance(const int8_t* J, int n, TensorInstance* out, std::string* why);
int tensor_run(TensorInstance* ti, const TensorRun& r, cudaStream_t st, std::string* why);
// Streaming kernel for NP in (8192, 16384] (tensor_stream.cu): support test, build from the plain engine's bit planes, launch.
bool stream_supported(int n);
// Whether the kernel can run n at all: NP in (4096, 16384] (AUTO uses it below 8193 where no other tensor kernel runs), and the
// measured device time of one step of nchains anneals, in microseconds.
bool stream_runs(int n);
double stream_step_us(int n, int nchains);
int stream_build(const uint32_t* bits, int K, int nwj, int n, TensorInstance* out, cudaStream_t st, std::string* why);
int stream_wave_chains();
int stream_run(TensorInstance* ti, const TensorRun& r, const int32_t* bias_perm, cudaStream_t st, std::string* why);
// Planes kernel (tensor_planes.cu): J on chip as one (|J| <= 4) or two e2m1 planes, NP = 2048 .. 6144 (one plane) or
// 4096 (two).
struct PlanesInstance {
    int n = 0, R = 0, W = 0;
    uint8_t* d_J = nullptr;      // [W][256 RP][128 RP] packed e2m1
    int32_t* d_bias = nullptr;   // bias at permuted column
    Workspace ws;                // error word, flags, exchange buffers
    int* last_err = nullptr;     // error word of the last launch
    int last_ctas = 0;
};
bool planes_supported(int n, int maxabs);
// measured device time of one step of nchains anneals (all waves), in microseconds
double planes_step_us(int n, int maxabs, int nchains, int sms);
// anneals one wave advances at most
int planes_wave_chains(int n, int maxabs);
// upper bound of a launch's CTAs on this device
int planes_max_ctas();
// from the plain engine's bit planes on the device ([K][np][nwj])
int planes_build(const uint32_t* bits, int K, int nwj, int n, const int32_t* bias, int maxabs, PlanesInstance* out,
                 cudaStream_t st, std::string* why);
int planes_run(PlanesInstance* pi, const TensorRun& r, cudaStream_t st, std::string* why);
void planes_free(PlanesInstance* pi);
// After the stream has reached the launch: -3 if a bounded device wait expired, 0 otherwise.
int tensor_check_error(const int* err, cudaStream_t st, std::string* why);
void tensor_free_instance(TensorInstance* ti);

}  // namespace anc
