// Host side of liblexb: the C ABI declared in include/lexb.h over the CUDA runtime.
// It mirrors lex_cuda::device (crates/lex-cuda/src/device.rs): a Gpu that owns a stream,
// Buffers, Pipelines (a planned kernel + launch shape) and Steps, with string errors
// instead of panics.  Kernels are compiled ahead of time for sm_100a and live in this
// library; there is no NVRTC step and no CPU path.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <mutex>
#include <new>
#include <queue>
#include <map>
#include <string>
#include <tuple>
#include <unordered_map>
#include <vector>

#include "../../include/lexb.h"
#include "gemm_fp4_sm100.cuh"
#include "gemm_fp4_sm100_pair.cuh"
#include "gemm_fp4_few_sm100.cuh"
#include "matvec_fp4_sm100.cuh"
#include "matmul_q_fp4_sm100.cuh"
#include "matmul_q_chain_sm100.cuh"

// Scratch of lexb_gemm_fp4_splitk_static: split-K partial products [splits][m][n] f32.  Part of
// the library image, so every GPU that loads the library holds these 32 MiB until the process exits.
static __device__ __align__(256) float g_splitk_static_scratch[LEXB_STATIC_SCRATCH_BYTES / sizeof(float)];

namespace {

thread_local std::string g_last_error;
thread_local bool t_injected = false;     // the failure being reported was made by lexb_debug_fail_next

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
    if (t_injected) g_last_error += " [injected]";
    t_injected = false;
    return code;
}

#define CUDA_TRY(expr)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (expr);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return fail(LEXB_ERR_CUDA, "%s: %s (%s)", #expr, cudaGetErrorString(e_), cudaGetErrorName(e_)); \
    } while (0)

// Host-side failure injection (tests only): lexb_debug_fail_next arms one site; the n-th call that reaches it
// from then on fails with the given CUDA error instead of being made.  It stands where the reference's
// injectable driver table would (the `api!` table, crates/lex-cuda/src/device.rs:88-132); nothing on the
// device is made to fail.
enum { SITE_ALLOC = 1, SITE_COPY = 2, SITE_LAUNCH = 3, SITE_ENCODE = 4, SITE_COUNT = 5 };
struct Injection { int countdown = 0; int error = 0; };
Injection g_inject[SITE_COUNT];
std::mutex g_inject_lock;

cudaError_t take_injected(int site) {
    std::lock_guard<std::mutex> lk(g_inject_lock);
    Injection& in = g_inject[site];
    if (in.countdown > 0 && --in.countdown == 0) {
        t_injected = true;
        return static_cast<cudaError_t>(in.error);
    }
    return cudaSuccess;
}

#define CUDA_TRY_AT(site, expr)                                                                 \
    do {                                                                                        \
        cudaError_t e_ = take_injected(site);                                                   \
        if (e_ == cudaSuccess) e_ = (expr);                                                     \
        if (e_ != cudaSuccess)                                                                  \
            return fail(LEXB_ERR_CUDA, "%s: %s (%s)", #expr, cudaGetErrorString(e_), cudaGetErrorName(e_)); \
    } while (0)
#define LAUNCH_TRY(expr) CUDA_TRY_AT(SITE_LAUNCH, expr)
// in front of a <<<...>>> launch
#define INJECT_LAUNCH()                                                                         \
    do {                                                                                        \
        if (cudaError_t e_ = take_injected(SITE_LAUNCH))                                        \
            return fail(LEXB_ERR_CUDA, "kernel launch: %s (%s)", cudaGetErrorString(e_), cudaGetErrorName(e_)); \
    } while (0)

cudaError_t x_malloc(void** p, size_t bytes) {
    if (cudaError_t e = take_injected(SITE_ALLOC)) { *p = nullptr; return e; }
    return cudaMalloc(p, bytes);
}
template <typename T> cudaError_t x_malloc(T** p, size_t bytes) { return x_malloc(reinterpret_cast<void**>(p), bytes); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// (KERNEL_FEW: what a launch of a pipeline of kernel 1 or 3 may run instead; no selector)
enum { KERNEL_MATVEC = 1, KERNEL_TCGEN05 = 2, KERNEL_TCGEN05_PAIR = 3, KERNEL_MATMUL_Q = 4, KERNEL_FEW = 5 };
thread_local bool t_plan_q16 = false;      // set by lexb_matmul_int8_plan around its call of lexb_gemm_fp4_plan
thread_local float* t_plan_partial = nullptr;      // a split-K workspace to borrow instead of allocating one (run_host_in_parts)

}  // namespace

struct lexb_gpu {
    int device = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;       // own_stream or the caller's
    uint32_t* d_status = nullptr;
    bool pdl = true;                         // programmatic dependent launch of the two-CTA GEMM
    float* static_scratch = nullptr;         // device address of g_splitk_static_scratch on this device, once resolved
    // Job tables of chained runs, kept by content: a decode loop issues the same lists token after token, and a
    // table found here needs no copy in front of its launch (a copy would put the launch behind the whole
    // kernel before it).  A table is never written again once copied.
    // (the jobs, then the table of tiles, which follows from them - their parts of K among them - and the device)
    struct ChainTable { std::vector<lexb::MqChainJob> host; std::vector<lexb::MqChainTile> tiles; uint32_t grid; lexb::MqChainJob* dev; };
    std::unordered_multimap<uint64_t, ChainTable> chain_tables;
    // Digit rows of a run's activations (matmul_q_pieces_kernel's output: [8 m][k / 2] digit rows, [k / 256][2048]
    // scale blocks, [m] magnitudes per activation buffer), one arena per stream: every run on that stream writes its
    // buffers' digit rows into it from the start, in stream order.  An arena that has become too small is replaced by one
    // of at least twice its size and kept until the handle closes (launches in flight may read it).
    struct ChainArena {
        uint8_t* buf = nullptr;
        size_t bytes = 0;
        std::map<std::tuple<size_t, uint32_t, uint32_t>, CUtensorMap> maps;      // of the digit rows at an offset, by tokens and K
    };
    std::map<cudaStream_t, ChainArena> chain_arenas;
    std::vector<uint8_t*> retired_arenas;
    unsigned long long* d_trace = nullptr;   // phase timers of the last two-CTA launch, when tracing is on
    size_t trace_ctas = 0;
    uint32_t trace_toggle = 0;
    cudaDeviceProp prop{};
    EncodeTiledFn encode_tiled = nullptr;
    size_t smem_optin = 0;
    std::mutex held_lock;
    uint32_t held[lexb::FEW_MAX_CLUSTER + 1u] = {};      // clusters of that many blocks the device holds (held_clusters)
    // lexb_gemm_fp4_run_host in parts: one copy stream each way beside the launch stream
    static constexpr uint32_t HOST_PARTS = 4;
    struct HostPath {
        std::mutex lock;
        cudaStream_t in = nullptr, out = nullptr;
        cudaEvent_t event[2u * HOST_PARTS + 2u] = {};
    } host;
};

// (`device`: buffers and pipelines may be freed after their handle was closed, which must not be read then)
struct lexb_buffer {
    lexb_gpu* gpu;
    void* ptr;
    size_t bytes;
    bool owned;
    int device = 0;
};

// How the matvec's launch is laid out (plan_matvec).
struct MatvecShape {
    uint32_t parts = 8;         // parts that K is summed in
    uint32_t cluster = 1;       // blocks that share a row block's K
    uint32_t warps = 8;         // per block
    uint32_t sm_warps = 24;     // warps per SM the registers are cut to (24 or 16)
    uint32_t kc = 0, smem = 0;  // K columns of x staged at a time, shared memory per block
    uint32_t clusters = 0, per = 0;   // clusters (blocks, without clusters) of the launch, groups of row blocks each works through
};

struct lexb_pipeline {
    lexb_gpu* gpu;
    int device = 0;
    uint32_t kernel;
    uint32_t m, n, k;
    bool residual;
    // tcgen05 GEMM
    uint32_t tm, stages, w_stages, tmem_cols, m_tiles, n_acc, flags;
    uint32_t raw_stages = lexb::PAIR_RAW_STAGES;
    uint32_t k_sub = 1;         // two-CTA kernel: K steps per ring stage
    uint32_t x_rows = lexb::PAIR_XBLK_ROWS;     // two-CTA kernel: tokens per CTA and token block (tm / 2 for tiles below 512 tokens)
    uint32_t k_splits = 1, kb_per_split = 0, tok_blocks = 2;
    double us = 1e30;           // ... what the planner expects a launch to take
    bool cluster_split = false; // ... the parts of K summed within a cluster, but for a gather
    uint32_t ws_pitch = 0;      // block-scaled kernel: bytes per row of one scale load
    bool x_f32 = false;         // ... with f32 activations
    bool x_q16 = false;         // ... with int16 activations and one f32 scale per 16 (lexb_matmul_int8_plan): bindings [xq, xs, wq, ...]
    bool w_const = false;       // the caller declared wq/ws constant (LEXB_SCHED_WEIGHTS_CONSTANT): loaded ahead of the stream's order
                                // by the kernels that can (block-scaled kernel, two-CTA GEMM)
    bool w_volatile = false;    // ... or said they may change (LEXB_SCHED_WEIGHTS_MAY_CHANGE): never loaded early, not even in a list
    bool splits_asked = false;  // ... whose K split the caller gave
    bool mq_pre = false;        // ... with the tokens' digit rows from the pieces kernel: buffers and their tensor map
    uint8_t* pre_buf = nullptr; // [8 m][k / 2] digit rows, then [k / 256][2048] scale blocks, then [m] magnitudes
    CUtensorMap pre_map{};
    float* partial = nullptr;   // split-K workspace [k_splits][m][n], owned by the pipeline (a part of run_host's: by the whole's)
    bool partial_borrowed = false;
    // matvec
    MatvecShape mv;
    uint32_t kc;                // ... K columns of x staged at a time
    uint32_t grid, threads, smem;
    char entry[96];
    // tensor maps of x, keyed by the device pointer they were encoded for
    struct MapEntry {
        const void *x, *wq, *ws;
        CUtensorMap map, map_wq, map_ws;
    };
    mutable std::vector<MapEntry> maps;
    mutable std::mutex maps_lock;
    // few tokens: what a launch without a gather runs instead (gemm_fp4_few_kernel)
    lexb_pipeline* few = nullptr;
    uint32_t cluster = 1;
    // lexb_gemm_fp4_run_host in parts: tokens of a part (0: whole), the pipelines of a part and of a shorter last one
    uint32_t host_part = 0;
    mutable lexb_pipeline* host_pipes[2] = {nullptr, nullptr};
    mutable std::mutex host_lock;
};

namespace {

int use(lexb_gpu* g) {
    if (!g) return fail(LEXB_ERR_ARG, "null gpu handle");
    CUDA_TRY(cudaSetDevice(g->device));
    return LEXB_OK;
}

// Device memory of a buffer or a pipeline.  A failure is this call's: it does not stay behind as the next launch's error.
cudaError_t free_on(int device, std::initializer_list<void*> memory) {
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess)
        for (void* p : memory)
            if (cudaError_t f = cudaFree(p)) e = f;
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

int check_buf(const lexb_buffer* b, const lexb_gpu* g, size_t need, const char* what) {
    if (!b) return fail(LEXB_ERR_ARG, "%s: null buffer", what);
    if (b->gpu != g) return fail(LEXB_ERR_ARG, "%s: buffer belongs to another gpu handle", what);
    if (b->bytes < need) return fail(LEXB_ERR_ARG, "%s: buffer holds %zu bytes, the shape needs %zu", what, b->bytes, need);
    if ((reinterpret_cast<uintptr_t>(b->ptr) & 15u) != 0) return fail(LEXB_ERR_ARG, "%s: device pointer is not 16-byte aligned", what);
    return LEXB_OK;
}

uint32_t round_up(uint32_t v, uint32_t to) { return (v + to - 1) / to * to; }

uint32_t env_u32(const char* name, uint32_t dflt) {
    const char* s = getenv(name);
    if (!s || !*s) return dflt;
    return static_cast<uint32_t>(strtoul(s, nullptr, 10));
}

// one-block kernel for lexb_selftest_bounded_wait: a barrier with one expected arrival that
// never comes; the wait gives up after limit_cycles and reports.
__global__ void bounded_wait_selftest_kernel(uint32_t* status, long long limit_cycles) {
    __shared__ __align__(8) uint64_t bar;
    const uint32_t b = lexb::smem_u32(&bar);
    if (threadIdx.x == 0) {
        lexb::mbar_init(b, 1);
        lexb::fence_mbar_init();
        const long long t0 = clock64();
        bool done = false;
        while (!(done = lexb::mbar_try_wait(b, 0))) {
            if (clock64() - t0 > limit_cycles) break;
        }
        if (!done) atomicOr(status, lexb::ST_WAIT_NEVER);
    }
}

// every staged weight as f16 bits: one thread per group of 16
__global__ void dequant_fp4_f16_kernel(uint32_t n, uint32_t k, const uint8_t* __restrict__ wq,
                                       const uint8_t* __restrict__ ws, const float* __restrict__ wg,
                                       uint16_t* __restrict__ out) {
    const uint32_t groups_per_row = k / 16u;
    const size_t total = static_cast<size_t>(n) * groups_per_row;
    for (size_t gi = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; gi < total;
         gi += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const uint32_t row = static_cast<uint32_t>(gi / groups_per_row);
        const uint2 q = *reinterpret_cast<const uint2*>(wq + gi * 8u);
        uint4 lo, hi;
        lexb::decode_group16(q, ws[gi], lexb::make_row_scale(wg[row]), lo, hi);
        uint4* o = reinterpret_cast<uint4*>(out + gi * 16u);
        o[0] = lo;
        o[1] = hi;
    }
}

// a = silu(g) * u = g * (1 / (1 + exp(-g))) * u, evaluated in f32 in that order
// (crates/lex-front/src/llama.rs:879-888, sigmoid as crates/lex-front/src/ir.rs:244), four columns per thread.
template <typename OutT>
__global__ void silu_mul_kernel(uint32_t rows, uint32_t cols, const float* __restrict__ g, size_t g_pitch,
                                const float* __restrict__ u, size_t u_pitch, OutT* __restrict__ out) {
    lexb::allow_dependents();
    lexb::grid_dependency_wait();
    const uint32_t c4 = cols / 4u;
    const size_t total = static_cast<size_t>(rows) * c4;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t r = i / c4, c = (i - r * c4) * 4u;
        const float4 gv = *reinterpret_cast<const float4*>(g + r * g_pitch + c);
        const float4 uv = *reinterpret_cast<const float4*>(u + r * u_pitch + c);
        const float gg[4] = {gv.x, gv.y, gv.z, gv.w}, uu[4] = {uv.x, uv.y, uv.z, uv.w};
        float y[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            y[j] = lexb::silu_mul_f32(gg[j], uu[j]);
        }
        if constexpr (sizeof(OutT) == 4) {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + r * cols + c) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
            uint2 packed;
            packed.x = lexb::pack_f16x2_rn(y[0], y[1]);
            packed.y = lexb::pack_f16x2_rn(y[2], y[3]);
            *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(out) + r * cols + c) = packed;
        }
    }
}

// A launch that may be scheduled while the one ahead drains; the kernel waits for it (grid_dependency_wait) before it
// touches memory.  The two small elementwise kernels cost 3 us each between GEMMs, most of it the gaps on either side.
struct PdlLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    PdlLaunch(lexb_gpu* g, uint32_t blocks, uint32_t threads, bool pdl) {
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(threads);
        cfg.stream = g->stream;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 1 : 0;
    }
};

// lex_msl::int8::quant16 (crates/lex-msl/src/int8.rs:47-114), operation for operation: per group of 16 the largest
// magnitude mx, inv = 32767 / mx (0 for a group of zeros), q = round-to-nearest-even(v * inv) as int16, scale mx / 32767.
template <bool XH>
__global__ void quant16_kernel(const void* __restrict__ x, short* __restrict__ xq, float* __restrict__ xs, size_t groups) {
    lexb::allow_dependents();
    lexb::grid_dependency_wait();
    const size_t g = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
    if (g >= groups) return;
    float v[16];
    if (XH) {
        const uint4* xp = reinterpret_cast<const uint4*>(x) + g * 2u;
        const uint4 raw[2] = {xp[0], xp[1]};
        const __half2* hp = reinterpret_cast<const __half2*>(raw);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 f = __half22float2(hp[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    } else {
        const float4* xp = reinterpret_cast<const float4*>(x) + g * 4u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 f = xp[i];
            v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
    }
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) mx = fmaxf(mx, fabsf(v[i]));
    const float inv = mx > 0.0f ? __fdiv_rn(32767.0f, mx) : 0.0f;
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        w[i] = (static_cast<uint32_t>(__float2int_rn(__fmul_rn(v[2 * i], inv))) & 0xFFFFu) |
               ((static_cast<uint32_t>(__float2int_rn(__fmul_rn(v[2 * i + 1], inv))) & 0xFFFFu) << 16);
    uint4* out = reinterpret_cast<uint4*>(xq) + g * 2u;
    out[0] = make_uint4(w[0], w[1], w[2], w[3]);
    out[1] = make_uint4(w[4], w[5], w[6], w[7]);
    xs[g] = __fdiv_rn(mx, 32767.0f);
}

int encode_2d(const lexb_pipeline* p, CUtensorMap* map, CUtensorMapDataType dt, uint32_t esize, const void* ptr,
              uint64_t inner, uint64_t outer, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swz,
              const char* what) {
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {inner * esize};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    if (cudaError_t ie = take_injected(SITE_ENCODE))
        return fail(LEXB_ERR_CUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)ie);
    CUresult r = p->gpu->encode_tiled(map, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LEXB_ERR_CUDA, "cuTensorMapEncodeTiled(%s) failed with CUresult %d", what, (int)r);
    return LEXB_OK;
}

// Tensor maps for one binding, cached by the device pointers they were encoded for.
int get_maps(const lexb_pipeline* p, const void* x, const void* wq, const void* ws, lexb_pipeline::MapEntry* out) {
    std::lock_guard<std::mutex> lk(p->maps_lock);
    const bool pair = p->kernel == KERNEL_TCGEN05_PAIR || p->kernel == KERNEL_MATMUL_Q || p->kernel == KERNEL_FEW;
    for (const auto& e : p->maps)
        if (e.x == x && (!pair || (e.wq == wq && e.ws == ws))) {
            *out = e;
            return LEXB_OK;
        }
    lexb_pipeline::MapEntry e{};
    e.x = x; e.wq = wq; e.ws = ws;
    int rc;
    // x f16[m, k] row-major; box = 64 columns (128 bytes, the swizzle span) x the tile's tokens, never
    // taller than the tensor.  Rows past m are filled with zeros by the copy engine.
    const uint32_t box_rows = pair ? (p->m < p->x_rows ? p->m : p->x_rows) : (p->tm < p->m ? p->tm : p->m);
    if (p->kernel != KERNEL_MATMUL_Q &&      // that kernel reads x with plain loads
        (rc = encode_2d(p, &e.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, p->k, p->m, lexb::GEMM_BK, box_rows,
                        CU_TENSOR_MAP_SWIZZLE_128B, "x")))
        return rc;
    if (pair) {
        // wq u8[n, k/2]: 128 rows x 128 bytes (256 columns of K), swizzled; ws u8[n, k/16]: 128 rows x 16 bytes
        if ((rc = encode_2d(p, &e.map_wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, p->k / 2, p->n, lexb::PAIR_RAW_K / 2,
                            lexb::GEMM_TN, CU_TENSOR_MAP_SWIZZLE_128B, "wq")))
            return rc;
        const uint32_t ws_box = p->kernel == KERNEL_MATMUL_Q ? p->ws_pitch : lexb::PAIR_RAW_K / 16;
        if ((rc = encode_2d(p, &e.map_ws, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ws, p->k / 16, p->n, ws_box,
                            lexb::GEMM_TN, CU_TENSOR_MAP_SWIZZLE_NONE, "ws")))
            return rc;
    }
    if (p->maps.size() >= 64) p->maps.erase(p->maps.begin());
    p->maps.push_back(e);
    *out = e;
    return LEXB_OK;
}

// The weights of the launch that follows in a step list: a hint for the block-scaled kernel, which pulls
// their first stages into L2 before it ends.
struct NextWeights {
    const lexb_pipeline* pipe;
    const lexb_buffer *x, *wq, *ws;
};

// How a launch sits in its stream.  `early_weights`: the block-scaled kernel may load wq/ws before the launch ahead of
// it has finished (the caller declared them constant, or the step list shows that nothing in flight writes them).
// `fence`: launched without programmatic stream serialization, so that it starts only when everything ahead of it
// in the stream is done - the first launch of a step list, behind which the list's own launches overlap one another only.
// `in_order`: launched with it, but every read waits for the launches ahead, that of weights declared constant too.
struct Order {
    bool early_weights = false;
    bool fence = false;
    bool in_order = false;
    bool early(const lexb_pipeline* p) const { return !in_order && (p->w_const || (early_weights && !p->w_volatile)); }
};

using PairKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const lexb::GemmArgs);
template <bool TRACE>
PairKernel pair_kernel(bool paired, bool cluster) {
    return paired ? (cluster ? lexb::gemm_fp4_tcgen05_pair_split_kernel<TRACE, true> : lexb::gemm_fp4_tcgen05_pair_kernel<TRACE, true>)
                  : (cluster ? lexb::gemm_fp4_tcgen05_pair_split_kernel<TRACE, false> : lexb::gemm_fp4_tcgen05_pair_kernel<TRACE, false>);
}

using FewKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const lexb::FewArgs);
FewKernel few_kernel(uint32_t m) {
    const uint32_t cols = lexb::few_cols(m);
    return cols == 16u ? lexb::gemm_fp4_few_kernel<16> : cols == 32u ? lexb::gemm_fp4_few_kernel<32> : lexb::gemm_fp4_few_kernel<64>;
}

using PiecesKernel = void (*)(const lexb::MqPiecesList, uint32_t);
PiecesKernel pieces_kernel(int xmode) {
    return xmode == 2 ? lexb::matmul_q_pieces_kernel<2> : xmode == 1 ? lexb::matmul_q_pieces_kernel<1> : lexb::matmul_q_pieces_kernel<0>;
}

using MatvecKernel = void (*)(const lexb::MatvecArgs);
MatvecKernel matvec_kernel(uint32_t m, uint32_t k, uint32_t sm_warps) {
    const bool ragged = k % lexb::MV_SLICE != 0u;
    if (m > 8u) return ragged ? lexb::matvec_fp4_kernel<true, true, 24> : lexb::matvec_fp4_kernel<true, false, 24>;
    if (sm_warps == 16u) return ragged ? lexb::matvec_fp4_kernel<false, true, 16> : lexb::matvec_fp4_kernel<false, false, 16>;
    return ragged ? lexb::matvec_fp4_kernel<false, true, 24> : lexb::matvec_fp4_kernel<false, false, 24>;
}
// Clusters of c blocks that the device holds at once: fewer than its SMs' blocks / c, because a cluster stays within one
// part of the chip (at two blocks an SM about 30 clusters of 8, not 37).
uint32_t matvec_clusters(MatvecKernel kernel, uint32_t c, uint32_t threads, uint32_t smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return static_cast<uint32_t>(clusters);
}

// The matvec's launch.  K is summed in 8 parts (4, 2 or 1 if it has no more slices; a row's result depends on k alone), held
// by one block or by a cluster of 2, 4 or 8; blocks have 8 warps or 4, and as many row blocks at a time as their warps
// hold all of their parts.  A cluster divides the staged x, so that a long k at several tokens still leaves room for enough
// warps per SM (m = 4, k = 17408: 157 KB of x in one block, 20 KB each in eight); it costs a barrier across the cluster.
// A short k puts several row blocks in a block, which leaves SMs idle where there are few of them: hence blocks of 4 warps.
//
// Every form is priced in us, with figures fitted to 12,600 launches on a B200 (m = 1-16, n = 128-28672, k = 64-17408, back to
// back on one stream; the form chosen takes 1.3 % more than the fastest in the mean, 8 % at the 95th percentile): the slices of the
// fullest SM at its rate, or a warp's own chain of them, the first three of which are in flight together (`three`, then
// `slice`); per group of row blocks `group` for its sums and `output` per turn of the threads over its outputs; `cluster`
// and `cluster_group` for the barriers; x from the L2; a chunked x per wave of blocks.  `uneven`: where more blocks fit an
// SM than its even share, the fullest one gets more.
template <typename Held>
bool plan_matvec(uint32_t m, uint32_t n, uint32_t k, uint32_t kc_asked, uint32_t sms, size_t smem_optin, size_t smem_sm, Held held, MatvecShape* out) {
    struct Price { double rate24, rate16, three, slice, group, output, cluster, cluster_group, x, chunk, uneven; };
    static const Price UP_TO_8 = {0.053, 0.044, 0.50, 0.45, 0.13, 0.22, 2.1, 1.1, 6.2e-5, 2.1, 0.58},
                       PAST_8 = {0.043, 0.043, 0.017, 0.71, 0.23, 0.45, 2.4, 2.3, 7.5e-5, 1.8, 0.98};
    const bool ring = m <= 8u;
    const Price& f = ring ? UP_TO_8 : PAST_8;
    const uint32_t row_blocks = n / lexb::MV_ROWS, slices = (k + lexb::MV_SLICE - 1u) / lexb::MV_SLICE;
    uint32_t parts = lexb::MV_PARTS;
    while (parts / 2u >= slices) parts /= 2u;                            // (a short k leaves no warp without a slice)
    const uint32_t part_slices = (slices + parts - 1u) / parts;
    double best = 1e30;
    for (uint32_t c = 1; c <= parts; c *= 2u) {
        const uint32_t pp = parts / c;
        for (uint32_t warps = 8; warps >= 4u && warps >= pp; warps /= 2u) {
            for (uint32_t sm_warps = 24; sm_warps >= (ring ? 16u : 24u); sm_warps -= 8u) {
                uint32_t kc = kc_asked;
                if (!kc) {
                    // the whole of K if a block's share of x fits in 96 KiB of shared memory (blocks are then persistent
                    // and stage x once), else the largest multiple of 1024 columns that does
                    const uint32_t budget = 98304u;
                    kc = round_up(k, lexb::MV_SLICE * parts);
                    while (kc > lexb::MV_ROUND && m * lexb::matvec_x_pitch(kc / c) > budget) kc -= lexb::MV_ROUND;
                }
                const uint32_t smem = lexb::matvec_smem_bytes(m, kc, warps, c, ring);
                if (smem > smem_optin) continue;
                const uint32_t per_sm = std::min(static_cast<uint32_t>(smem_sm / (smem + 1024u)), sm_warps / warps);
                const uint32_t at_once = warps / pp, groups = (row_blocks + at_once - 1u) / at_once;      // row blocks a cluster works on at once: a group
                MatvecShape v{parts, c, warps, sm_warps, kc, smem, 0, 0};
                auto price = [&](uint32_t resident) {
                    const uint32_t most = std::max(1u, std::min(groups, resident));
                    v.per = kc < k ? 1u : (groups + most - 1u) / most;
                    v.clusters = (groups + v.per - 1u) / v.per;
                    const uint32_t blocks = v.clusters * c;
                    double deep = (blocks + sms - 1u) / sms;                              // blocks of the fullest SM
                    const double crowd = std::min<double>(per_sm, 2.0 * deep);
                    if (crowd > deep) deep += f.uneven * (crowd - deep);
                    const double chain = v.per * part_slices, busy = (sm_warps == 24u ? f.rate24 : f.rate16) * deep * warps * chain;
                    const double alone = f.three * std::min(chain, 3.0) + f.slice * std::max(chain - 3.0, 0.0);
                    return std::cbrt(busy * busy * busy + alone * alone * alone) + v.per * (f.group + f.output * ((m * at_once + 8u * warps - 1u) / (8u * warps))) +
                           (c > 1u ? f.cluster + f.cluster_group * v.per : 0.0) + f.x * deep * m * k / c +
                           (kc < k ? f.chunk * ((blocks + sms * per_sm - 1u) / (sms * per_sm)) : 0.0);
                };
                const uint32_t room = sms * per_sm / c;
                double us = price(room);
                if (us < best && c > 1u) {                               // (the device holds fewer clusters than its blocks make up)
                    const uint32_t fit = held(c, warps, sm_warps, smem);
                    us = fit ? price(std::min(room, fit)) : 1e30;
                }
                if (us < best) {
                    best = us;
                    *out = v;
                }
            }
        }
    }
    return best != 1e30;
}

// Clusters of c blocks that the device holds at once with one block an SM, asked for once per handle.
uint32_t held_clusters(lexb_gpu* g, uint32_t c) {
    const uint32_t sms = static_cast<uint32_t>(g->prop.multiProcessorCount);
    if (c == 1u) return sms;
    std::lock_guard<std::mutex> lk(g->held_lock);
    uint32_t& held = g->held[c];
    if (!held) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(lexb::FEW_THREADS);
        cfg.dynamicSmemBytes = static_cast<unsigned>(g->smem_optin);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = c;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, lexb::gemm_fp4_few_kernel<16>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        held = clusters > 0 ? std::min(static_cast<uint32_t>(clusters), sms / c) : ~0u;
    }
    return held == ~0u ? 0u : held;
}

// What a launch of the two-CTA GEMM takes, us: `start`; per wave of tiles `wave` for a block's start and its store and `kstep` per K
// step, for tiles of 512 / 256 / 128 / 64 tokens; `store` per MB of y; with K in parts, per MB of partial products and once,
// `reduce` by the second launch, `cluster` in clusters.  At least `least` blocks of 256 columns in a part.
struct PairPrices {
    double start, kstep[4], wave[4], store, reduce, reduce_mb, cluster, cluster_mb;
    uint32_t least;
};
// Fitted to 4,466 launches of 487 shapes (m = 9-2048, n = 128-28672, k = 256-17408) on a B200, before tiles of 128 and 64 tokens were
// decoded two K steps a turn: rms error 5 % then, the form chosen 0.8 % above the fastest in the mean (the prices before, 159 launches
// with the table decode: 9 %).  A K step of those tiles now takes 0.23 us (17408 x 5120, m = 128: 23.3 us), not the 0.319 here, so they
// and their splits are priced too dear against tiles of 256 tokens and the few-token kernel; not fitted again.  Past 10 GFLOP of more
// than 64 tokens the prices of the table decode: a launch that is repeated runs into the power cap, which bursts do not show; the line
// rests on one shape (1572 x 6656 x 1024 with down behind it: 62.4 us by them, 64.6 by FITTED), and plans jump across it.
const PairPrices& pair_prices(uint32_t m, uint32_t n, uint32_t k) {
    static const PairPrices FITTED = {0.20, {0.598, 0.337, 0.319, 0.319}, {7.69, 5.85, 4.46, 3.70}, 0.157, 1.04, 0.288, 0.25, 0.271, 2u},
                            LARGE = {4.51, {0.559, 0.311, 0.310, 0.304}, {8.05, 5.32, 4.02, 4.14}, 0.0, -1.12, 0.300, -1.12, 0.300, 4u};
    return m <= 64u || 2.0 * m * n * k < 1e10 ? FITTED : LARGE;
}

// The few-token kernel's launch for a pipeline, if it takes the shape.
int plan_few(lexb_gpu* g, lexb_pipeline* p) {
    const uint32_t m = p->m, n = p->n, k = p->k;
    if (p->kernel != KERNEL_TCGEN05_PAIR && !env_u32("LEXB_FEW_C", 0)) return LEXB_OK;      // (the matvec keeps m <= 8)
    if (m > lexb::FEW_MAX_TOKENS || n % lexb::FEW_ROWS || k % lexb::FEW_K) return LEXB_OK;
    const uint32_t tiles = n / lexb::FEW_ROWS, U = k / lexb::FEW_K;
    // Fitted to 694 shapes (m = 9-64, clusters of 1, 2, 3, 4, 6 and 8; rms error 6.5 %, the cluster chosen takes 0.7 % more than the
    // fastest in the mean), us: 2.95, 1.04 to 1.07 per block of weights of the longest share, the cluster's barriers and sums, the
    // segments' stores, y.
    const uint32_t forced = env_u32("LEXB_FEW_C", 0);
    uint32_t best_c = 0, best_clusters = 0;
    double best = forced ? 1e30 : p->us;
    for (uint32_t c = 1; c <= lexb::FEW_MAX_CLUSTER; c++) {
        if (forced ? c != forced : c == 5u || c == 7u) continue;
        const uint32_t clusters = std::min(held_clusters(g, c), tiles);
        if (!clusters || (tiles / clusters) * U < c) continue;
        const uint32_t blocks = ((tiles + clusters - 1u) / clusters * U + c - 1u) / c, segments = (blocks + U - 1u) / U;
        const double us = 2.95 + blocks * (m <= 16u ? 1.039 : m <= 32u ? 1.045 : 1.07) + (c > 1u ? 1.76 + 0.0111 * m : 0.0) + 0.0085 * segments * m +
                          0.376e-5 * m * n;
        if (us < best) {
            best = us;
            best_c = c;
            best_clusters = clusters;
        }
    }
    if (!best_c) return LEXB_OK;
    lexb_pipeline* f = new (std::nothrow) lexb_pipeline();
    if (!f) return fail(LEXB_ERR_ARG, "out of host memory");
    f->gpu = g;
    f->kernel = KERNEL_FEW;
    f->m = m; f->n = n; f->k = k; f->tm = m;
    f->residual = p->residual; f->w_const = p->w_const; f->w_volatile = p->w_volatile;
    f->cluster = best_c; f->grid = best_c * best_clusters; f->threads = lexb::FEW_THREADS;
    f->stages = env_u32("LEXB_FEW_SX", m <= 32u ? 4u : 3u); f->raw_stages = std::max(4u, env_u32("LEXB_FEW_SR", m <= 32u ? 5u : 4u));      // (four at least: see the decode)
    f->smem = lexb::few_smem_bytes(m, f->stages, f->raw_stages);
    if (f->smem > g->smem_optin) { delete f; return LEXB_OK; }
    p->few = f;
    return LEXB_OK;
}

int launch_one(lexb_gpu* g, const lexb_pipeline* p, const lexb_buffer* x, const lexb_buffer* wq, const lexb_buffer* ws,
               const lexb_buffer* wg, const lexb_buffer* r, lexb_buffer* y, const lexb::GatherDst* gather = nullptr,
               const NextWeights* next = nullptr, Order order = Order{}, lexb_buffer* act = nullptr,
               const lexb_buffer* xs_q16 = nullptr) {
    const bool pdl = g->pdl && !order.fence;
    // gate/up fused: `act` (or a gather whose destination buffers are f16 activations) replaces y
    const bool silu = act != nullptr || (gather && gather->silu);
    if (!p) return fail(LEXB_ERR_ARG, "null pipeline");
    if (p->gpu != g) return fail(LEXB_ERR_ARG, "pipeline was planned on another gpu handle");
    const bool fuses_silu = p->kernel == KERNEL_TCGEN05_PAIR && !p->residual;
    if (p->few && !gather && !(g->d_trace && p->grid <= g->trace_ctas)) p = p->few;      // (it has no phase timers)
    const size_t m = p->m, n = p->n, k = p->k;
    int rc;
    if ((rc = check_buf(x, g, m * k * (p->x_f32 ? 4 : 2), p->x_q16 ? "xq" : "x"))) return rc;
    if (p->x_q16) {
        if ((rc = check_buf(xs_q16, g, m * (k / 16) * 4, "xs"))) return rc;
    } else if (xs_q16) {
        return fail(LEXB_ERR_ARG, "an activation-scale buffer was bound to a pipeline that takes f16 or f32 activations");
    }
    if ((rc = check_buf(wq, g, n * k / 2, "wq"))) return rc;
    if ((rc = check_buf(ws, g, n * k / 16, "ws"))) return rc;
    if ((rc = check_buf(wg, g, n * 4, "wg"))) return rc;
    if (silu) {
        if (!fuses_silu)
            return fail(LEXB_ERR_UNSUPPORTED, "silu(gate) * up is fused into the two-CTA GEMM only (m > 8, n %% 128 == 0, k %% 256 == 0, no residual)");
        if (act && (rc = check_buf(act, g, m * (n / 2) * 2, "act"))) return rc;
    } else if (!gather && (rc = check_buf(y, g, m * n * 4, "y"))) return rc;
    if (gather && p->kernel != KERNEL_TCGEN05_PAIR)
        return fail(LEXB_ERR_UNSUPPORTED, "the fused all-gather exists in the two-CTA GEMM only (m > 16, n %% 128 == 0, k %% 256 == 0)");
    if (p->residual) {
        if ((rc = check_buf(r, g, m * n * 4, "r"))) return rc;
    } else if (r) {
        return fail(LEXB_ERR_ARG, "a residual buffer was bound to a pipeline planned without one");
    }
    if (p->kernel == KERNEL_TCGEN05 || p->kernel == KERNEL_TCGEN05_PAIR) {
        lexb_pipeline::MapEntry maps;
        if ((rc = get_maps(p, x->ptr, wq->ptr, ws->ptr, &maps))) return rc;
        lexb::GemmArgs a{};
        a.wq = static_cast<const uint8_t*>(wq->ptr);
        a.ws = static_cast<const uint8_t*>(ws->ptr);
        a.wg = static_cast<const float*>(wg->ptr);
        a.r = r ? static_cast<const float*>(r->ptr) : nullptr;
        a.y = y ? static_cast<float*>(y->ptr) : nullptr;
        a.act = act ? static_cast<uint16_t*>(act->ptr) : nullptr;
        a.silu_gather = (gather && gather->silu) ? 1u : 0u;
        lexb::GatherDst gd{};
        if (gather) {
            gd = *gather;
            for (uint32_t d = 0; d < gd.world; d++) a.gather_y[d] = gd.y[d];
            a.gather_world = gd.world; a.gather_n = gd.n_total; a.gather_n0 = gd.n0;
        }
        a.status = g->d_status;
        a.trace = (g->d_trace && p->kernel == KERNEL_TCGEN05_PAIR && p->grid <= g->trace_ctas) ? g->d_trace : nullptr;
        // with room for two launches the records alternate between the two halves, so that two launches in a row
        // can be read side by side (the gap between them on the GPU's global timer)
        if (a.trace && 2u * p->grid <= g->trace_ctas) a.trace += 16ull * p->grid * (g->trace_toggle++ & 1u);
        a.m = p->m; a.n = p->n; a.k = p->k;
        a.tm = p->tm; a.stages = p->stages; a.w_stages = p->w_stages; a.raw_stages = p->raw_stages; a.k_sub = p->k_sub; a.x_rows = p->x_rows;
        // bit 0: operand-collector hint; bit 1 (two-CTA kernel): the packed weights are constant - declared, or
        // proven from the step list - so their copy and decode may run ahead of the stream's order
        a.flags = p->flags | (order.early(p) ? 2u : 0u);
        a.k_splits = p->k_splits; a.kb_per_split = p->kb_per_split; a.partial = p->partial; a.tok_blocks = p->tok_blocks;
        a.tmem_cols = p->tmem_cols; a.m_tiles = p->m_tiles; a.n_acc = p->n_acc;
        a.x_tx_bytes = p->kernel == KERNEL_TCGEN05_PAIR ? (p->m < p->x_rows ? p->m : p->x_rows) * 128u
                                                        : (p->tm < p->m ? p->tm : p->m) * 128u;
        if (p->kernel == KERNEL_TCGEN05_PAIR) {
            // Programmatic dependent launch: this kernel's blocks may be scheduled while the previous
            // launch of the stream drains (they wait for it before touching global memory), which
            // hides most of the gap between two launches.  LEXB_PDL=0 turns it off.
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(p->grid);
            cfg.blockDim = dim3(p->threads);
            cfg.dynamicSmemBytes = p->smem;
            cfg.stream = g->stream;
            const bool in_cluster = p->cluster_split && !gather;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            attr[1].id = cudaLaunchAttributeClusterDimension;
            attr[1].val.clusterDim.x = 2u * p->k_splits;
            attr[1].val.clusterDim.y = 1;
            attr[1].val.clusterDim.z = 1;
            cfg.attrs = pdl ? attr : attr + 1;
            cfg.numAttrs = (pdl ? 1u : 0u) + (in_cluster ? 1u : 0u);
            const bool paired = lexb::pair_paired(p->k_sub, (p->flags & 4u) != 0u, p->w_stages, p->raw_stages);
            const PairKernel kernel = a.trace ? pair_kernel<true>(paired, in_cluster) : pair_kernel<false>(paired, in_cluster);
            LAUNCH_TRY(cudaLaunchKernelEx(&cfg, kernel, maps.map, maps.map_wq, maps.map_ws, a));
            if (p->k_splits > 1 && !in_cluster) {
                CUDA_TRY(cudaGetLastError());
                const size_t elems = static_cast<size_t>(p->m) * p->n;       // n % 128 == 0: a multiple of 4
                const uint32_t blocks = static_cast<uint32_t>(std::min<size_t>((elems / 4 + 255) / 256, static_cast<size_t>(g->prop.multiProcessorCount) * 8u));
                cudaLaunchConfig_t rc_cfg{};
                rc_cfg.gridDim = dim3(blocks);
                rc_cfg.blockDim = dim3(256);
                rc_cfg.stream = g->stream;
                rc_cfg.attrs = attr;
                rc_cfg.numAttrs = g->pdl ? 1 : 0;
                const auto reduce = p->k_splits == 2u ? lexb::splitk_reduce_kernel<2> : p->k_splits == 3u ? lexb::splitk_reduce_kernel<3> : p->k_splits == 4u ? lexb::splitk_reduce_kernel<4> : lexb::splitk_reduce_kernel<0>;
                LAUNCH_TRY(cudaLaunchKernelEx(&rc_cfg, reduce, static_cast<const float*>(p->partial), p->k_splits, elems,
                                            a.r, a.y, gd, a.act, p->n));
            }
        } else {
            PdlLaunch launch(g, p->grid, p->threads, pdl);
            launch.cfg.dynamicSmemBytes = p->smem;
            LAUNCH_TRY(cudaLaunchKernelEx(&launch.cfg, lexb::gemm_fp4_tcgen05_kernel, maps.map, a));
        }
    } else if (p->kernel == KERNEL_FEW) {
        lexb_pipeline::MapEntry maps;
        if ((rc = get_maps(p, x->ptr, wq->ptr, ws->ptr, &maps))) return rc;
        lexb::FewArgs a{};
        a.wg = static_cast<const float*>(wg->ptr);
        a.r = r ? static_cast<const float*>(r->ptr) : nullptr;
        a.y = y ? static_cast<float*>(y->ptr) : nullptr;
        a.act = act ? static_cast<uint16_t*>(act->ptr) : nullptr;
        a.status = g->d_status;
        a.m = p->m; a.n = p->n; a.k = p->k;
        a.cluster = p->cluster; a.x_stages = p->stages; a.raw_stages = p->raw_stages;
        a.flags = order.early(p) ? 2u : 0u;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(p->grid);
        cfg.blockDim = dim3(p->threads);
        cfg.dynamicSmemBytes = p->smem;
        cfg.stream = g->stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = p->cluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 2 : 1;
        LAUNCH_TRY(cudaLaunchKernelEx(&cfg, few_kernel(p->m), maps.map, maps.map_wq, maps.map_ws, a));
    } else if (p->kernel == KERNEL_MATMUL_Q) {
        lexb_pipeline::MapEntry maps;
        if ((rc = get_maps(p, x->ptr, wq->ptr, ws->ptr, &maps))) return rc;
        lexb::MatmulQArgs a{};
        a.x = x->ptr;
        a.xs = xs_q16 ? static_cast<const float*>(xs_q16->ptr) : nullptr;
        a.wg = static_cast<const float*>(wg->ptr);
        a.r = r ? static_cast<const float*>(r->ptr) : nullptr;
        a.y = static_cast<float*>(y->ptr);
        a.partial = p->partial;
        // the row tiles' arrival counters sit behind the partial products in the same allocation
        a.counters = p->partial ? reinterpret_cast<uint32_t*>(p->partial + static_cast<size_t>(p->k_splits) * p->m * p->n) : nullptr;
        a.status = g->d_status;
        a.m = p->m; a.n = p->n; a.k = p->k; a.stages = p->stages;
        a.k_splits = p->k_splits; a.kb_per_split = p->kb_per_split;
        a.ws_pitch = p->ws_pitch;
        // a step on its own: the pieces kernel can be what it waits behind, and the weights are loaded beside that kernel
        const uint32_t pieces_fence = p->mq_pre && order.in_order ? 1u : 0u;
        a.flags = (order.early(p) || (pieces_fence && !p->w_volatile) ? 1u : 0u) | (p->cluster > 1u ? 2u : 0u);
        lexb_pipeline::MapEntry nmaps = maps;         // placeholders when there is no hint (next_grid = 0)
        if (next && next->pipe && next->pipe->kernel == KERNEL_MATMUL_Q && next->pipe->gpu == g && next->wq && next->ws &&
            next->x && (a.flags & 1u) && get_maps(next->pipe, next->x->ptr, next->wq->ptr, next->ws->ptr, &nmaps) == LEXB_OK) {
            const lexb_pipeline* q = next->pipe;
            a.next_grid = q->grid; a.next_k_splits = q->k_splits; a.next_kb_per_split = q->kb_per_split;
            a.next_kb_all = q->k / lexb::MQ_STAGE_K; a.next_stages = q->stages; a.next_ws_pitch = q->ws_pitch;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(p->grid);
        cfg.blockDim = dim3(p->threads);
        cfg.dynamicSmemBytes = p->smem;
        cfg.stream = g->stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = p->cluster;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        const bool serial = !(g->pdl && (!order.fence || p->mq_pre));        // (behind the pieces kernel, that one is the fence)
        cfg.attrs = serial ? attr + 1 : attr;
        cfg.numAttrs = serial ? 1 : 2;
        a.trace = (g->d_trace && p->grid <= g->trace_ctas) ? g->d_trace : nullptr;
        const size_t pieces_bytes = lexb::matmul_q_pieces_bytes(p->m, p->k), sfb_bytes = lexb::matmul_q_sfb_total(p->m, p->k);
        if (p->mq_pre) {
            a.pre_sfb = p->pre_buf + pieces_bytes;
            a.pre_amax = reinterpret_cast<const uint32_t*>(p->pre_buf + pieces_bytes + sfb_bytes);
            cudaLaunchConfig_t pc{};
            pc.gridDim = dim3(p->m, (p->k / lexb::MQ_STAGE_K + 31u) / 32u);      // a warp per stage
            pc.blockDim = dim3(1024);
            pc.stream = g->stream;
            pc.attrs = attr;
            pc.numAttrs = pdl ? 1 : 0;
            lexb::MqPiecesList list{};
            list.job[0] = lexb::MqPiecesJob{x->ptr, a.xs, p->pre_buf, p->k};
            LAUNCH_TRY(cudaLaunchKernelEx(&pc, pieces_kernel(p->x_q16 ? 2 : p->x_f32 ? 1 : 0), list, pieces_fence));
        }
        const CUtensorMap& bmap = p->mq_pre ? p->pre_map : maps.map_wq;      // a placeholder without the pieces kernel
#define LEXB_MQ_LAUNCH(TR, XF, PR) LAUNCH_TRY(cudaLaunchKernelEx(&cfg, lexb::matmul_q_fp4_kernel<TR, XF, PR>, maps.map_wq, maps.map_ws, nmaps.map_wq, nmaps.map_ws, bmap, a))
        if (p->mq_pre) {
            if (p->x_f32) { if (a.trace) LEXB_MQ_LAUNCH(true, 1, true); else LEXB_MQ_LAUNCH(false, 1, true); }
            else { if (a.trace) LEXB_MQ_LAUNCH(true, 0, true); else LEXB_MQ_LAUNCH(false, 0, true); }
        } else {
            if (p->x_q16) { if (a.trace) LEXB_MQ_LAUNCH(true, 2, false); else LEXB_MQ_LAUNCH(false, 2, false); }
            else if (p->x_f32) { if (a.trace) LEXB_MQ_LAUNCH(true, 1, false); else LEXB_MQ_LAUNCH(false, 1, false); }
            else { if (a.trace) LEXB_MQ_LAUNCH(true, 0, false); else LEXB_MQ_LAUNCH(false, 0, false); }
        }
#undef LEXB_MQ_LAUNCH
    } else {
        lexb::MatvecArgs a{};
        a.x = static_cast<const __half*>(x->ptr);
        a.wq = static_cast<const uint8_t*>(wq->ptr);
        a.ws = static_cast<const uint8_t*>(ws->ptr);
        a.wg = static_cast<const float*>(wg->ptr);
        a.r = r ? static_cast<const float*>(r->ptr) : nullptr;
        a.y = static_cast<float*>(y->ptr);
        a.m = p->m; a.n = p->n; a.k = p->k; a.kc = p->kc;
        auto log2u = [](uint32_t v) { uint32_t l = 0; while (v >>= 1) l++; return l; };
        a.log_cluster = log2u(p->mv.cluster);
        a.log_parts = log2u(p->mv.parts);
        a.log_group = log2u(p->mv.warps * p->mv.cluster / p->mv.parts);
        a.log_tokens = log2u(std::min(p->mv.warps, 2u * p->m - 1u));
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(p->grid);
        cfg.blockDim = dim3(p->threads);
        cfg.dynamicSmemBytes = p->smem;
        cfg.stream = g->stream;
        cudaLaunchAttribute attr[2];
        uint32_t attrs = 0;
        if (pdl) {
            attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
        }
        if (p->mv.cluster > 1u) {
            attr[attrs].id = cudaLaunchAttributeClusterDimension;
            attr[attrs].val.clusterDim.x = p->mv.cluster;
            attr[attrs].val.clusterDim.y = 1;
            attr[attrs++].val.clusterDim.z = 1;
        }
        cfg.attrs = attr;
        cfg.numAttrs = attrs;
        const auto kernel = matvec_kernel(p->m, p->k, p->mv.sm_warps);
        LAUNCH_TRY(cudaLaunchKernelEx(&cfg, kernel, a));
    }
    CUDA_TRY(cudaGetLastError());
    return LEXB_OK;
}

// Consecutive steps of a list that can run as one persistent kernel (matmul_q_chain_sm100.cuh): block-scaled
// matmul_q of up to 8 tokens with the default ring depth and digit-row source of their token count, the same t and activation type
// (n and k may differ), K whole or split by the planner, weights declared constant or untouched by the list so far.  LEXB_CHAIN=0 turns it off.
// (two accumulator sets of 2 x 64 columns: 8 tokens x 8 digit rows)
static uint32_t chain_max_m() {
    static const uint32_t v = env_u32("LEXB_CHAIN_MAX_M", lexb::MQC_MAX_TOKENS);
    return v > lexb::MQC_MAX_TOKENS ? lexb::MQC_MAX_TOKENS : v;
}
// From this many tokens on the digit rows of a run come from matmul_q_pieces_kernel, not from piece warps in every block.
static uint32_t chain_pre_min_m() {
    static const uint32_t v = env_u32("LEXB_CHAIN_PRE_MIN_M", 3);
    return v;
}
// Address ranges a step reads and writes, for the dependence checks of a step list.
struct Range { const char *lo, *hi; };
inline bool meet(Range a, Range b) { return a.lo < b.hi && b.lo < a.hi; }
struct StepRanges {
    Range x{}, wq{}, ws{}, wg{}, r{}, y{};
    bool valid = false;          // false: a null pipeline, buffer list or buffer (the step's own launch reports it)
};

StepRanges step_ranges(const lexb_step& s) {
    StepRanges out;
    const lexb_pipeline* p = s.pipeline;
    const uint32_t q = p && p->x_q16 ? 1u : 0u;       // int16 activations bring their scales as a second binding
    if (!p || !s.buffers || s.nbuffers != (p->residual ? 6u : 5u) + q) return out;
    for (uint32_t b = 0; b < s.nbuffers; b++)
        if (!s.buffers[b] || !s.buffers[b]->ptr) return out;
    auto range = [](const lexb_buffer* b, size_t bytes) { const char* p0 = static_cast<const char*>(b->ptr); return Range{p0, p0 + bytes}; };
    const size_t m = p->m, n = p->n, k = p->k, out_bytes = m * n * 4;
    out.x = range(s.buffers[0], m * k * (p->x_f32 ? 4 : 2));
    out.wq = range(s.buffers[1 + q], n * k / 2);
    out.ws = range(s.buffers[2 + q], n * k / 16);
    out.wg = range(s.buffers[3 + q], n * 4);
    out.r = p->residual ? range(s.buffers[4 + q], out_bytes) : Range{nullptr, nullptr};
    out.y = range(s.buffers[(p->residual ? 5 : 4) + q], out_bytes);
    out.valid = true;
    return out;
}

// What the steps of one lexb_run_launches / lexb_time_launches call have written so far.  The call's first launch
// is a fence (it starts when all earlier work of the stream is done; the only launch of a call reads nothing before that), so a later step whose packed weights meet
// none of these ranges reads weights that nothing in flight writes: its kernel may load them ahead of the
// stream's order.  That is proven here from the list, as the reference's in-order contract
// (crates/lex-cuda/src/device.rs:629-672) leaves no other way to know it.
struct ListProof {
    std::vector<Range> written;      // distinct y ranges
    bool weights_untouched(const StepRanges& s) const {
        for (const Range& w : written)
            if (meet(s.wq, w) || meet(s.ws, w) || meet(s.wg, w)) return false;
        return true;
    }
    void add(const StepRanges& s) {
        for (const Range& w : written)
            if (w.lo == s.y.lo && w.hi == s.y.hi) return;
        written.push_back(s.y);
    }
};

bool chain_member(const lexb_gpu* g, const lexb_step& s, const lexb_pipeline* first) {
    const lexb_pipeline* p = s.pipeline;
    if (!p || !s.buffers || p->gpu != g || p->kernel != KERNEL_MATMUL_Q || p->x_q16 || p->m > chain_max_m() || (p->k_splits != 1u && p->splits_asked)) return false;
    if (p->mq_pre != (p->m > 4u)) return false;                                      // (a plan forced the other way by LEXB_MQ_PRE stays as planned)
    if (p->w_volatile || s.nbuffers != (p->residual ? 6u : 5u)) return false;
    if (p->k / lexb::MQ_STAGE_K > 0xFFFFu) return false;
    if ((p->k / lexb::MQ_STAGE_K) % lexb::MQ_WS_GROUP == 1u) return false;          // a scale-byte group of one stage is seen by half the scale warps only
    if (p->stages != (p->m <= 4u ? lexb::MQ_MAX_STAGES : 7u) || lexb::matmul_q_chain_smem_bytes(p->stages, p->m) > g->smem_optin) return false;
    return !first || (p->m == first->m && p->x_f32 == first->x_f32 && p->stages == first->stages);
}
// The digit rows of a run come from the pieces kernel: from 3 tokens on, past 4 in any case, and wherever the steps differ in K
// or a plan splits it (the in-block derivation walks one K, in one part).
bool chain_pre(const lexb_step* steps, size_t count) {
    const lexb_pipeline* p0 = steps[0].pipeline;
    if (p0->m >= chain_pre_min_m() || p0->m > 4u) return true;
    for (size_t i = 0; i < count; i++)
        if (steps[i].pipeline->k != p0->k || steps[i].pipeline->k_splits != 1u) return true;
    return false;
}

// Stages per part of K of a step in a run.
uint32_t chain_part(const lexb_pipeline* p) { return p->k_splits == 1u ? p->k / lexb::MQ_STAGE_K : p->kb_per_split; }

// Of the first `len` steps of a list, which one launch can take: how many it should.  Steps whose plans keep K whole always share it.
// The parts of a split K stay in one block of a run, where the step's own launch spreads them: two steps of 640 x 17408 are 10 blocks
// of 68 stages there and 40 blocks of 9 alone (48 us and 30), three 27B layers 106 us and 160.  So a run with split plans is priced
// against its steps' own launches, with the number of steps with which it and what is left cost least.  Fitted to 150 lists timed both
// ways (2-6 steps, t = 1-8, n = 128-20480, k = 512-17408; median error 3 % and 6 %), us: a run 12.4 and 0.546 per stage of its fullest
// block; a list 5.2, a step of it 3.2, 0.536 per stage of each wave of blocks, 1.2 for a split, the walk over the tokens for their
// digits, in front of the product past 4 tokens.  A run is given up where it costs a tenth more.  On 100 other lists the way taken takes
// 0.997 of the faster of the two whole ways in the mean and 1.06 at most; every run taken, 1.02 and 1.9.  LEXB_CHAIN_SPLITS=1: it is
// taken whatever it costs.
size_t run_that_pays(const lexb_step* steps, size_t len, uint32_t sms) {
    size_t unsplit = 0;
    while (unsplit < len && steps[unsplit].pipeline->k_splits == 1u) unsplit++;
    if (unsplit == len || env_u32("LEXB_CHAIN_SPLITS", 0) != 0u) return len;
    using Tiles = std::vector<std::pair<uint32_t, uint32_t>>;    // (stages of a row tile, tiles), longest first
    auto add = [](Tiles& tiles, uint32_t stages, uint32_t count) {
        auto at = std::find_if(tiles.begin(), tiles.end(), [&](const auto& e) { return e.first <= stages; });
        if (at != tiles.end() && at->first == stages) at->second += count;
        else tiles.insert(at, {stages, count});
    };
    auto fullest = [&](const Tiles& tiles) {                     // stages of the fullest block, dealt out as well as can be
        uint64_t total = 0, count = 0, most = 0;
        for (const auto& e : tiles) count += e.second;
        const uint64_t blocks = std::min<uint64_t>(count, sms);
        count = 0;
        for (const auto& e : tiles) {
            count += e.second;
            total += static_cast<uint64_t>(e.first) * e.second;
            most = std::max(most, (count + blocks - 1u) / blocks * e.first);
        }
        return static_cast<double>(std::max(most, (total + blocks - 1u) / blocks));
    };
    constexpr double RUN = 12.4, RUN_STAGE = 0.546, LIST = 5.18, STEP = 3.17, STEP_STAGE = 0.536, STEP_SPLIT = 1.19, STEP_PIECES = 3.39, WALK = 0.0132;
    // us of steps i, i + 1, ... in launches of their own, those that keep K whole as one run if that is less
    std::vector<double> apart(len + 1u, 0.0);
    Tiles tiles;
    double split_alone = 0.0, whole_alone = 0.0;
    for (size_t i = len, whole_steps = 0; i-- > 0;) {
        const lexb_pipeline* p = steps[i].pipeline;
        const uint32_t rows = p->n / lexb::MQ_ROWS, kb = p->k / lexb::MQ_STAGE_K, waves = (rows * p->k_splits + sms - 1u) / sms;
        const double us = STEP + STEP_STAGE * waves * chain_part(p) + (p->m > 4u ? STEP_PIECES + WALK * kb : WALK * p->m * kb);
        if (p->k_splits == 1u) {
            add(tiles, kb, rows);
            whole_alone += us;
            whole_steps++;
        } else {
            split_alone += us + STEP_SPLIT;
        }
        apart[i] = split_alone + (whole_steps > 1u ? std::min(whole_alone, RUN - LIST + RUN_STAGE * fullest(tiles)) : whole_alone);
    }
    tiles.clear();
    double without = LIST + apart[0], with = 1e30;
    size_t best = 0;
    for (size_t i = 0; i < len; i++) {
        add(tiles, steps[i].pipeline->k / lexb::MQ_STAGE_K, steps[i].pipeline->n / lexb::MQ_ROWS);
        if (i == 0 || i + 1u < unsplit) continue;
        const double us = RUN + RUN_STAGE * fullest(tiles) + apart[i + 1u];
        if (i + 1u == unsplit) without = us;
        else if (us <= with) {
            with = us;
            best = i + 1u;
        }
    }
    return with <= 1.1 * without ? best : unsplit >= 2u ? unsplit : 0u;
}

// Length of the run of steps starting at i that one persistent kernel can take (0: step i is launched on its own).
// The run's copy warp starts on the weights at once, so every member's weights must be declared constant or be
// untouched by the steps of this call so far (`proof`) and by the run's own members.
size_t chain_run(const lexb_gpu* g, const lexb_step* steps, size_t nsteps, size_t i, const ListProof& proof) {
    static const bool on = env_u32("LEXB_CHAIN", 1) != 0;
    if (!on || !chain_member(g, steps[i], nullptr)) return 0;
    const StepRanges first = step_ranges(steps[i]);
    if (!first.valid) return 0;                                  // a null buffer entry: the step's own launch reports it
    if (!steps[i].pipeline->w_const && !proof.weights_untouched(first)) return 0;
    // The run's row tiles are spread over the blocks with no order between blocks, so a step joins the run only
    // if nothing it reads (x, r, the weights) is written by a step already in it and nothing it writes (y) is
    // read or written by one: such a step starts the next launch, and the stream orders it.
    std::vector<StepRanges> in_run{first};
    auto conflicts = [&](const StepRanges& c, bool declared_const) {
        if (!declared_const && !proof.weights_untouched(c)) return true;
        for (const StepRanges& e : in_run) {
            if (meet(c.x, e.y) || meet(c.r, e.y) || meet(c.y, e.x) || meet(c.y, e.r) || meet(c.y, e.y)) return true;
            if (meet(c.wq, e.y) || meet(c.ws, e.y) || meet(c.wg, e.y) || meet(c.y, e.wq) || meet(c.y, e.ws) || meet(c.y, e.wg)) return true;
        }
        return false;
    };
    size_t len = 1;
    bool alike = true;                           // (steps of several lengths: their tiles are dealt out one by one, once per list)
    while (i + len < nsteps && len < (alike ? 4096u : 64u) && chain_member(g, steps[i + len], steps[i].pipeline)) {
        const StepRanges c = step_ranges(steps[i + len]);
        if (!c.valid || conflicts(c, steps[i + len].pipeline->w_const)) break;
        if (steps[i + len].pipeline->k != steps[i].pipeline->k) {
            if (len >= 64u) break;
            alike = false;
        }
        in_run.push_back(c);
        len++;
    }
    if (len >= 2) len = run_that_pays(steps + i, len, static_cast<uint32_t>(g->prop.multiProcessorCount));
    if (len != 1) return len;
    // a single step with more row tiles than SMs: the persistent kernel takes them without a second wave of
    // block set-ups (n = 28672: 224 tiles)
    static const bool single = env_u32("LEXB_CHAIN_SINGLE", 1) != 0;
    const uint32_t tiles = (steps[i].pipeline->n + lexb::MQ_ROWS - 1u) / lexb::MQ_ROWS;
    return single && steps[i].pipeline->k_splits == 1u && tiles > static_cast<uint32_t>(g->prop.multiProcessorCount) ? 1 : 0;
}

// The table of a run's row tiles: block b works through entries b, b + grid, ...; a row of entries without a job ends it.  Tiles go
// to the block with the fewest stages so far, the longest tiles first, so that steps of several K end together.
std::vector<lexb::MqChainTile> chain_tiles(const lexb_step* steps, size_t count, uint32_t sms, uint32_t* grid_out) {
    std::vector<std::pair<uint32_t, uint32_t>> order;            // (stages of a tile, step), longest first
    uint32_t total = 0;
    for (size_t i = 0; i < count; i++) {
        const lexb_pipeline* p = steps[i].pipeline;
        order.emplace_back(p->k / lexb::MQ_STAGE_K, static_cast<uint32_t>(i));
        total += p->n / lexb::MQ_ROWS;
    }
    std::stable_sort(order.begin(), order.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
    const uint32_t grid = std::min(total, sms);
    const bool alike = order.front().first == order.back().first;
    std::vector<std::vector<lexb::MqChainTile>> of(grid);
    using Load = std::pair<uint64_t, uint32_t>;                  // (stages, block)
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> least;
    if (!alike)
        for (uint32_t b = 0; b < grid; b++) least.emplace(0, b);
    uint32_t turn = 0;
    for (const auto& e : order) {
        const lexb_pipeline* p = steps[e.second].pipeline;
        for (uint32_t n0 = 0; n0 < p->n; n0 += lexb::MQ_ROWS) {
            uint32_t b = turn;
            if (alike) {
                turn = turn + 1u == grid ? 0u : turn + 1u;
            } else {
                const Load l = least.top();
                least.pop();
                b = l.second;
                least.emplace(l.first + e.first, b);
            }
            of[b].push_back(lexb::MqChainTile{e.second, n0, e.first | (p->ws_pitch << 16), chain_part(p)});
        }
    }
    size_t rows = 0;
    for (const auto& v : of) rows = std::max(rows, v.size());
    std::vector<lexb::MqChainTile> out((rows + 1u) * grid, lexb::MqChainTile{lexb::MQC_NO_JOB, 0, 0, 0});
    for (uint32_t b = 0; b < grid; b++)
        for (size_t t = 0; t < of[b].size(); t++) out[t * grid + b] = of[b][t];
    *grid_out = grid;
    return out;
}

int launch_chain(lexb_gpu* g, const lexb_step* steps, size_t count, bool fence) {
    bool pdl_next = g->pdl && !fence;            // the run's first kernel launch is the fence, when one is asked for
    const lexb_pipeline* p0 = steps[0].pipeline;
    const uint32_t m = p0->m;
    std::vector<lexb::MqChainJob> jobs(count);
    int rc;
    const bool pre = chain_pre(steps, count);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    struct Act { const void* x; uint32_t k; size_t offset; };    // PRE: the run's distinct activation buffers and their place in the arena
    std::vector<Act> acts;
    std::vector<uint32_t> act_of(pre ? count : 0);
    size_t arena_need = 0;
    for (size_t i = 0; i < count; i++) {
        const lexb_pipeline* p = steps[i].pipeline;
        lexb_buffer* const* b = steps[i].buffers;
        const lexb_buffer *x = b[0], *wq = b[1], *ws = b[2], *wg = b[3], *r = p->residual ? b[4] : nullptr;
        const lexb_buffer* y = p->residual ? b[5] : b[4];
        const size_t n = p->n, k = p->k;
        if ((rc = check_buf(x, g, m * k * (p->x_f32 ? 4 : 2), "x"))) return rc;
        if ((rc = check_buf(wq, g, n * k / 2, "wq"))) return rc;
        if ((rc = check_buf(ws, g, n * k / 16, "ws"))) return rc;
        if ((rc = check_buf(wg, g, n * 4, "wg"))) return rc;
        if ((rc = check_buf(y, g, m * n * 4, "y"))) return rc;
        if (r && (rc = check_buf(r, g, m * n * 4, "r"))) return rc;
        lexb_pipeline::MapEntry maps;
        if ((rc = get_maps(p, x->ptr, wq->ptr, ws->ptr, &maps))) return rc;
        jobs[i].wq = maps.map_wq;
        jobs[i].ws = maps.map_ws;
        jobs[i].x = x->ptr;
        jobs[i].wg = static_cast<const float*>(wg->ptr);
        jobs[i].r = r ? static_cast<const float*>(r->ptr) : nullptr;
        jobs[i].y = static_cast<float*>(y->ptr);
        jobs[i].n = p->n;
        jobs[i].k = p->k;
        jobs[i].per = chain_part(p);
        if (pre) {
            size_t e = 0;
            while (e < acts.size() && (acts[e].x != x->ptr || acts[e].k != p->k)) e++;
            if (e == acts.size()) {
                acts.push_back(Act{x->ptr, p->k, arena_need});
                arena_need += (lexb::matmul_q_pre_bytes(m, p->k) + 255u) / 256u * 256u;
            }
            act_of[i] = static_cast<uint32_t>(e);
        }
    }
    if (pre) {
        if (g->chain_arenas.size() >= 64 && !g->chain_arenas.count(g->stream)) {
            // streams come and go: start over (nothing in flight may still read the arenas)
            CUDA_TRY(cudaDeviceSynchronize());
            for (auto& e : g->chain_arenas) cudaFree(e.second.buf);
            for (uint8_t* b : g->retired_arenas) cudaFree(b);
            g->chain_arenas.clear();
            g->retired_arenas.clear();
        }
        lexb_gpu::ChainArena& arena = g->chain_arenas[g->stream];
        if (arena.bytes < arena_need) {
            const size_t bytes = std::max(arena_need, 2u * arena.bytes);
            uint8_t* buf = nullptr;
            CUDA_TRY(x_malloc(&buf, bytes));
            if (arena.buf) g->retired_arenas.push_back(arena.buf);
            arena.buf = buf;
            arena.bytes = bytes;
            arena.maps.clear();
        }
        if (arena.maps.size() + acts.size() > 4096u) arena.maps.clear();
        std::vector<const CUtensorMap*> act_map(acts.size());
        for (size_t e = 0; e < acts.size(); e++) {
            const auto key = std::make_tuple(acts[e].offset, m, acts[e].k);
            auto it = arena.maps.find(key);
            if (it == arena.maps.end()) {
                CUtensorMap map;
                if ((rc = encode_2d(p0, &map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, arena.buf + acts[e].offset, acts[e].k / 2u, 8u * m, 128u, 8u * m,
                                    CU_TENSOR_MAP_SWIZZLE_128B, "digit rows of a run")))
                    return rc;
                it = arena.maps.emplace(key, map).first;
            }
            act_map[e] = &it->second;
        }
        for (size_t i = 0; i < count; i++) {
            const Act& act = acts[act_of[i]];
            jobs[i].pre = *act_map[act_of[i]];
            jobs[i].pre_sfb = arena.buf + act.offset + lexb::matmul_q_pieces_bytes(m, act.k);
            jobs[i].pre_amax = reinterpret_cast<const uint32_t*>(jobs[i].pre_sfb + lexb::matmul_q_sfb_total(m, act.k));
        }
        for (size_t e0 = 0; e0 < acts.size(); e0 += lexb::MQ_PIECES_LIST) {
            const size_t e1 = std::min<size_t>(acts.size(), e0 + lexb::MQ_PIECES_LIST);
            lexb::MqPiecesList list{};
            uint32_t kb_most = 0;
            for (size_t e = e0; e < e1; e++) {
                list.job[e - e0] = lexb::MqPiecesJob{acts[e].x, nullptr, arena.buf + acts[e].offset, acts[e].k};
                kb_most = std::max(kb_most, acts[e].k / lexb::MQ_STAGE_K);
            }
            cudaLaunchConfig_t pc{};
            pc.gridDim = dim3(m, (kb_most + 31u) / 32u, static_cast<uint32_t>(e1 - e0));      // a warp per stage
            pc.blockDim = dim3(1024);
            pc.stream = g->stream;
            pc.attrs = attr;
            pc.numAttrs = pdl_next ? 1 : 0;
            pdl_next = g->pdl;
            LAUNCH_TRY(cudaLaunchKernelEx(&pc, pieces_kernel(p0->x_f32 ? 1 : 0), list, 0u));
        }
    }
    const size_t table_bytes = sizeof(lexb::MqChainJob) * count;
    uint64_t h = 1469598103934665603ull;
    {
        const uint64_t* words = reinterpret_cast<const uint64_t*>(jobs.data());      // (a job is whole 64-byte lines)
        for (size_t i = 0; i < table_bytes / 8u; i++) {
            h = (h ^ words[i]) * 0x9E3779B97F4A7C15ull;
            h ^= h >> 32;
        }
    }
    const lexb_gpu::ChainTable* table = nullptr;
    auto hit = g->chain_tables.equal_range(h);
    for (auto it = hit.first; it != hit.second && !table; ++it)
        if (it->second.host.size() == count && !memcmp(it->second.host.data(), jobs.data(), table_bytes)) table = &it->second;
    if (!table) {
        if (g->chain_tables.size() >= 4096) {
            // (tables of launches still in flight are freed only after them)
            CUDA_TRY(cudaStreamSynchronize(g->stream));
            for (auto& e : g->chain_tables) cudaFree(e.second.dev);
            g->chain_tables.clear();
        }
        uint32_t grid = 0;
        std::vector<lexb::MqChainTile> tiles = chain_tiles(steps, count, static_cast<uint32_t>(g->prop.multiProcessorCount), &grid);
        const size_t tile_bytes = sizeof(lexb::MqChainTile) * tiles.size();
        lexb::MqChainJob* d_jobs = nullptr;
        CUDA_TRY(x_malloc(&d_jobs, table_bytes + tile_bytes));
        auto it = g->chain_tables.emplace(h, lexb_gpu::ChainTable{std::move(jobs), std::move(tiles), grid, d_jobs});
        table = &it->second;
        // (the source is the cache's own copy: it outlives the transfer)
        auto copy = [&]() -> int {
            CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(d_jobs, table->host.data(), table_bytes, cudaMemcpyHostToDevice, g->stream));
            CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(d_jobs + count, table->tiles.data(), tile_bytes, cudaMemcpyHostToDevice, g->stream));
            return LEXB_OK;
        };
        if ((rc = copy())) {                     // (a table that was not copied is not kept)
            cudaStreamSynchronize(g->stream);
            g->chain_tables.erase(it);
            cudaFree(d_jobs);
            return rc;
        }
    }
    lexb::MqChainArgs a{};
    a.jobs = table->dev;
    a.tiles = reinterpret_cast<const lexb::MqChainTile*>(table->dev + count);
    a.m = m; a.stages = p0->stages;
    a.status = g->d_status;
    // blocks of this kernel do not wait for one another, and there is at most one per SM
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(table->grid);
    cfg.blockDim = dim3(pre ? lexb::MQC_THREADS_PRE : lexb::MQC_THREADS);
    cfg.dynamicSmemBytes = lexb::matmul_q_chain_smem_bytes(p0->stages, m);
    cfg.stream = g->stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_next ? 1 : 0;
    if (pre) {
        if (p0->x_f32) LAUNCH_TRY(cudaLaunchKernelEx(&cfg, lexb::matmul_q_chain_kernel<true, true>, a));
        else LAUNCH_TRY(cudaLaunchKernelEx(&cfg, lexb::matmul_q_chain_kernel<false, true>, a));
    } else {
        if (p0->x_f32) LAUNCH_TRY(cudaLaunchKernelEx(&cfg, lexb::matmul_q_chain_kernel<true, false>, a));
        else LAUNCH_TRY(cudaLaunchKernelEx(&cfg, lexb::matmul_q_chain_kernel<false, false>, a));
    }
    return LEXB_OK;
}

int launch_step(lexb_gpu* g, const lexb_step& s, const lexb_step* following = nullptr, Order order = Order{}) {
    if (!s.pipeline || !s.buffers) return fail(LEXB_ERR_ARG, "step without pipeline or buffers");
    const bool res = s.pipeline->residual;
    const uint32_t q = s.pipeline->x_q16 ? 1u : 0u;
    if (s.nbuffers != (res ? 6u : 5u) + q)
        return fail(LEXB_ERR_ARG, "step binds %u buffers, the pipeline takes %u: [%s, wq, ws, wg, %sy]", s.nbuffers,
                    (res ? 6u : 5u) + q, q ? "xq, xs" : "x", res ? "r, " : "");
    if (q) {
        // matmul_int8's bindings (crates/lex-msl/src/int8.rs:121-125): [xq, xs, wq, ws, wg, (r), y]
        lexb_buffer* const* c = s.buffers;
        return launch_one(g, s.pipeline, c[0], c[2], c[3], c[4], res ? c[5] : nullptr, res ? c[6] : c[5], nullptr, nullptr, order,
                          nullptr, c[1]);
    }
    lexb_buffer* const* b = s.buffers;
    NextWeights nw{};
    static const bool hints = env_u32("LEXB_NEXT_HINT", 1) != 0;     // LEXB_NEXT_HINT=0: no prefetch of the next step's weights
    if (hints && following && following->pipeline && following->buffers && following->nbuffers >= 5u && !following->pipeline->x_q16)
        nw = NextWeights{following->pipeline, following->buffers[0], following->buffers[1], following->buffers[2]};
    return launch_one(g, s.pipeline, b[0], b[1], b[2], b[3], res ? b[4] : nullptr, res ? b[5] : b[4], nullptr,
                      nw.pipe ? &nw : nullptr, order);
}

// Issues the steps of a list once, in order, forming runs; `proof` and `first` carry over between the passes of
// lexb_time_launches.  `first`: nothing of this call has been launched yet - that launch is the call's fence.
// `lone`: a single step, issued once.  Nothing follows that could use a fence: the launch's set-up is hidden behind the launch
// ahead, but like a fence it reads nothing before all earlier work of the stream is done, whatever was declared constant.
int issue_list(lexb_gpu* g, const lexb_step* steps, size_t nsteps, ListProof& proof, bool& first, const lexb_step* after_last, bool lone = false) {
    int rc;
    for (size_t i = 0; i < nsteps;) {
        if (const size_t len = chain_run(g, steps, nsteps, i, proof)) {
            if ((rc = launch_chain(g, steps + i, len, first))) return rc;
            for (size_t e = i; e < i + len; e++) proof.add(step_ranges(steps[e]));
            first = false;
            i += len;
            continue;
        }
        const StepRanges sr = step_ranges(steps[i]);
        Order order;
        order.fence = first && !lone;
        order.in_order = lone;
        order.early_weights = sr.valid && proof.weights_untouched(sr);
        const lexb_step* following = i + 1 < nsteps ? &steps[i + 1] : after_last;
        if ((rc = launch_step(g, steps[i], following, order))) return rc;
        if (sr.valid) proof.add(sr);
        first = false;
        i++;
    }
    return LEXB_OK;
}

}  // namespace

extern "C" {

const char* lexb_last_error(void) { return g_last_error.c_str(); }
const char* lexb_version(void) { return "lexb 0.1 (sm_100a; gemm_fp4: tcgen05 GEMM + split-K matvec)"; }

int lexb_open(int device, lexb_gpu** out) {
    if (!out) return fail(LEXB_ERR_ARG, "lexb_open: null out");
    *out = nullptr;
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0)
        return fail(LEXB_ERR_UNSUPPORTED, "no CUDA device (%s); this library has no CPU path", cudaGetErrorString(e));
    if (device < 0 || device >= count) return fail(LEXB_ERR_ARG, "device %d out of range (%d devices)", device, count);
    lexb_gpu* g = new (std::nothrow) lexb_gpu();
    if (!g) return fail(LEXB_ERR_ARG, "out of host memory");
    g->device = device;
    auto bail = [&](int code) { lexb_close(g); return code; };
    if (cudaSetDevice(device) != cudaSuccess) return bail(fail(LEXB_ERR_CUDA, "cudaSetDevice(%d) failed", device));
    if (cudaGetDeviceProperties(&g->prop, device) != cudaSuccess) return bail(fail(LEXB_ERR_CUDA, "cudaGetDeviceProperties failed"));
    if (g->prop.major != 10)
        return bail(fail(LEXB_ERR_UNSUPPORTED, "device %d is %s (compute %d.%d); the kernels are built for sm_100a only",
                         device, g->prop.name, g->prop.major, g->prop.minor));
    g->smem_optin = g->prop.sharedMemPerBlockOptin;
    g->pdl = env_u32("LEXB_PDL", 1) != 0;
    if (cudaStreamCreateWithFlags(&g->own_stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(fail(LEXB_ERR_CUDA, "cudaStreamCreate failed"));
    g->stream = g->own_stream;
    if (cudaMalloc(&g->d_status, sizeof(uint32_t)) != cudaSuccess || cudaMemsetAsync(g->d_status, 0, sizeof(uint32_t), g->stream) != cudaSuccess ||
        cudaStreamSynchronize(g->stream) != cudaSuccess)
        return bail(fail(LEXB_ERR_CUDA, "allocating the status word failed"));
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || !fn ||
        qres != cudaDriverEntryPointSuccess)
        return bail(fail(LEXB_ERR_CUDA, "the driver does not export cuTensorMapEncodeTiled"));
    g->encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
    const int max_smem = static_cast<int>(g->smem_optin);
    if (cudaFuncSetAttribute(lexb::gemm_fp4_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<true>(true, true), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<true>(true, false), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<true>(false, true), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<true>(false, false), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<false>(true, true), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<false>(true, false), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<false>(false, true), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(pair_kernel<false>(false, false), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::gemm_fp4_few_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::gemm_fp4_few_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::gemm_fp4_few_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<true, true, 24>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<true, false, 24>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<false, true, 24>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<false, true, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<false, false, 24>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matvec_fp4_kernel<false, false, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_chain_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_chain_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_chain_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_chain_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<false, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<false, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<false, 1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<false, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<false, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<true, 0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<true, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<true, 1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<true, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess ||
        cudaFuncSetAttribute(lexb::matmul_q_fp4_kernel<true, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) != cudaSuccess)
        return bail(fail(LEXB_ERR_CUDA, "cudaFuncSetAttribute(max dynamic shared memory) failed: %s", cudaGetErrorString(cudaGetLastError())));
    *out = g;
    return LEXB_OK;
}

void lexb_close(lexb_gpu* g) {
    if (!g) return;
    cudaSetDevice(g->device);
    if (g->own_stream) {
        cudaStreamSynchronize(g->own_stream);
        cudaStreamDestroy(g->own_stream);
    }
    if (g->host.in) cudaStreamDestroy(g->host.in);
    if (g->host.out) cudaStreamDestroy(g->host.out);
    for (cudaEvent_t e : g->host.event)
        if (e) cudaEventDestroy(e);
    if (g->d_status) cudaFree(g->d_status);
    if (g->d_trace) cudaFree(g->d_trace);
    for (auto& e : g->chain_tables) cudaFree(e.second.dev);
    g->chain_tables.clear();
    for (auto& e : g->chain_arenas) cudaFree(e.second.buf);
    for (uint8_t* b : g->retired_arenas) cudaFree(b);
    delete g;
}

int lexb_info(lexb_gpu* g, lexb_device_info* out) {
    int rc = use(g);
    if (rc) return rc;
    if (!out) return fail(LEXB_ERR_ARG, "lexb_info: null out");
    memset(out, 0, sizeof *out);
    snprintf(out->name, sizeof out->name, "%s", g->prop.name);
    out->cc_major = g->prop.major;
    out->cc_minor = g->prop.minor;
    out->sm_count = g->prop.multiProcessorCount;
    out->unified_memory = 0;
    out->max_threadgroup_bytes = g->smem_optin;
    out->recommended_working_set_bytes = g->prop.totalGlobalMem;
    out->l2_bytes = static_cast<size_t>(g->prop.l2CacheSize);
    return LEXB_OK;
}

int lexb_set_stream(lexb_gpu* g, void* cuda_stream) {
    int rc = use(g);
    if (rc) return rc;
    g->stream = cuda_stream ? static_cast<cudaStream_t>(cuda_stream) : g->own_stream;
    return LEXB_OK;
}
void* lexb_get_stream(lexb_gpu* g) { return g ? static_cast<void*>(g->stream) : nullptr; }

int lexb_sync(lexb_gpu* g) {
    int rc = use(g);
    if (rc) return rc;
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_alloc(lexb_gpu* g, size_t bytes, lexb_buffer** out) {
    int rc = use(g);
    if (rc) return rc;
    if (!out) return fail(LEXB_ERR_ARG, "lexb_alloc: null out");
    *out = nullptr;
    void* p = nullptr;
    CUDA_TRY(x_malloc(&p, bytes ? bytes : 1));
    lexb_buffer* b = new (std::nothrow) lexb_buffer{g, p, bytes, true, g->device};
    if (!b) {
        cudaFree(p);
        return fail(LEXB_ERR_ARG, "out of host memory");
    }
    *out = b;
    return LEXB_OK;
}

int lexb_zeroed(lexb_gpu* g, size_t bytes, lexb_buffer** out) {
    int rc = lexb_alloc(g, bytes, out);
    if (rc) return rc;
    if (bytes) {
        cudaError_t e = cudaMemsetAsync((*out)->ptr, 0, bytes, g->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
        if (e != cudaSuccess) {
            lexb_free(*out);
            *out = nullptr;
            return fail(LEXB_ERR_CUDA, "zeroing %zu bytes failed: %s", bytes, cudaGetErrorString(e));
        }
    }
    return LEXB_OK;
}

int lexb_wrap(lexb_gpu* g, void* device_ptr, size_t bytes, lexb_buffer** out) {
    if (!g || !out) return fail(LEXB_ERR_ARG, "lexb_wrap: null argument");
    if (!device_ptr && bytes) return fail(LEXB_ERR_ARG, "lexb_wrap: null device pointer");
    lexb_buffer* b = new (std::nothrow) lexb_buffer{g, device_ptr, bytes, false, g->device};
    if (!b) return fail(LEXB_ERR_ARG, "out of host memory");
    *out = b;
    return LEXB_OK;
}

int lexb_free(lexb_buffer* b) {
    if (!b) return LEXB_OK;
    int rc = LEXB_OK;
    if (b->owned && b->ptr) {
        const cudaError_t e = free_on(b->device, {b->ptr});
        if (e != cudaSuccess) rc = fail(LEXB_ERR_CUDA, "cudaFree: %s", cudaGetErrorString(e));
    }
    delete b;
    return rc;
}

void* lexb_buffer_ptr(const lexb_buffer* b) { return b ? b->ptr : nullptr; }
size_t lexb_buffer_bytes(const lexb_buffer* b) { return b ? b->bytes : 0; }

int lexb_upload(lexb_gpu* g, lexb_buffer* dst, size_t off, const void* src, size_t bytes) {
    int rc = use(g);
    if (rc) return rc;
    if (!dst || (!src && bytes)) return fail(LEXB_ERR_ARG, "lexb_upload: null argument");
    if (off > dst->bytes || bytes > dst->bytes - off)
        return fail(LEXB_ERR_ARG, "lexb_upload: %zu bytes at offset %zu overrun a buffer of %zu", bytes, off, dst->bytes);
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(static_cast<char*>(dst->ptr) + off, src, bytes, cudaMemcpyHostToDevice, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_download(lexb_gpu* g, const lexb_buffer* src, size_t off, void* dst, size_t bytes) {
    int rc = use(g);
    if (rc) return rc;
    if (!src || (!dst && bytes)) return fail(LEXB_ERR_ARG, "lexb_download: null argument");
    if (off > src->bytes || bytes > src->bytes - off)
        return fail(LEXB_ERR_ARG, "lexb_download: %zu bytes at offset %zu overrun a buffer of %zu", bytes, off, src->bytes);
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(dst, static_cast<const char*>(src->ptr) + off, bytes, cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_memset(lexb_gpu* g, lexb_buffer* dst, int byte, size_t bytes) {
    int rc = use(g);
    if (rc) return rc;
    if (!dst) return fail(LEXB_ERR_ARG, "lexb_memset: null buffer");
    if (bytes > dst->bytes) return fail(LEXB_ERR_ARG, "lexb_memset: %zu bytes overrun a buffer of %zu", bytes, dst->bytes);
    CUDA_TRY(cudaMemsetAsync(dst->ptr, byte, bytes, g->stream));
    return LEXB_OK;
}

int lexb_host_alloc(size_t bytes, void** out) {
    if (!out) return fail(LEXB_ERR_ARG, "lexb_host_alloc: null out");
    CUDA_TRY(cudaHostAlloc(out, bytes ? bytes : 1, cudaHostAllocDefault));
    return LEXB_OK;
}
int lexb_host_free(void* p) {
    if (p) CUDA_TRY(cudaFreeHost(p));
    return LEXB_OK;
}

int lexb_gemm_fp4_plan(lexb_gpu* g, uint32_t m, uint32_t n, uint32_t k, int residual, const lexb_sched* sched,
                       lexb_pipeline** out) {
    int rc = use(g);
    if (rc) return rc;
    if (!out) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_plan: null out");
    *out = nullptr;
    if (m == 0 || n == 0 || k == 0) return fail(LEXB_ERR_SHAPE, "gemm_fp4: empty extent (m=%u n=%u k=%u)", m, n, k);
    lexb_sched s{};
    if (sched) s = *sched;
    if (!s.kernel) s.kernel = env_u32("LEXB_KERNEL", 0);
    if (!s.tm) s.tm = env_u32("LEXB_TM", 0);
    if (!s.stages) s.stages = env_u32("LEXB_STAGES", 0);
    if (!s.kc) s.kc = env_u32("LEXB_KC", 0);
    if (!s.w_stages) s.w_stages = env_u32("LEXB_WSTAGES", 0);
    if (!s.k_splits) s.k_splits = env_u32("LEXB_KSPLITS", 0);
    // m <= 8: matvec (it also takes 9..16 when asked, but the GEMMs are faster there).  Otherwise the
    // two-CTA GEMM when the shape allows it (k in blocks of 256); the one-CTA kernel takes the rest.
    uint32_t kernel = s.kernel;
    if (!kernel) {
        if (m <= 8 || ((n % lexb::GEMM_TN || k % lexb::GEMM_BK) && m <= 16)) kernel = KERNEL_MATVEC;
        else if (n % lexb::GEMM_TN == 0 && k % lexb::PAIR_RAW_K == 0)
            kernel = KERNEL_TCGEN05_PAIR;
        else kernel = KERNEL_TCGEN05;
    }
    if (kernel == KERNEL_MATVEC && m > 16) return fail(LEXB_ERR_SHAPE, "the matvec kernel takes m <= 16, not %u", m);
    if (kernel < KERNEL_MATVEC || kernel > KERNEL_MATMUL_Q) return fail(LEXB_ERR_ARG, "unknown kernel selector %u", kernel);

    lexb_pipeline* p = new (std::nothrow) lexb_pipeline();
    if (!p) return fail(LEXB_ERR_ARG, "out of host memory");
    p->gpu = g;
    p->device = g->device;
    p->kernel = kernel;
    p->m = m; p->n = n; p->k = k;
    p->residual = residual != 0;
    auto bail = [&](int code) { lexb_pipeline_free(p); return code; };
    const char* stem = residual ? "gemm_fp4_res" : "gemm_fp4";
    p->w_const = (s.flags & LEXB_SCHED_WEIGHTS_CONSTANT) != 0u;
    p->w_volatile = (s.flags & LEXB_SCHED_WEIGHTS_MAY_CHANGE) != 0u;
    if (p->w_const && p->w_volatile)
        return bail(fail(LEXB_ERR_ARG, "LEXB_SCHED_WEIGHTS_CONSTANT and LEXB_SCHED_WEIGHTS_MAY_CHANGE exclude one another"));

    if (kernel == KERNEL_MATMUL_Q) {
        // Only through lexb_matmul_fp4_plan or an explicit selector: its arithmetic is matmul_q_x's
        // (weights not rounded to f16), within gemm_fp4's tolerance but not its rounding.
        if (m > lexb::MQ_MAX_TOKENS) return bail(fail(LEXB_ERR_SHAPE, "the block-scaled kernel takes at most %u tokens, not %u", lexb::MQ_MAX_TOKENS, m));
        if (n % lexb::MQ_ROWS) return bail(fail(LEXB_ERR_SHAPE, "matmul_q (nvfp4): %u rows per block do not divide n = %u", lexb::MQ_ROWS, n));
        if (k % lexb::MQ_STAGE_K) return bail(fail(LEXB_ERR_SHAPE, "matmul_q (nvfp4): blocks of %u columns do not divide k = %u", lexb::MQ_STAGE_K, k));
        uint32_t stages = s.stages ? s.stages : (m <= 4u ? lexb::MQ_MAX_STAGES : (m <= 8u ? 7u : (m <= 16u ? 5u : 3u)));     // what fits shared memory
        const uint32_t max_stages = m <= 16u ? lexb::MQ_MAX_STAGES : lexb::MQ_WIDE_MAX_STAGES;    // ... and, past 16 tokens, tensor memory
        if (stages < 2 || stages > max_stages || lexb::matmul_q_smem_bytes(m, stages) > g->smem_optin)
            return bail(fail(LEXB_ERR_ARG, "stages = %u outside [2, %u] or over the shared-memory limit", stages, max_stages));
        const uint32_t tiles = n / lexb::MQ_ROWS, kb_all = k / lexb::MQ_STAGE_K;
        const uint32_t sms = static_cast<uint32_t>(g->prop.multiProcessorCount);
        // one K range per block; split K when the row tiles alone leave most SMs idle
        uint32_t splits = s.k_splits ? s.k_splits : (tiles * 2u <= sms ? sms / tiles : 1u);
        if (splits > lexb::MQ_MAX_SPLITS) splits = lexb::MQ_MAX_SPLITS;
        while (splits > 1u && kb_all / splits < 4u) splits--;
        if (splits < 1u) splits = 1u;
        const uint32_t per = (kb_all + splits - 1u) / splits;
        splits = (kb_all + per - 1u) / per;
        p->k_splits = splits; p->kb_per_split = per; p->stages = stages;
        p->splits_asked = s.k_splits != 0u;
        p->ws_pitch = k / 16u < 16u * lexb::MQ_WS_GROUP ? k / 16u : 16u * lexb::MQ_WS_GROUP;
        // In order by default, as the reference's launches are (crates/lex-cuda/src/device.rs:629-672): wq/ws are
        // loaded ahead of the stream's order only when the caller declares them constant or a step list shows
        // that nothing in flight writes them (ListProof); never when the caller says they may change.
        p->flags = 0u;
        // The blocks of a row tile are a cluster and add up its splits there, where the device holds all of the launch's clusters at
        // once (they are packed less tightly than blocks); else, and with a split that the caller gives, through a workspace.
        if (splits > 1u && !s.k_splits && held_clusters(g, splits) >= tiles && env_u32("LEXB_CLUSTER_SPLIT", 1u) != 0u) p->cluster = splits;
        if (splits > 1u && p->cluster == 1u) {
            // partial products [splits][m][n], then one arrival counter per row tile (zero between launches)
            const size_t pbytes = sizeof(float) * splits * static_cast<size_t>(m) * n;
            cudaError_t e = x_malloc(&p->partial, pbytes + sizeof(uint32_t) * tiles);
            // cleared on the launch stream and waited for: a launch on any stream may follow at once
            if (e == cudaSuccess) e = cudaMemsetAsync(reinterpret_cast<char*>(p->partial) + pbytes, 0, sizeof(uint32_t) * tiles, g->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
            if (e != cudaSuccess) return bail(fail(LEXB_ERR_CUDA, "allocating the split-K workspace: %s", cudaGetErrorString(e)));
        }
        // From 5 tokens on the digit rows are derived once per launch by a small kernel ahead of this one
        // (each block deriving them itself is what bounds the kernel there); LEXB_MQ_PRE=0/1 forces either way.
        // (past 16 tokens there is no in-block path.)  Of int16 activations every value is widened in both walks over them, all
        // of a token for its magnitude and the block's own K range for the digits, so up to 4 tokens the length of the two
        // decides: in the block against ahead, quant16 and product a call, 28672x4096 at t = 1 / 2 / 3 / 4: -2.5 / -0.9 / +0.8 /
        // +2.0 us (lengths 32 to 128), 5120x17408: -1.5 / +0.2 / +1.3 / +2.3 (91 to 364), 4096x4096: -1.9 to -1.1 (20 to 80).
        p->x_q16 = t_plan_q16;
        const uint32_t walk = m * (kb_all + per);
        const bool ahead = m > 4u || (p->x_q16 && m > 1u && walk > (m == 2u ? 150u : 95u));
        p->mq_pre = m > 16u || env_u32("LEXB_MQ_PRE", ahead ? 1u : 0u) != 0;
        if (p->mq_pre) {
            cudaError_t e = x_malloc(&p->pre_buf, lexb::matmul_q_pre_bytes(m, k));
            if (e != cudaSuccess) return bail(fail(LEXB_ERR_CUDA, "allocating the digit-row buffers: %s", cudaGetErrorString(e)));
            int erc = encode_2d(p, &p->pre_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, p->pre_buf, k / 2u, 8u * m, 128u, 8u * m,
                                CU_TENSOR_MAP_SWIZZLE_128B, "digit rows");
            if (erc) return bail(erc);
        }
        p->grid = tiles * splits;
        p->threads = p->mq_pre ? 32u * (2u + lexb::MQ_SCALE_WARPS) : lexb::MQ_THREADS;
        p->smem = lexb::matmul_q_smem_bytes(m, stages);
        p->tm = m;
        if (p->entry[0] == 0)
            snprintf(p->entry, sizeof p->entry, "%s_%u_%u_%u_%u_%u_%u", stem, m, n, k, m, lexb::MQ_ROWS, lexb::MQ_STAGE_K);
    } else if (kernel == KERNEL_TCGEN05) {
        if (n % lexb::GEMM_TN) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4: bn = %u does not divide n = %u", lexb::GEMM_TN, n));
        if (k % lexb::GEMM_BK) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4: bk = %u does not divide k = %u", lexb::GEMM_BK, k));
        uint32_t tm = s.tm;
        if (!tm) {
            const uint32_t tiles = (m + 255u) / 256u;
            tm = round_up((m + tiles - 1u) / tiles, 16u);
        }
        if (tm < 16 || tm > 256 || tm % 16) return bail(fail(LEXB_ERR_ARG, "tm = %u is not a multiple of 16 in [16, 256]", tm));
        const uint32_t stage_bytes = lexb::gemm_stage_bytes(tm);
        uint32_t max_stages = 0;
        while (max_stages < 12 && lexb::gemm_smem_bytes(tm, max_stages + 1) <= g->smem_optin) max_stages++;
        if (max_stages < 2) return bail(fail(LEXB_ERR_UNSUPPORTED, "tm = %u leaves room for %u stages (%u bytes each)", tm, max_stages, stage_bytes));
        // (no more of them than K steps: a short k then leaves room for the next launch's blocks beside this one's)
        uint32_t stages = s.stages ? s.stages : std::min(max_stages, std::max(2u, k / lexb::GEMM_BK));
        if (stages < 2 || stages > max_stages) return bail(fail(LEXB_ERR_ARG, "stages = %u outside [2, %u] for tm = %u", stages, max_stages, tm));
        // two alternating accumulators whenever they fit the 512 columns of TMEM
        const uint32_t n_acc = 2;
        uint32_t cols = 32;
        while (cols < n_acc * tm) cols *= 2;
        p->tm = tm; p->stages = stages; p->tmem_cols = cols; p->n_acc = n_acc; p->m_tiles = (m + tm - 1) / tm;
        p->grid = p->m_tiles * (n / lexb::GEMM_TN);
        p->threads = lexb::GEMM_THREADS;
        p->smem = lexb::gemm_smem_bytes(tm, stages);
        snprintf(p->entry, sizeof p->entry, "%s_%u_%u_%u_%u_%u_%u", stem, m, n, k, tm, lexb::GEMM_TN, lexb::GEMM_BK);
    } else if (kernel == KERNEL_TCGEN05_PAIR) {
        if (n % lexb::GEMM_TN) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4 (pair): %u rows per CTA do not divide n = %u", lexb::GEMM_TN, n));
        if (k % lexb::PAIR_RAW_K) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4 (pair): the packed-weight block of %u columns does not divide k = %u", lexb::PAIR_RAW_K, k));
        // Tiles of 512 tokens (two blocks of 256: each weight decoded once for 512 tokens), 256, 128 or 64 (one block;
        // the MMAs' N shrinks with it, the decode per tile does not); tm asks for one of them at any m
        if (s.tm && s.tm != 64u && s.tm != 128u && s.tm != 256u && s.tm != 512u)
            return bail(fail(LEXB_ERR_ARG, "tm = %u: the two-CTA kernel's tiles hold 64, 128, 256 or 512 tokens", s.tm));
        p->tm = s.tm ? s.tm : (m > 256u ? 512u : m > 128u ? 256u : m > 64u ? 128u : 64u);
        p->tok_blocks = p->tm == 512u ? 2u : 1u;
        p->flags = env_u32("LEXB_COLLECTOR", 0) ? 1u : 0u; p->tmem_cols = lexb::PAIR_TMEM_COLS; p->n_acc = 1;
        p->m_tiles = (m + p->tm - 1) / p->tm;
        const uint32_t n_pairs = (n + 2u * lexb::GEMM_TN - 1) / (2u * lexb::GEMM_TN);
        // Two ways to fill the SM pairs when whole tiles fill them badly (few tiles, or a short last wave).  Split K:
        // each split takes whole blocks of 256 columns (PairPrices' `least` of them, or more) and leaves a partial product, summed by a
        // second launch or within a cluster.  Smaller tiles: more of them; every weight is decoded once per tile of tokens, but a tile's
        // partial product and its store shrink with it and fewer splits are needed.  (Below 256 tokens a K step
        // costs about the same: it is the decode that bounds it, not the MMAs.)
        // Every (tile, splits) pair is priced (PairPrices), the cheapest wins; a smaller tile or a further split must win by 2 %.
        const uint32_t sm_pairs = static_cast<uint32_t>(g->prop.multiProcessorCount) / 2u;
        const uint32_t raw_blocks = k / lexb::PAIR_RAW_K;
        uint32_t splits = s.k_splits ? s.k_splits : 1u;
        // The parts of K are summed in a cluster of their pairs where the device holds the clusters of all tiles at once - they are
        // packed less tightly than pairs, and a second wave costs more than the reduction launch (m = 201, 6144 x 4096 in 3 parts:
        // 24 clusters of 6, 18.2 us with the launch, 31.3 in clusters; in 2 parts 19.9 and 18.0) - and for tiles of up to 256
        // tokens: those of 512 would take two turns of shared memory (512 x 5120 x 17408 in 3 parts: 84.0 and 86.5).  A split
        // that the caller gives goes through the workspace.
        auto in_cluster = [&](uint32_t tile_tokens, uint32_t tiles, uint32_t parts) {
            return parts > 1u && parts <= lexb::PAIR_CLUSTER_SPLITS && tile_tokens <= 256u && tiles <= held_clusters(g, 2u * parts);
        };
        {
            const PairPrices& price = pair_prices(m, n, k);
            auto model = [&](uint32_t ti, uint32_t c, uint32_t* eff_out) {
                const uint32_t tt = 512u >> ti;
                const uint32_t mt = (m + tt - 1u) / tt;
                const uint32_t rbs = (raw_blocks + c - 1u) / c, eff = (raw_blocks + rbs - 1u) / rbs;
                const double waves = static_cast<double>((mt * n_pairs * eff + sm_pairs - 1u) / sm_pairs);
                const double mb = static_cast<double>(m) * n * 4e-6;                      // of y
                double us = price.start + waves * (rbs * 4.0 * price.kstep[ti] + price.wave[ti]);
                if (eff == 1u) us += price.store * mb;
                else if (!s.k_splits && in_cluster(tt, mt * n_pairs, eff)) us += price.cluster + (price.cluster_mb * eff + price.store) * mb;
                else us += price.reduce + price.reduce_mb * eff * mb;
                *eff_out = eff;
                return us;
            };
            double best = 1e30;
            uint32_t best_tt = p->tm, best_c = splits;
            for (uint32_t ti = 0; ti < 4u; ti++) {
                const uint32_t tt = 512u >> ti;
                if (s.tm ? tt != s.tm : (tt != 64u && tt / 2u >= m)) continue;      // the caller's tile; or no tile more than half empty
                for (uint32_t c = 1; c <= 8u && (c == 1u || raw_blocks / c >= price.least); c++) {
                    if (s.k_splits && c != s.k_splits) continue;                    // the caller fixed the splits
                    uint32_t eff = 0;
                    const double us = model(ti, c, &eff);
                    if (eff != c && !s.k_splits) continue;                          // the same plan as a smaller c
                    if (us < best * 0.98) {
                        best = us;
                        best_tt = tt;
                        best_c = c;
                    }
                }
            }
            p->us = best;
            splits = best_c;
            p->tm = best_tt;
            p->tok_blocks = best_tt == 512u ? 2u : 1u;
            p->m_tiles = (m + p->tm - 1u) / p->tm;
        }
        p->x_rows = p->tm == 512u ? lexb::PAIR_XBLK_ROWS : p->tm / 2u;
        // packed-weight blocks in flight: 2; 5 with tiles of 128 tokens or fewer, whose decode takes every second block (two more
        // than the W ring's 3 stages: pair_paired), or 3 beside ring depths that the caller gives
        const uint32_t raw_stages = env_u32("LEXB_RAWSTAGES", p->tm > 128u ? lexb::PAIR_RAW_STAGES : s.stages || s.w_stages ? 3u : 5u);
        p->raw_stages = raw_stages;
        if (splits < 1u || splits > raw_blocks) return bail(fail(LEXB_ERR_ARG, "k_splits = %u outside [1, %u]", splits, raw_blocks));
        // Ring depths.  Tiles of 512 tokens: x ring of 4 stages of 32 KiB, W ring of 3 of 16 KiB, two packed-weight
        // blocks: 212 KiB; their K step is bound by the MMAs.  Smaller tiles: a K step's MMAs take half as long or
        // less and the shared-memory pipe would set the pace, so the decoded W tiles go to tensor memory (the columns
        // behind the accumulator: 256 with tiles of 256 tokens, 384 below; 32 columns per K step) and the MMAs read
        // them from there.  A ring stage then holds two K steps (x 2 x 16 KiB with 256 tokens, W 64 columns; x ring of
        // 4, W ring of 4 or 6) or, with tiles of 128 tokens or fewer, a whole block of four (x ring of 3, W ring of 3),
        // and the MMA warp waits and commits once per stage.  Depths the caller gives that do not fit that way are
        // taken as stages of one K step (at most 8 W stages in tensor memory); more than 8 W stages, or
        // LEXB_WTMEM=0, put the W ring in shared memory (x 6, W 5 by default).
        const bool w_tmem = p->tok_blocks == 1u && s.w_stages <= 8u && env_u32("LEXB_WTMEM", 1u) != 0u;
        uint32_t k_sub = w_tmem ? env_u32("LEXB_KSUB", p->x_rows <= 64u ? 4u : 2u) : 1u;
        if (k_sub != 1u && k_sub != 2u && k_sub != 4u) k_sub = 1u;
        const uint32_t w_cols = p->x_rows <= 64u ? 384u : 256u;             // TMEM columns behind the accumulator
        const uint32_t w_max = k_sub ? w_cols / (32u * k_sub) : 0u;
        if (k_sub > 1u && (s.w_stages > w_max ||
                            lexb::pair_smem_bytes(1u, s.stages ? s.stages : (k_sub == 4u ? 2u : 4u), 2u, raw_stages, true, k_sub, p->x_rows) > g->smem_optin))
            k_sub = 1u;
        const uint32_t stages = s.stages ? s.stages : (p->tok_blocks == 2u ? 4u : k_sub == 4u ? (p->x_rows == 128u ? 2u : 3u) : k_sub == 2u ? 4u : w_tmem ? 8u : 6u);
        const uint32_t w_stages = s.w_stages ? s.w_stages : (p->tok_blocks == 2u ? 3u : k_sub >= 2u ? w_cols / (32u * k_sub) : w_tmem ? 8u : 5u);
        const uint32_t need = lexb::pair_smem_bytes(p->tok_blocks, stages, w_stages, raw_stages, w_tmem, k_sub, p->x_rows);
        if (stages < 2 || w_stages < 2 || raw_stages < 2 || need > g->smem_optin)
            return bail(fail(LEXB_ERR_ARG, "stages = %u with w_stages = %u and %u packed-weight blocks need %u bytes of shared memory (limit %zu)",
                             stages, w_stages, raw_stages, need, g->smem_optin));
        p->k_sub = k_sub;
        p->stages = stages; p->w_stages = w_stages;
        if (w_tmem) p->flags |= 4u;
        const uint32_t tiles_final = p->m_tiles * n_pairs;
        const uint32_t rb_per_split = (raw_blocks + splits - 1u) / splits;
        splits = (raw_blocks + rb_per_split - 1u) / rb_per_split;          // no empty split
        p->k_splits = splits;
        p->kb_per_split = rb_per_split * (lexb::PAIR_RAW_K / lexb::GEMM_BK);
        // (a block's sums go where its rings were)
        p->cluster_split = !s.k_splits && in_cluster(p->tm, tiles_final, splits) && env_u32("LEXB_CLUSTER_SPLIT", 1u) != 0u &&
                           lexb::pair_ring_bytes(p->tok_blocks, stages, w_stages, raw_stages, w_tmem, k_sub, p->x_rows) >= p->tm * 512u;
        p->partial_borrowed = splits > 1u && t_plan_partial;
        if (p->partial_borrowed) {
            p->partial = t_plan_partial;
        } else if (splits > 1u) {
            cudaError_t e = x_malloc(&p->partial, sizeof(float) * splits * static_cast<size_t>(m) * n);
            if (e != cudaSuccess) return bail(fail(LEXB_ERR_CUDA, "allocating the split-K workspace: %s", cudaGetErrorString(e)));
        }
        // From host memory: y leaves at 55 GB/s, 10 to 20 times slower than it is made, so it should start to leave early.
        // Where one row of tiles fills at least half of the machine, a part's launch takes less time than its
        // copy out and only the first part's copy in and launch are waited for.
        if (!s.tm && !s.stages && !s.w_stages && !s.k_splits && m >= 192u && 2u * n_pairs >= sm_pairs)
            p->host_part = round_up((m + lexb_gpu::HOST_PARTS - 1u) / lexb_gpu::HOST_PARTS, 64u);
        p->grid = 2u * tiles_final * splits;
        p->threads = lexb::PAIR_THREADS;
        p->smem = need;
        snprintf(p->entry, sizeof p->entry, "%s_%u_%u_%u_%u_%u_%u", stem, m, n, k, p->tm, 2u * lexb::GEMM_TN, lexb::GEMM_BK);
    } else {
        if (n % lexb::MV_ROWS) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4 (matvec): %u rows per block do not divide n = %u", lexb::MV_ROWS, n));
        if (k % 32u) return bail(fail(LEXB_ERR_SHAPE, "gemm_fp4 (matvec): 32 does not divide k = %u", k));
        if (s.kc % lexb::MV_ROUND) return bail(fail(LEXB_ERR_ARG, "kc = %u is not a multiple of %u", s.kc, lexb::MV_ROUND));
        auto held = [&](uint32_t c, uint32_t warps, uint32_t sm_warps, uint32_t smem) {
            return matvec_clusters(matvec_kernel(m, k, sm_warps), c, 32u * warps, smem);
        };
        MatvecShape v;
        if (!plan_matvec(m, n, k, s.kc, static_cast<uint32_t>(g->prop.multiProcessorCount), g->smem_optin, g->prop.sharedMemPerMultiprocessor, held, &v))
            return bail(fail(LEXB_ERR_UNSUPPORTED, "kc = %u needs %u bytes of shared memory", s.kc, lexb::matvec_smem_bytes(m, s.kc, 4, 8, m <= 8u)));
        p->mv = v;
        p->kc = v.kc; p->threads = 32u * v.warps; p->smem = v.smem; p->grid = v.clusters * v.cluster;
        snprintf(p->entry, sizeof p->entry, "%s_%u_%u_%u_%u_%u_%u", stem, m, n, k, m, lexb::MV_ROWS, lexb::MV_SLICE);
    }
    if (!s.kernel && !s.tm && !s.stages && !s.kc && !s.w_stages && !s.k_splits && env_u32("LEXB_FEW", 1u) && (rc = plan_few(g, p))) return bail(rc);
    *out = p;
    return LEXB_OK;
}

int lexb_matmul_fp4_plan(lexb_gpu* g, uint32_t t, uint32_t n_out, uint32_t n_in, int residual, int x_half,
                         const lexb_sched* sched, lexb_pipeline** out) {
    if (!out) return fail(LEXB_ERR_ARG, "lexb_matmul_fp4_plan: null out");
    *out = nullptr;
    lexb_sched s{};
    if (sched) s = *sched;
    s.kernel = KERNEL_MATMUL_Q;
    int rc = lexb_gemm_fp4_plan(g, t, n_out, n_in, residual, &s, out);
    if (rc) return rc;
    // the reference's name for the program: matvec / matmul{t}, layout tag, rows x columns, _res, _xh
    // (crates/lex-front/src/llama.rs:416-422, :459-465)
    char tag[16];
    if (t == 1) snprintf(tag, sizeof tag, "matvec");
    else snprintf(tag, sizeof tag, "matmul%u", t);
    (*out)->x_f32 = !x_half;
    snprintf((*out)->entry, sizeof (*out)->entry, "%s_nvfp4_%ux%u%s%s", tag, n_out, n_in, residual ? "_res" : "", x_half ? "_xh" : "");
    return LEXB_OK;
}

int lexb_matmul_int8_plan(lexb_gpu* g, uint32_t t, uint32_t n_out, uint32_t n_in, int residual, const lexb_sched* sched,
                          lexb_pipeline** out) {
    if (!out) return fail(LEXB_ERR_ARG, "lexb_matmul_int8_plan: null out");
    *out = nullptr;
    lexb_sched s{};
    if (sched) s = *sched;
    s.kernel = KERNEL_MATMUL_Q;
    t_plan_q16 = true;
    int rc = lexb_gemm_fp4_plan(g, t, n_out, n_in, residual, &s, out);
    t_plan_q16 = false;
    if (rc) return rc;
    // the reference's name for the kernel (crates/lex-msl/src/int8.rs:129-132)
    snprintf((*out)->entry, sizeof (*out)->entry, "matmul_int8_%ux%ux%u%s", t, n_out, n_in, residual ? "_res" : "");
    return LEXB_OK;
}

int lexb_quant16(lexb_gpu* g, uint32_t m, uint32_t k, int x_half, const lexb_buffer* x, lexb_buffer* xq, lexb_buffer* xs) {
    int rc = use(g);
    if (rc) return rc;
    if (m == 0 || k == 0 || k % 32u) return fail(LEXB_ERR_SHAPE, "quant16: %u inputs are not whole groups of 32", k);
    const size_t mm = m, kk = k;
    if ((rc = check_buf(x, g, mm * kk * (x_half ? 2 : 4), "x"))) return rc;
    if ((rc = check_buf(xq, g, mm * kk * 2, "xq"))) return rc;
    if ((rc = check_buf(xs, g, mm * (kk / 16) * 4, "xs"))) return rc;
    const size_t groups = mm * kk / 16;
    const uint32_t blocks = static_cast<uint32_t>((groups + 255) / 256);
    INJECT_LAUNCH();
    PdlLaunch launch(g, blocks, 256, g->pdl);
    const void* xp = x->ptr;
    short* q = static_cast<short*>(xq->ptr);
    float* s = static_cast<float*>(xs->ptr);
    if (x_half) CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, quant16_kernel<true>, xp, q, s, groups));
    else CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, quant16_kernel<false>, xp, q, s, groups));
    CUDA_TRY(cudaGetLastError());
    return LEXB_OK;
}

void lexb_pipeline_free(lexb_pipeline* p) {
    if (!p) return;
    for (lexb_pipeline* part : p->host_pipes) lexb_pipeline_free(part);
    delete p->few;
    if (p->partial || p->pre_buf) free_on(p->device, {p->partial_borrowed ? nullptr : p->partial, p->pre_buf});
    delete p;
}

int lexb_pipeline_describe(const lexb_pipeline* p, lexb_lowered* out) {
    if (!p || !out) return fail(LEXB_ERR_ARG, "lexb_pipeline_describe: null argument");
    memset(out, 0, sizeof *out);
    snprintf(out->entry, sizeof out->entry, "%s", p->entry);
    out->grid = p->grid;
    out->grid2 = 1;
    out->threads = p->threads;
    out->threadgroup_bytes = p->smem;
    out->nbind = (p->residual ? 6 : 5) + (p->x_q16 ? 1 : 0);
    out->writes[out->nbind - 1] = 1;
    out->kernel = p->kernel;
    out->m = p->m; out->n = p->n; out->k = p->k; out->residual = p->residual;
    if (p->kernel == KERNEL_MATMUL_Q) {
        out->bm = p->m; out->bn = lexb::MQ_ROWS; out->bk = lexb::MQ_STAGE_K; out->stages = p->stages;
        out->k_splits = p->k_splits;
        out->scratch_bytes = p->partial ? sizeof(float) * p->k_splits * static_cast<uint64_t>(p->m) * p->n : 0;
    } else if (p->kernel == KERNEL_TCGEN05 || p->kernel == KERNEL_TCGEN05_PAIR) {
        out->bm = p->tm; out->bn = p->kernel == KERNEL_TCGEN05_PAIR ? 2u * lexb::GEMM_TN : lexb::GEMM_TN;
        out->bk = lexb::GEMM_BK; out->stages = p->stages;
        out->k_splits = p->k_splits;
        out->scratch_bytes = p->partial ? sizeof(float) * p->k_splits * static_cast<uint64_t>(p->m) * p->n : 0;
    } else {
        out->bm = p->m; out->bn = lexb::MV_ROWS; out->bk = lexb::MV_SLICE; out->stages = 1;
    }
    return LEXB_OK;
}

static lexb_route matvec_route(const MatvecShape& v) {
    lexb_route r{};
    r.cluster = v.cluster; r.parts = v.parts; r.groups = v.per; r.kc = v.kc;
    r.blocks = v.clusters * v.cluster; r.threads = 32u * v.warps;
    return r;
}

int lexb_pipeline_route(const lexb_pipeline* p, lexb_route* out) {
    if (!p || !out) return fail(LEXB_ERR_ARG, "lexb_pipeline_route: null argument");
    *out = lexb_route{};
    const lexb_pipeline* l = p->few ? p->few : p;
    if (l->kernel == KERNEL_MATVEC) *out = matvec_route(l->mv);
    else {
        out->cluster = l->cluster_split ? l->k_splits : l->cluster;
        out->blocks = l->grid; out->threads = l->threads;
    }
    out->host_part = p->host_part;
    return LEXB_OK;
}

int lexb_matvec_route(uint32_t sms, uint32_t m, uint32_t n, uint32_t k, uint32_t kc, lexb_route* out) {
    if (!out) return fail(LEXB_ERR_ARG, "lexb_matvec_route: null out");
    *out = lexb_route{};
    if (sms == 0 || m == 0 || m > 16u || n == 0 || n % lexb::MV_ROWS || k == 0 || k % 32u || kc % lexb::MV_ROUND)
        return fail(LEXB_ERR_SHAPE, "the matvec takes m <= 16, n %% %u == 0, k %% 32 == 0, kc %% %u == 0; not m=%u n=%u k=%u kc=%u", lexb::MV_ROWS, lexb::MV_ROUND, m, n, k, kc);
    const size_t smem_optin = 227u * 1024u, smem_sm = 228u * 1024u;
    auto held = [&](uint32_t c, uint32_t warps, uint32_t sm_warps, uint32_t smem) {      // (about four fifths: see matvec_clusters)
        return sms * std::min(static_cast<uint32_t>(smem_sm / (smem + 1024u)), sm_warps / warps) * 4u / (5u * c);
    };
    MatvecShape v;
    if (!plan_matvec(m, n, k, kc, sms, smem_optin, smem_sm, held, &v)) return fail(LEXB_ERR_UNSUPPORTED, "kc = %u leaves no room in shared memory", kc);
    *out = matvec_route(v);
    return LEXB_OK;
}

int lexb_gemm_fp4_launch(lexb_gpu* g, const lexb_pipeline* p, const lexb_buffer* x, const lexb_buffer* wq,
                         const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r, lexb_buffer* y) {
    int rc = use(g);
    if (rc) return rc;
    return launch_one(g, p, x, wq, ws, wg, r, y);
}

int lexb_gemm_fp4_launch_gather(lexb_gpu* g, const lexb_pipeline* p, const lexb_buffer* x, const lexb_buffer* wq,
                                const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r, void* const* y_of_rank,
                                uint32_t world, uint32_t n_total, uint32_t n0) {
    int rc = use(g);
    if (rc) return rc;
    if (!p || !y_of_rank) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_launch_gather: null argument");
    if (world == 0 || world > lexb::GATHER_MAX) return fail(LEXB_ERR_ARG, "world = %u outside [1, %u]", world, lexb::GATHER_MAX);
    if (n_total % 4u || n0 % 4u || static_cast<uint64_t>(n0) + p->n > n_total)
        return fail(LEXB_ERR_ARG, "columns [%u, %u) do not fit a gathered row of %u", n0, n0 + p->n, n_total);
    lexb::GatherDst gd{};
    gd.world = world; gd.n_total = n_total; gd.n0 = n0; gd.n_local = p->n;
    for (uint32_t d = 0; d < world; d++) {
        if (!y_of_rank[d] || (reinterpret_cast<uintptr_t>(y_of_rank[d]) & 15u))
            return fail(LEXB_ERR_ARG, "y of rank %u is null or not 16-byte aligned", d);
        gd.y[d] = static_cast<float*>(y_of_rank[d]);
    }
    return launch_one(g, p, x, wq, ws, wg, r, nullptr, &gd);
}

int lexb_gemm_fp4_silu_launch(lexb_gpu* g, const lexb_pipeline* p, const lexb_buffer* x, const lexb_buffer* wq,
                              const lexb_buffer* ws, const lexb_buffer* wg, lexb_buffer* act) {
    int rc = use(g);
    if (rc) return rc;
    if (!act) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_silu_launch: null act");
    return launch_one(g, p, x, wq, ws, wg, nullptr, nullptr, nullptr, nullptr, Order{}, act);
}

int lexb_gemm_fp4_silu_launch_gather(lexb_gpu* g, const lexb_pipeline* p, const lexb_buffer* x, const lexb_buffer* wq,
                                     const lexb_buffer* ws, const lexb_buffer* wg, void* const* act_of_rank, uint32_t world,
                                     uint32_t n_total, uint32_t n0) {
    int rc = use(g);
    if (rc) return rc;
    if (!p || !act_of_rank) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_silu_launch_gather: null argument");
    if (world == 0 || world > lexb::GATHER_MAX) return fail(LEXB_ERR_ARG, "world = %u outside [1, %u]", world, lexb::GATHER_MAX);
    if (n_total % 8u || n0 % 8u || static_cast<uint64_t>(n0) + p->n > n_total)
        return fail(LEXB_ERR_ARG, "interleaved rows [%u, %u) do not fit %u rows in all", n0, n0 + p->n, n_total);
    lexb::GatherDst gd{};
    gd.world = world; gd.n_total = n_total; gd.n0 = n0; gd.n_local = p->n; gd.silu = 1u;
    for (uint32_t d = 0; d < world; d++) {
        if (!act_of_rank[d] || (reinterpret_cast<uintptr_t>(act_of_rank[d]) & 15u))
            return fail(LEXB_ERR_ARG, "act of rank %u is null or not 16-byte aligned", d);
        gd.y[d] = static_cast<float*>(act_of_rank[d]);
    }
    return launch_one(g, p, x, wq, ws, wg, nullptr, nullptr, &gd);
}

int lexb_interleave_rows(lexb_gpu* g, const lexb_buffer* a, const lexb_buffer* b, size_t rows, size_t row_bytes, lexb_buffer* out) {
    int rc = use(g);
    if (rc) return rc;
    if (!a || !b || !out) return fail(LEXB_ERR_ARG, "lexb_interleave_rows: null buffer");
    if (rows == 0 || row_bytes == 0) return fail(LEXB_ERR_SHAPE, "lexb_interleave_rows: empty extent");
    if (a->bytes < rows * row_bytes || b->bytes < rows * row_bytes || out->bytes < 2 * rows * row_bytes)
        return fail(LEXB_ERR_ARG, "lexb_interleave_rows: %zu rows of %zu bytes do not fit the buffers", rows, row_bytes);
    char* o = static_cast<char*>(out->ptr);
    CUDA_TRY_AT(SITE_COPY, cudaMemcpy2DAsync(o, 2 * row_bytes, a->ptr, row_bytes, row_bytes, rows, cudaMemcpyDeviceToDevice, g->stream));
    CUDA_TRY_AT(SITE_COPY, cudaMemcpy2DAsync(o + row_bytes, 2 * row_bytes, b->ptr, row_bytes, row_bytes, rows, cudaMemcpyDeviceToDevice, g->stream));
    return LEXB_OK;
}

int lexb_gemm_fp4_enqueue_host(lexb_gpu* g, const lexb_pipeline* p, const void* x_host, lexb_buffer* x_dev,
                               const lexb_buffer* wq, const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r,
                               lexb_buffer* y_dev, void* y_host) {
    int rc = use(g);
    if (rc) return rc;
    if (!p || !x_host || !y_host || !x_dev || !y_dev) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_enqueue_host: null argument");
    if (p->x_q16) return fail(LEXB_ERR_UNSUPPORTED, "lexb_gemm_fp4_enqueue_host takes f16 or f32 activations; quantise on the device (lexb_quant16) and launch a step");
    const size_t xb = static_cast<size_t>(p->m) * p->k * (p->x_f32 ? 4 : 2), yb = static_cast<size_t>(p->m) * p->n * 4;
    if (x_dev->bytes < xb || y_dev->bytes < yb) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_enqueue_host: staging buffers too small");
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(x_dev->ptr, x_host, xb, cudaMemcpyHostToDevice, g->stream));
    if ((rc = launch_one(g, p, x_dev, wq, ws, wg, r, y_dev))) return rc;
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(y_host, y_dev->ptr, yb, cudaMemcpyDeviceToHost, g->stream));
    return LEXB_OK;
}

static bool is_pinned(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost;
}

// May the call go in parts?  Part 0 of y is stored and copied out before the last part of x is copied in, so nothing the call
// writes (x_dev, y_dev, y_host) may meet anything else it touches, in host memory or on the device (one address space:
// a buffer may wrap mapped host memory).  r and y_dev as one buffer stay in parts: a part reads its own tokens of r only.
// A stream that is being captured keeps the one copy, launch and copy (the wait then fails as it always did).
static bool host_parts_apply(const lexb_gpu* g, const lexb_pipeline* p, const void* x_host, const lexb_buffer* x_dev, const lexb_buffer* wq,
                             const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r, const lexb_buffer* y_dev, const void* y_host) {
    if (!p->host_part || p->gpu != g || x_dev->gpu != g || y_dev->gpu != g || !wq || !ws || !wg || g->d_trace) return false;
    const size_t m = p->m, n = p->n, k = p->k;
    auto range = [](const void* at, size_t bytes) { return Range{static_cast<const char*>(at), static_cast<const char*>(at) + bytes}; };
    const Range written[3] = {range(x_dev->ptr, m * k * 2), range(y_dev->ptr, m * n * 4), range(y_host, m * n * 4)};
    const Range read[5] = {range(x_host, m * k * 2), range(wq->ptr, n * k / 2), range(ws->ptr, n * k / 16), range(wg->ptr, n * 4),
                           r ? range(r->ptr, m * n * 4) : Range{nullptr, nullptr}};
    for (uint32_t w = 0; w < 3u; w++) {
        for (uint32_t v = 0; v < w; v++)
            if (meet(written[w], written[v])) return false;
        for (uint32_t v = 0; v < 5u; v++)
            if (meet(written[w], read[v]) && !(w == 1u && v == 4u && r->ptr == y_dev->ptr)) return false;
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(g->stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    return is_pinned(x_host) && is_pinned(y_host);
}

// The call below in parts of p->host_part tokens: the copies in, the launches and the copies out on three streams, ordered
// by events, so that a part is copied out while the next is copied in and multiplied.  A part has the whole's K split, in the
// whole's workspace, so y's bits do not depend on the way taken.  The launch stream waits for the last
// copy, as if it had made them all.  Pinned memory only: copies of pageable memory do not return before they are made.
static int run_host_in_parts(lexb_gpu* g, const lexb_pipeline* p, const void* x_host, lexb_buffer* x_dev, const lexb_buffer* wq,
                             const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r, lexb_buffer* y_dev, void* y_host) {
    std::lock_guard<std::mutex> hold(g->host.lock);
    lexb_gpu::HostPath& h = g->host;
    if (!h.out) {
        for (cudaEvent_t& e : h.event)
            if (!e) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        if (!h.in) CUDA_TRY(cudaStreamCreateWithFlags(&h.in, cudaStreamNonBlocking));
        CUDA_TRY(cudaStreamCreateWithFlags(&h.out, cudaStreamNonBlocking));
    }
    auto issue = [&]() -> int {
        int rc;
        CUDA_TRY(cudaEventRecord(h.event[0], g->stream));
        CUDA_TRY(cudaStreamWaitEvent(h.in, h.event[0], 0));
        uint32_t i = 0;
        for (uint32_t t0 = 0; t0 < p->m; t0 += p->host_part, i++) {
            const uint32_t tokens = std::min(p->host_part, p->m - t0);
            lexb_pipeline*& part = p->host_pipes[tokens == p->host_part ? 0 : 1];
            {
                std::lock_guard<std::mutex> plan(p->host_lock);
                if (!part) {
                    lexb_sched s{};
                    s.kernel = KERNEL_TCGEN05_PAIR;
                    s.k_splits = p->k_splits;                            // the sums of one launch of the whole, bit for bit
                    s.flags = (p->w_const ? LEXB_SCHED_WEIGHTS_CONSTANT : 0u) | (p->w_volatile ? LEXB_SCHED_WEIGHTS_MAY_CHANGE : 0u);
                    t_plan_partial = p->partial;                         // (one part at a time, in the launch stream's order)
                    rc = lexb_gemm_fp4_plan(g, tokens, p->n, p->k, p->residual, &s, &part);
                    t_plan_partial = nullptr;
                    if (rc) return rc;
                }
            }
            const size_t xo = static_cast<size_t>(t0) * p->k * 2, xb = static_cast<size_t>(tokens) * p->k * 2;
            const size_t yo = static_cast<size_t>(t0) * p->n * 4, yb = static_cast<size_t>(tokens) * p->n * 4;
            lexb_buffer xd{g, static_cast<char*>(x_dev->ptr) + xo, xb, false}, yd{g, static_cast<char*>(y_dev->ptr) + yo, yb, false}, rd{};
            if (r) {
                if ((rc = check_buf(r, g, yo + yb, "r"))) return rc;
                rd = lexb_buffer{g, static_cast<char*>(r->ptr) + yo, yb, false};
            }
            CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(xd.ptr, static_cast<const char*>(x_host) + xo, xb, cudaMemcpyHostToDevice, h.in));
            CUDA_TRY(cudaEventRecord(h.event[2u + 2u * i], h.in));
            CUDA_TRY(cudaStreamWaitEvent(g->stream, h.event[2u + 2u * i], 0));
            if ((rc = launch_one(g, part, &xd, wq, ws, wg, r ? &rd : nullptr, &yd))) return rc;
            CUDA_TRY(cudaEventRecord(h.event[3u + 2u * i], g->stream));
            CUDA_TRY(cudaStreamWaitEvent(h.out, h.event[3u + 2u * i], 0));
            CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(static_cast<char*>(y_host) + yo, yd.ptr, yb, cudaMemcpyDeviceToHost, h.out));
        }
        CUDA_TRY(cudaEventRecord(h.event[1], h.out));
        CUDA_TRY(cudaStreamWaitEvent(g->stream, h.event[1], 0));
        return LEXB_OK;
    };
    const int rc = issue();
    if (rc) {                                                            // nothing of a call that failed stays in flight
        cudaStreamSynchronize(h.in);
        cudaStreamSynchronize(g->stream);
        cudaStreamSynchronize(h.out);
    }
    return rc;
}

int lexb_gemm_fp4_run_host(lexb_gpu* g, const lexb_pipeline* p, const void* x_host, lexb_buffer* x_dev,
                           const lexb_buffer* wq, const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r,
                           lexb_buffer* y_dev, void* y_host) {
    int rc = use(g);
    if (rc) return rc;
    if (!p || !x_host || !y_host || !x_dev || !y_dev) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_run_host: null argument");
    if (p->x_q16) return fail(LEXB_ERR_UNSUPPORTED, "lexb_gemm_fp4_run_host takes f16 or f32 activations; quantise on the device (lexb_quant16) and launch a step");
    const size_t xb = static_cast<size_t>(p->m) * p->k * (p->x_f32 ? 4 : 2), yb = static_cast<size_t>(p->m) * p->n * 4;
    if (x_dev->bytes < xb || y_dev->bytes < yb) return fail(LEXB_ERR_ARG, "lexb_gemm_fp4_run_host: staging buffers too small");
    if (host_parts_apply(g, p, x_host, x_dev, wq, ws, wg, r, y_dev, y_host)) {
        if ((rc = run_host_in_parts(g, p, x_host, x_dev, wq, ws, wg, r, y_dev, y_host))) return rc;
        CUDA_TRY(cudaStreamSynchronize(g->stream));
        return LEXB_OK;
    }
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(x_dev->ptr, x_host, xb, cudaMemcpyHostToDevice, g->stream));
    if ((rc = launch_one(g, p, x_dev, wq, ws, wg, r, y_dev))) return rc;
    CUDA_TRY_AT(SITE_COPY, cudaMemcpyAsync(y_host, y_dev->ptr, yb, cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_run_launches(lexb_gpu* g, const lexb_step* steps, size_t nsteps, double* cpu_s, double* wall_s) {
    int rc = use(g);
    if (rc) return rc;
    if (!steps && nsteps) return fail(LEXB_ERR_ARG, "lexb_run_launches: null steps");
    const auto t0 = std::chrono::steady_clock::now();
    ListProof proof;
    bool first = true;
    if ((rc = issue_list(g, steps, nsteps, proof, first, nullptr, nsteps == 1))) return rc;
    const auto t1 = std::chrono::steady_clock::now();
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    const auto t2 = std::chrono::steady_clock::now();
    if (cpu_s) *cpu_s = std::chrono::duration<double>(t1 - t0).count();
    if (wall_s) *wall_s = std::chrono::duration<double>(t2 - t0).count();
    return LEXB_OK;
}

int lexb_run_each_timed(lexb_gpu* g, const lexb_step* steps, size_t nsteps, double* seconds_out) {
    int rc = use(g);
    if (rc) return rc;
    if ((!steps || !seconds_out) && nsteps) return fail(LEXB_ERR_ARG, "lexb_run_each_timed: null argument");
    std::vector<cudaEvent_t> ev(nsteps + 1, nullptr);
    auto cleanup = [&]() { for (auto e : ev) if (e) cudaEventDestroy(e); };
    for (auto& e : ev)
        if (cudaEventCreate(&e) != cudaSuccess) { cleanup(); return fail(LEXB_ERR_CUDA, "cudaEventCreate failed"); }
    cudaEventRecord(ev[0], g->stream);
    ListProof proof;
    for (size_t i = 0; i < nsteps; i++) {
        const StepRanges sr = step_ranges(steps[i]);
        Order order;
        order.fence = i == 0;
        order.early_weights = sr.valid && proof.weights_untouched(sr);
        if ((rc = launch_step(g, steps[i], i + 1 < nsteps ? &steps[i + 1] : nullptr, order))) { cleanup(); return rc; }
        if (sr.valid) proof.add(sr);
        cudaEventRecord(ev[i + 1], g->stream);
    }
    cudaError_t e = cudaStreamSynchronize(g->stream);
    if (e != cudaSuccess) { cleanup(); return fail(LEXB_ERR_CUDA, "synchronise: %s", cudaGetErrorString(e)); }
    for (size_t i = 0; i < nsteps; i++) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
        seconds_out[i] = ms * 1e-3;
    }
    cleanup();
    return LEXB_OK;
}

int lexb_list_runs(lexb_gpu* g, const lexb_step* steps, size_t nsteps, uint32_t* run_len_out) {
    int rc = use(g);
    if (rc) return rc;
    if ((!steps || !run_len_out) && nsteps) return fail(LEXB_ERR_ARG, "lexb_list_runs: null argument");
    ListProof proof;
    for (size_t i = 0; i < nsteps;) {
        const size_t len = chain_run(g, steps, nsteps, i, proof);
        const size_t take = len ? len : 1;
        for (size_t e = i; e < i + take; e++) {
            run_len_out[e] = static_cast<uint32_t>(take);
            const StepRanges sr = step_ranges(steps[e]);
            if (sr.valid) proof.add(sr);
        }
        i += take;
    }
    return LEXB_OK;
}

int lexb_time_launches(lexb_gpu* g, const lexb_step* steps, size_t nsteps, uint32_t reps, double* seconds_out) {
    int rc = use(g);
    if (rc) return rc;
    if ((!steps && nsteps) || !seconds_out) return fail(LEXB_ERR_ARG, "lexb_time_launches: null argument");
    cudaEvent_t a, b;
    CUDA_TRY(cudaEventCreate(&a));
    CUDA_TRY(cudaEventCreate(&b));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    cudaEventRecord(a, g->stream);
    ListProof proof;
    bool first = true;
    for (uint32_t r = 0; r < reps; r++) {
        // the list repeats: the step after the last one is the first one again
        const lexb_step* after_last = (r + 1 < reps && nsteps) ? &steps[0] : nullptr;
        if ((rc = issue_list(g, steps, nsteps, proof, first, after_last))) { cudaEventDestroy(a); cudaEventDestroy(b); return rc; }
    }
    cudaEventRecord(b, g->stream);
    cudaError_t e = cudaStreamSynchronize(g->stream);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (e != cudaSuccess) return fail(LEXB_ERR_CUDA, "timing: %s", cudaGetErrorString(e));
    *seconds_out = ms * 1e-3;
    return LEXB_OK;
}

int lexb_status_word(lexb_gpu* g, uint32_t* out) {
    int rc = use(g);
    if (rc) return rc;
    if (!out) return fail(LEXB_ERR_ARG, "lexb_status_word: null out");
    // read and cleared in the launch stream's order, then waited for: the legacy default stream would not be
    // ordered with the library's non-blocking stream
    CUDA_TRY(cudaMemcpyAsync(out, g->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaMemsetAsync(g->d_status, 0, sizeof(uint32_t), g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_trace_enable(lexb_gpu* g, uint32_t max_ctas) {
    int rc = use(g);
    if (rc) return rc;
    if (g->d_trace) {
        CUDA_TRY(cudaFree(g->d_trace));
        g->d_trace = nullptr;
        g->trace_ctas = 0;
    }
    if (max_ctas) {
        CUDA_TRY(x_malloc(&g->d_trace, sizeof(unsigned long long) * 16u * max_ctas));
        CUDA_TRY(cudaMemsetAsync(g->d_trace, 0, sizeof(unsigned long long) * 16u * max_ctas, g->stream));
        CUDA_TRY(cudaStreamSynchronize(g->stream));
        g->trace_ctas = max_ctas;
    }
    return LEXB_OK;
}

int lexb_trace_read(lexb_gpu* g, uint64_t* out, uint32_t ctas) {
    int rc = use(g);
    if (rc) return rc;
    if (!out || !g->d_trace || ctas > g->trace_ctas) return fail(LEXB_ERR_ARG, "lexb_trace_read: tracing is off or the request is too large");
    CUDA_TRY(cudaMemcpyAsync(out, g->d_trace, sizeof(uint64_t) * 16u * ctas, cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_selftest_bounded_wait(lexb_gpu* g, uint32_t limit_us) {
    int rc = use(g);
    if (rc) return rc;
    if (limit_us == 0 || limit_us > 1000000u) return fail(LEXB_ERR_ARG, "limit_us must be in [1, 1000000]");
    const long long cycles = static_cast<long long>(limit_us) * (g->prop.clockRate / 1000);   // clockRate is kHz
    INJECT_LAUNCH();
    bounded_wait_selftest_kernel<<<1, 32, 0, g->stream>>>(g->d_status, cycles);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(g->stream));
    return LEXB_OK;
}

int lexb_dequant_fp4_f16(lexb_gpu* g, uint32_t n, uint32_t k, const lexb_buffer* wq, const lexb_buffer* ws,
                         const lexb_buffer* wg, lexb_buffer* w_f16) {
    int rc = use(g);
    if (rc) return rc;
    if (n == 0 || k == 0 || k % 16u) return fail(LEXB_ERR_SHAPE, "dequant_fp4: group 16 does not divide k = %u", k);
    const size_t nn = n, kk = k;
    if ((rc = check_buf(wq, g, nn * kk / 2, "wq"))) return rc;
    if ((rc = check_buf(ws, g, nn * kk / 16, "ws"))) return rc;
    if ((rc = check_buf(wg, g, nn * 4, "wg"))) return rc;
    if ((rc = check_buf(w_f16, g, nn * kk * 2, "w_f16"))) return rc;
    const size_t groups = nn * kk / 16;
    const uint32_t threads = 256;
    const uint32_t blocks = static_cast<uint32_t>(std::min<size_t>((groups + threads - 1) / threads, static_cast<size_t>(g->prop.multiProcessorCount) * 32u));
    INJECT_LAUNCH();
    dequant_fp4_f16_kernel<<<blocks, threads, 0, g->stream>>>(n, k, static_cast<const uint8_t*>(wq->ptr),
                                                              static_cast<const uint8_t*>(ws->ptr),
                                                              static_cast<const float*>(wg->ptr),
                                                              static_cast<uint16_t*>(w_f16->ptr));
    CUDA_TRY(cudaGetLastError());
    return LEXB_OK;
}

int lexb_gemm_fp4_splitk_static(lexb_gpu* g, uint32_t m, uint32_t n, uint32_t k, uint32_t k_splits, const lexb_buffer* x,
                                const lexb_buffer* wq, const lexb_buffer* ws, const lexb_buffer* wg, const lexb_buffer* r,
                                lexb_buffer* y) {
    int rc = use(g);
    if (rc) return rc;
    if (m < lexb::PAIR_XBLK_ROWS || n == 0 || n % lexb::GEMM_TN || k == 0 || k % lexb::PAIR_RAW_K)
        return fail(LEXB_ERR_SHAPE, "gemm_fp4 (static scratch): needs m >= %u, n %% %u == 0, k %% %u == 0; got m=%u n=%u k=%u",
                    lexb::PAIR_XBLK_ROWS, lexb::GEMM_TN, lexb::PAIR_RAW_K, m, n, k);
    const uint32_t raw_blocks = k / lexb::PAIR_RAW_K;
    if (k_splits < 2u || k_splits > 8u || k_splits > raw_blocks)
        return fail(LEXB_ERR_ARG, "k_splits = %u outside [2, %u]", k_splits, raw_blocks < 8u ? raw_blocks : 8u);
    const uint32_t rb_per_split = (raw_blocks + k_splits - 1u) / k_splits;
    const uint32_t splits = (raw_blocks + rb_per_split - 1u) / rb_per_split;
    const uint64_t need = sizeof(float) * static_cast<uint64_t>(splits) * m * n;
    if (need > LEXB_STATIC_SCRATCH_BYTES)
        return fail(LEXB_ERR_UNSUPPORTED,
                    "gemm_fp4 (static scratch): %u splits of m=%u n=%u need %llu bytes of scratch, the built-in array holds %llu; "
                    "use fewer splits or a planned pipeline",
                    splits, m, n, (unsigned long long)need, (unsigned long long)LEXB_STATIC_SCRATCH_BYTES);
    if (!g->static_scratch) {
        // Once per device, with that device current (use() above): the symbol's name is a host-side
        // stand-in, the kernels need its device address.
        void* p = nullptr;
        CUDA_TRY(cudaGetSymbolAddress(&p, g_splitk_static_scratch));
        g->static_scratch = static_cast<float*>(p);
    }
    // The same launch shape lexb_gemm_fp4_plan builds for the two-CTA kernel, held on the stack.
    lexb_pipeline p;
    p.gpu = g;
    p.kernel = KERNEL_TCGEN05_PAIR;
    p.m = m; p.n = n; p.k = k;
    p.residual = r != nullptr;
    // one block of 256 tokens per tile up to m = 256, two beyond: the shape lexb_gemm_fp4_plan gives the same m
    p.tok_blocks = m > 256u ? 2u : 1u;
    p.tm = p.tok_blocks * 256u; p.stages = 4; p.w_stages = 3; p.tmem_cols = lexb::PAIR_TMEM_COLS; p.n_acc = 1; p.flags = 0;
    p.kc = 0;
    p.m_tiles = (m + p.tm - 1) / p.tm;
    p.k_splits = splits;
    p.kb_per_split = rb_per_split * (lexb::PAIR_RAW_K / lexb::GEMM_BK);
    p.grid = 2u * p.m_tiles * ((n + 2u * lexb::GEMM_TN - 1) / (2u * lexb::GEMM_TN)) * splits;
    p.threads = lexb::PAIR_THREADS;
    p.smem = lexb::pair_smem_bytes(2u, p.stages, p.w_stages);
    if (p.smem > g->smem_optin) return fail(LEXB_ERR_UNSUPPORTED, "the device offers %zu bytes of shared memory, the kernel needs %u", g->smem_optin, p.smem);
    const size_t mm = m, nn = n, kk = k;
    if ((rc = check_buf(x, g, mm * kk * 2, "x"))) return rc;
    if ((rc = check_buf(wq, g, nn * kk / 2, "wq"))) return rc;
    if ((rc = check_buf(ws, g, nn * kk / 16, "ws"))) return rc;
    if ((rc = check_buf(wg, g, nn * 4, "wg"))) return rc;
    if ((rc = check_buf(y, g, mm * nn * 4, "y"))) return rc;
    if (r && (rc = check_buf(r, g, mm * nn * 4, "r"))) return rc;
    CUtensorMap map_x, map_wq, map_ws;      // encoded on the host for this call, not cached
    if ((rc = encode_2d(&p, &map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x->ptr, k, m, lexb::GEMM_BK, lexb::PAIR_XBLK_ROWS,
                        CU_TENSOR_MAP_SWIZZLE_128B, "x")))
        return rc;
    if ((rc = encode_2d(&p, &map_wq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq->ptr, k / 2, n, lexb::PAIR_RAW_K / 2, lexb::GEMM_TN,
                        CU_TENSOR_MAP_SWIZZLE_128B, "wq")))
        return rc;
    if ((rc = encode_2d(&p, &map_ws, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ws->ptr, k / 16, n, lexb::PAIR_RAW_K / 16, lexb::GEMM_TN,
                        CU_TENSOR_MAP_SWIZZLE_NONE, "ws")))
        return rc;
    lexb::GemmArgs a{};
    a.wq = static_cast<const uint8_t*>(wq->ptr);
    a.ws = static_cast<const uint8_t*>(ws->ptr);
    a.wg = static_cast<const float*>(wg->ptr);
    a.r = r ? static_cast<const float*>(r->ptr) : nullptr;
    a.y = static_cast<float*>(y->ptr);
    a.status = g->d_status;
    a.trace = nullptr;
    a.m = m; a.n = n; a.k = k;
    a.tm = p.tm; a.stages = p.stages; a.w_stages = p.w_stages; a.raw_stages = p.raw_stages; a.k_sub = 1; a.x_rows = lexb::PAIR_XBLK_ROWS;
    a.flags = p.tok_blocks == 1u ? 4u : 0u;      // tiles of 256 tokens: W tiles in tensor memory, as the planned pipeline has them
    a.k_splits = splits; a.kb_per_split = p.kb_per_split; a.tok_blocks = p.tok_blocks;
    a.partial = g->static_scratch;          // every element of the partials is written before it is read: nothing to clear
    a.tmem_cols = p.tmem_cols; a.m_tiles = p.m_tiles; a.n_acc = 1;
    a.x_tx_bytes = lexb::PAIR_XBLK_BYTES;
    INJECT_LAUNCH();
    lexb::gemm_fp4_tcgen05_pair_kernel<false, false><<<p.grid, p.threads, p.smem, g->stream>>>(map_x, map_wq, map_ws, a);
    CUDA_TRY(cudaGetLastError());
    const size_t elems = mm * nn;
    const uint32_t blocks = static_cast<uint32_t>(std::min<size_t>((elems / 4 + 255) / 256, static_cast<size_t>(g->prop.multiProcessorCount) * 8u));
    INJECT_LAUNCH();
    lexb::splitk_reduce_kernel<0><<<blocks, 256, 0, g->stream>>>(g->static_scratch, splits, elems, a.r, a.y, lexb::GatherDst{},
                                                              static_cast<uint16_t*>(nullptr), n);
    CUDA_TRY(cudaGetLastError());
    return LEXB_OK;
}

int lexb_silu_mul(lexb_gpu* g, uint32_t rows, uint32_t cols, const lexb_buffer* gate, size_t gate_offset, size_t gate_pitch,
                  const lexb_buffer* up, size_t up_offset, size_t up_pitch, lexb_buffer* out, int out_f16) {
    int rc = use(g);
    if (rc) return rc;
    if (!gate || !up || !out) return fail(LEXB_ERR_ARG, "lexb_silu_mul: null buffer");
    if (rows == 0 || cols == 0 || cols % 4u) return fail(LEXB_ERR_SHAPE, "silu_mul: 4 must divide cols = %u", cols);
    if (gate_pitch < cols || up_pitch < cols || (gate_pitch | up_pitch | gate_offset | up_offset) % 4u)
        return fail(LEXB_ERR_ARG, "silu_mul: pitches and offsets are in f32 elements, multiples of 4, pitch >= cols");
    const size_t need_g = (gate_offset + static_cast<size_t>(rows - 1) * gate_pitch + cols) * 4;
    const size_t need_u = (up_offset + static_cast<size_t>(rows - 1) * up_pitch + cols) * 4;
    if ((rc = check_buf(gate, g, need_g, "gate"))) return rc;
    if ((rc = check_buf(up, g, need_u, "up"))) return rc;
    if ((rc = check_buf(out, g, static_cast<size_t>(rows) * cols * (out_f16 ? 2 : 4), "out"))) return rc;
    const size_t total = static_cast<size_t>(rows) * (cols / 4u);
    const uint32_t blocks = static_cast<uint32_t>(std::min<size_t>((total + 255) / 256, static_cast<size_t>(g->prop.multiProcessorCount) * 16u));
    const float* gp = static_cast<const float*>(gate->ptr) + gate_offset;
    const float* up_ = static_cast<const float*>(up->ptr) + up_offset;
    INJECT_LAUNCH();
    PdlLaunch launch(g, blocks, 256, g->pdl);
    if (out_f16)
        CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, silu_mul_kernel<uint16_t>, rows, cols, gp, gate_pitch, up_, up_pitch, static_cast<uint16_t*>(out->ptr)));
    else
        CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, silu_mul_kernel<float>, rows, cols, gp, gate_pitch, up_, up_pitch, static_cast<float*>(out->ptr)));
    CUDA_TRY(cudaGetLastError());
    return LEXB_OK;
}

int lexb_prefill_chunks(uint32_t tokens, uint32_t limit, int gemm_ok, uint32_t* chunks, uint32_t max_chunks, uint32_t* count) {
    static const uint32_t GEMM_SIZES[6] = {512, 256, 128, 64, 32, 16};
    const uint32_t MAX_BATCH = 8;
    if (!count) return fail(LEXB_ERR_ARG, "lexb_prefill_chunks: null count");
    // prefill_limit: the largest GEMM size that is <= the wanted chunk (512 when 0), else MAX_BATCH
    uint32_t lim = MAX_BATCH;
    if (gemm_ok) {
        const uint32_t want = limit ? limit : 512u;
        for (uint32_t s : GEMM_SIZES)
            if (s <= want) { lim = s; break; }
    }
    uint32_t left = tokens, n = 0;
    while (left > 0) {
        uint32_t take = left < MAX_BATCH ? left : MAX_BATCH;
        if (gemm_ok)
            for (uint32_t s : GEMM_SIZES)
                if (s <= lim && s <= left) { take = s; break; }
        if (chunks) {
            if (n >= max_chunks) return fail(LEXB_ERR_ARG, "lexb_prefill_chunks: more than %u chunks", max_chunks);
            chunks[n] = take;
        }
        n++;
        left -= take;
    }
    *count = n;
    return LEXB_OK;
}

int lexb_debug_fail_next(int site, int nth, int cuda_error) {
    if (site < 0 || site >= SITE_COUNT) return fail(LEXB_ERR_ARG, "lexb_debug_fail_next: site %d outside [0, %d]", site, SITE_COUNT - 1);
    if (nth < 0 || cuda_error < 0) return fail(LEXB_ERR_ARG, "lexb_debug_fail_next: negative argument");
    std::lock_guard<std::mutex> lk(g_inject_lock);
    if (site == 0) {
        for (auto& in : g_inject) in = Injection{};
        return LEXB_OK;
    }
    g_inject[site].countdown = nth;
    g_inject[site].error = cuda_error ? cuda_error : static_cast<int>(cudaErrorUnknown);
    return LEXB_OK;
}

int lexb_shard_rows(uint32_t n, uint32_t world, uint32_t rank, uint32_t* n0, uint32_t* n1) {
    if (!n0 || !n1) return fail(LEXB_ERR_ARG, "lexb_shard_rows: null out");
    if (world == 0 || rank >= world) return fail(LEXB_ERR_ARG, "rank %u outside world %u", rank, world);
    if (n % 128u) return fail(LEXB_ERR_SHAPE, "sharding splits whole 128-row tiles; 128 does not divide n = %u", n);
    const uint32_t tiles = n / 128u, base = tiles / world, extra = tiles % world;
    const uint32_t first = rank * base + (rank < extra ? rank : extra);
    const uint32_t count = base + (rank < extra ? 1u : 0u);
    *n0 = first * 128u;
    *n1 = (first + count) * 128u;
    return LEXB_OK;
}

}  // extern "C"
