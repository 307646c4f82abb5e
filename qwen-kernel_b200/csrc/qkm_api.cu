// The C ABI of include/qk_moe.h: context, weight upload, op-level entry points and
// the fused per-layer sequences.  Host-side C++; every kernel lives in the other
// translation units and is reached through qkm_kernels.h.
//
// The call sequences mirror the reference engine's dispatch order: decode
// src/main.cpp:4375-4404, batched prefill src/main.cpp:5050-5198.
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "qkm_alloc.h"
#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_tiles.cuh"

using namespace qkm;

struct qkm_layer_dev {
    bool uploaded = false;
    qkm_layer_weights w{};  // device pointers, raw ggml layout
    void* allocs[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    // tile-ordered copies for the streaming kernels (NULL where the type has none)
    void* tiles[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    void* router16 = nullptr;  // the router as f16 in the element order of the prefill GEMMs' rows
    float* router_norm2 = nullptr;   // largest |router row|^2
    float* w_norm = nullptr;   // [2][resident experts + 1] largest row norm of the gate / up matrices, the shared expert last
    bool tiles_ok = false;   // every tensor has tiles: the tensor-core sequences apply
    bool fused_ok = false;   // and every expert is resident: so does the fused decode sequence
};

struct qkm_ctx {
    qkm_config cfg{};
    int device = 0;
    cudaStream_t stream = nullptr;
    uint64_t launches = 0;
    char err[512] = {0};
    std::vector<qkm_layer_dev> layers;
    uint32_t efirst = 0, ecount = 0;  // resident experts (ecount == n_expert when unsharded)
    // scratch, sized for max_tokens
    qkm_sel* sel = nullptr;
    float* h = nullptr;
    void* route_scratch = nullptr;
    size_t route_scratch_bytes = 0;
    uint32_t* offsets = nullptr;
    uint32_t* pairs = nullptr;
    float* contrib = nullptr;  // allocated on first use
    float* y2 = nullptr;
    float* x_stage = nullptr;
    float* y_stage = nullptr;
    float* stack_x = nullptr;  // [n_layer][max_tokens][n_embd], allocated on first use
    float* stack_y = nullptr;
    // streaming path scratch
    int n_sms = 0;
    float* xscale = nullptr;          // decode: [max_tokens][n_embd/256] of the digit planes; prefill: [max_tokens] of the f16 rows
    uint32_t* n_items = nullptr;      // prefill: units of [0] gate/up, [1] down; [2], [3] their tickets
    uint32_t* status = nullptr;       // kernel status word (device)
    uint32_t* route_counter = nullptr; // ticket counter of the decode router's selection (device, stays zero)
    // fused decode sequence (router + grouping + planes -> gate/up -> down, three launches for one or many layers)
    bool dec_ok = false;               // dims fit the fused decode kernels
    int8_t* planes8 = nullptr;         // [min(max_tokens, 64)][n_embd/256][8][256]: of the expert-parallel calls' local tokens
    uint8_t* lut_gu = nullptr;         // table images the decode kernels copy to shared memory
    uint8_t* lut_dd = nullptr;         // table image of the decode IQ4_XS down kernel
    // its scratch for a number of (layer, token) rows; the last layer's records and hidden rows go to sel and h
    struct DecScratch {
        void* mem = nullptr;           // the one allocation that all of it lies in
        uint32_t rows = 0;
        double* logits = nullptr;      // [row][n_expert]
        int8_t* planes = nullptr;      // [row][8 n_embd]
        float* xscale = nullptr;       // [row][n_embd/256]
        float* contrib = nullptr;      // [row][n_used+1][n_embd], for the down kernel that groups by expert
        // of several layers
        qkm_sel* sel = nullptr;
        float* h = nullptr;            // [row][n_used+1][n_ff]
        DecodeGroup* groups = nullptr; // [row][n_used+1]
        uint32_t* counts = nullptr;    // [kDecMaxLayers]
    } dec_one, dec_many;               // for a layer on its own; for several (see stack_scratch)
    bool dec_grouped = false;          // contrib is there
    uint8_t* lut_pf = nullptr;         // table image of the prefill GEMMs
    uint32_t* status_host = nullptr;  // pinned mirror
    bool shapes_stream_ok = false;
    // prefill (tcgen05) scratch, allocated on first use
    void* xb = nullptr;               // [max_tokens][n_embd] f16, rows scaled by powers of two (xscale undoes it)
    float* xnorm = nullptr;           // [max_tokens] 2-norms of the rows
    void* hb = nullptr;               // [max_tokens*(n_used+1)][n_ff] hidden rows by pair position, f16 scaled per row
    float* hscale = nullptr;          // [max_tokens*(n_used+1)] the scales that undo the rows' scaling
    float* contrib_p = nullptr;       // [max_tokens*(n_used+1)][n_embd]
    uint32_t unit_rows = kWgemmRows;             // activation rows per unit of the work lists
    MmaItem* mma_items[2] = {nullptr, nullptr};  // gate/up, down
    uint32_t* pos_of = nullptr;       // [max_tokens*(n_used+1)]
    uint32_t* group_counts = nullptr; // [resident experts] pairs, then [max_tokens*n_used] a pair's number inside its expert
    void* argmax_scratch = nullptr; uint32_t argmax_rows = 0;
    // dense matrices for qkm_dense_gemm (tile-ordered copies) and its scratch, sized on demand
    static constexpr int kDenseSlots = 16;
    struct Dense { uint32_t type = 0, M = 0, K = 0; float w_scale = 1.f; void* tiles = nullptr; } dense[kDenseSlots];
    void* dense_xb = nullptr; float* dense_scale = nullptr;
    size_t dense_cap_elems = 0, dense_cap_rows = 0;
    // expert-parallel exchange plan of the last qkm_ep_dispatch, allocated on first use
    uint32_t ep_ranks = 0;
    uint32_t* ep_counts = nullptr;       // [n_ranks + 1] rows per destination rank, then their sum
    uint32_t* ep_counts_host = nullptr;  // pinned mirror
    uint32_t* ep_send_tok = nullptr;     // [max_tokens * min(n_ranks, n_used)]
    uint32_t* ep_send_pos = nullptr;     // [max_tokens][n_ranks]
    // peer-memory form of the exchange: this rank's receive buffers and every rank's as mapped here
    uint32_t pm_ranks = 0, pm_rank = 0, pm_cap = 0;   // slot_cap rows per source rank
    uint32_t pm_epoch = 0;                            // barriers issued so far (qkm_ep_barrier)
    bool pm_shared_in_partial = false;                // the last qkm_ep_forward_slots included the shared expert
    bool pm_rows_f16 = false;                         // the last qkm_ep_push sent f16 rows (layers on the tensor-core path)
    float* pm_xrecv = nullptr; qkm_sel* pm_selrecv = nullptr; float* pm_back = nullptr;   // mapped by the peers
    float* pm_partial = nullptr;                      // local partial rows where the fold does not store to the peers
    float* pm_xscale = nullptr;                       // [slot_cap] scales of the local rows sent as f16 (small batches)
    EpPeerTable pm_peers{};
    void* pm_opened[kMaxPeerRanks][3] = {};           // mappings this context opened from handles
    // decode stacks whose layers do not go together, as CUDA graphs: captured on first use of an argument set, a few sets kept
    static constexpr int kStackGraphs = 8;
    struct StackGraph {
        cudaGraphExec_t exec = nullptr;
        uint32_t first = 0, count = 0, n = 0;
        const float* x = nullptr;
        float* y = nullptr;
        cudaStream_t stream = nullptr;
        uint64_t launches = 0;       // kernels one replay launches
        uint64_t used = 0;           // for least-recently-used replacement
    } stack_graphs[kStackGraphs];
    uint64_t stack_clock = 0;
    // the host-buffer form of the stack copies chunk k+1 in and chunk k-1 out while chunk k computes
    static constexpr int kStackChunks = 3;
    static constexpr size_t kStackChunkBytes = 3u << 19;   // rows below which the stack with host buffers is not cut, see qkm_moe_decode_stack_host
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    cudaEvent_t ev_in[kStackChunks] = {}, ev_out[kStackChunks] = {}, ev_copies = nullptr;
    void drop_stack_graphs() {
        for (auto& g : stack_graphs) if (g.exec) { cudaGraphExecDestroy(g.exec); g.exec = nullptr; }
    }
    // per-stage profiling of the fused calls
    static constexpr int kMaxStages = 16;
    bool profiling = false;
    cudaEvent_t prof_ev[kMaxStages + 1] = {};
    char prof_label[kMaxStages][16] = {};
    int prof_n = 0;
    void prof_begin() {
        prof_n = 0;
        if (profiling) cudaEventRecord(prof_ev[0], stream);
    }
    void prof_mark(const char* label) {
        if (!profiling || prof_n >= kMaxStages) return;
        snprintf(prof_label[prof_n], 16, "%s", label);
        cudaEventRecord(prof_ev[++prof_n], stream);
    }
    Launch L() { return Launch{stream, &launches}; }
    // decode chain (router -> gate/up -> down -> next layer's router): each kernel is launched as a programmatic dependent of
    // the one before, so that its scheduling and set-up overlap that kernel's tail (1 token 26.0 -> 24.0 us a layer, 16: 72.0 -> 69.2);
    // not while stages are timed
    Launch Lchain() { return Launch{stream, &launches, !profiling}; }
};

namespace {

int fail(qkm_ctx* c, int code, const char* fmt, ...) {
    if (c) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(c->err, sizeof c->err, fmt, ap);
        va_end(ap);
    }
    return code;
}

template <int N>
cudaError_t dev_alloc_all(const Want (&want)[N]) {
    const int e = alloc_all(want, [](void** p, size_t bytes) { return (int)cudaMalloc(p, bytes); }, [](void* p) { cudaFree(p); });
    if (e) cudaGetLastError();   // reported by the caller; the next launch's check must not find it
    return (cudaError_t)e;
}

#define QKM_CUDA(c, call)                                                                       \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return fail((c), QKM_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                        __FILE__, __LINE__);                                                    \
    } while (0)

bool dims_ok(const qkm_dims& d) {
    // limits the reference enforces: src/main.cpp:955, :1298, :3620-3621
    return d.n_embd >= 256 && d.n_embd % 256 == 0 && d.n_ff >= 256 && d.n_ff % 256 == 0 &&
           d.n_expert >= 1 && d.n_expert <= 512 && d.n_used >= 1 && d.n_used <= 16 &&
           d.n_used <= d.n_expert;
}

size_t tensor_bytes(const qkm_ctx* c, int idx, const qkm_layer_weights& w) {
    const qkm_dims& d = c->cfg.dims;
    const size_t ne = c->ecount;
    switch (idx) {
        case 0: return (size_t)d.n_expert * row_bytes(w.router_type, d.n_embd);
        case 1: return (size_t)d.n_embd * 4;
        case 2: case 3: return ne * d.n_ff * row_bytes(w.gateup_type, d.n_embd);
        case 4: return ne * d.n_embd * row_bytes(w.down_type, d.n_ff);
        case 5: case 6: return (size_t)d.n_ff * row_bytes(QKM_TYPE_Q8_0, d.n_embd);
        case 7: return (size_t)d.n_embd * row_bytes(QKM_TYPE_Q8_0, d.n_ff);
    }
    return 0;
}

int check_tokens(qkm_ctx* c, uint32_t n) {
    if (!c) return QKM_ERR_ARG;
    if (n > c->cfg.max_tokens) return fail(c, QKM_ERR_BOUNDS, "n_tokens %u exceeds max_tokens %u", n, c->cfg.max_tokens);
    return QKM_OK;
}

int layer_ready(qkm_ctx* c, uint32_t layer) {
    if (!c) return QKM_ERR_ARG;
    if (layer >= c->cfg.n_layer) return fail(c, QKM_ERR_BOUNDS, "layer %u out of range (n_layer %u)", layer, c->cfg.n_layer);
    if (!c->layers[layer].uploaded) return fail(c, QKM_ERR_BUSY, "layer %u has no weights uploaded", layer);
    return QKM_OK;
}

// Scratch of the fused decode sequence: a stack's layers go through it together, as many as kDecRows (layer, token) rows allow: 40 layers of 16
// tokens, 12 of 64; 39 KB a row for 256 experts, top 8, and 74 KB more where the down kernel groups by expert (batches from 40 tokens on).  With
// 192 rows stacks of 64 tokens take 2 to 7 % longer, with 384 up to 1 %, with 1152 the same.
constexpr uint32_t kDecRows = 768;
// Up to this much for several layers is taken at qkm_open: what a context for fewer than 40 tokens, one that decodes, can need.  More only when a
// stack is first decoded (0.33 ms as a rule, once), since contexts that prefill, or step through their layers one by one, have no use for 85 to 105 MB.
constexpr size_t kDecAtOpen = 40u << 20;

// Bytes of the scratch for `rows` rows; with s.mem set, where its parts lie.
size_t dec_layout(const qkm_ctx* c, qkm_ctx::DecScratch& s, uint32_t rows, bool several) {
    const qkm_dims& d = c->cfg.dims;
    const size_t R = rows, S = d.n_used + 1;
    size_t at = 0;
    auto part = [&](auto& p, size_t bytes) {
        if (s.mem) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>((uint8_t*)s.mem + at);
        at += (bytes + 255) / 256 * 256;
    };
    part(s.logits, R * d.n_expert * sizeof(double));
    part(s.planes, R * 8 * d.n_embd);
    part(s.xscale, R * (d.n_embd / 256) * sizeof(float));
    if (c->dec_grouped) part(s.contrib, R * S * d.n_embd * sizeof(float));
    if (several) {
        part(s.sel, R * sizeof(qkm_sel));
        part(s.h, R * S * d.n_ff * sizeof(float));
        part(s.groups, R * S * sizeof(DecodeGroup));
        part(s.counts, kDecMaxLayers * sizeof(uint32_t));
    }
    return at;
}
cudaError_t dec_alloc(const qkm_ctx* c, qkm_ctx::DecScratch& s, uint32_t rows, bool several) {
    if (const cudaError_t e = cudaMalloc(&s.mem, dec_layout(c, s, rows, several))) {
        s.mem = nullptr;
        cudaGetLastError();   // reported by the caller; the next launch's check must not find it
        return e;
    }
    dec_layout(c, s, s.rows = rows, several);
    return cudaSuccess;
}
uint32_t dec_most_tokens(const qkm_ctx* c) { return c->cfg.max_tokens < 64 ? c->cfg.max_tokens : 64; }
uint32_t dec_most_rows(const qkm_ctx* c) {
    const uint32_t T = dec_most_tokens(c), fit = decode_gateup_rows((uint32_t)c->n_sms), most = kDecRows < fit ? kDecRows : fit;
    const uint64_t rows = (uint64_t)c->cfg.n_layer * T;
    return rows < most ? (uint32_t)rows : most;
}
cudaError_t alloc_decode(qkm_ctx* c) {
    const qkm_dims& d = c->cfg.dims;
    const uint32_t T = dec_most_tokens(c);
    const Want want[] = {{(void**)&c->planes8, (size_t)T * 8 * d.n_embd}, {(void**)&c->lut_gu, decode_gateup_lut_bytes()}, {(void**)&c->lut_dd, decode_down_lut_bytes()}};
    if (const cudaError_t e = dev_alloc_all(want)) return e;
    if (c->ecount != d.n_expert) return cudaSuccess;   // the fused sequence wants every expert
    c->dec_grouped = decode_down_group_ok(d) && (T >= 40 || !decode_down_any_ok(d));
    if (const cudaError_t e = dec_alloc(c, c->dec_one, T, false)) return e;
    if (c->cfg.n_layer > 1 && dec_layout(c, c->dec_many, dec_most_rows(c), true) <= kDecAtOpen) return dec_alloc(c, c->dec_many, dec_most_rows(c), true);
    return cudaSuccess;
}
// Whether the scratch for several layers is there, made when it is first wanted.  Where it cannot be had - the stream is being captured, or the
// memory is short - the layers go one by one.
bool stack_scratch(qkm_ctx* c) {
    if (c->dec_many.mem) return true;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // (another thread's capture is not broken by it)
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = dec_alloc(c, c->dec_many, dec_most_rows(c), true);
    cudaThreadExchangeStreamCaptureMode(&mode);
    return e == cudaSuccess;
}

}  // namespace

// ---------------------------------------------------------------- lifecycle

extern "C" QKM_API const char* qkm_version(void) { return "qk-moe-b200 0.1 (sm_100a)"; }

extern "C" QKM_API qkm_ctx* qkm_open(const qkm_config* cfg, char* err, size_t err_len) {
    auto bail = [&](const char* msg, const char* detail) -> qkm_ctx* {
        if (err && err_len) snprintf(err, err_len, "%s%s%s", msg, detail ? ": " : "", detail ? detail : "");
        return nullptr;
    };
    if (!cfg) return bail("qkm_open: NULL config", nullptr);
    if (!dims_ok(cfg->dims)) return bail("qkm_open: unsupported dims (n_embd,n_ff multiples of 256; n_expert<=512; n_used<=16)", nullptr);
    if (cfg->n_layer < 1 || cfg->max_tokens < 1) return bail("qkm_open: n_layer and max_tokens must be >= 1", nullptr);
    if (cfg->max_tokens >= (1u << 28)) return bail("qkm_open: max_tokens too large for the pair encoding", nullptr);
    uint32_t efirst = cfg->expert_first, ecount = cfg->expert_count;
    if (ecount == 0) { efirst = 0; ecount = cfg->dims.n_expert; }
    if ((uint64_t)efirst + ecount > cfg->dims.n_expert) return bail("qkm_open: expert range exceeds n_expert", nullptr);

    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) return bail("qkm_open: no CUDA device (this library has no CPU path)", cudaGetErrorString(e));
    int dev = cfg->device;
    if (dev < 0) { if (cudaGetDevice(&dev) != cudaSuccess) dev = 0; }
    if (dev >= ndev) return bail("qkm_open: device ordinal out of range", nullptr);
    if ((e = cudaSetDevice(dev)) != cudaSuccess) return bail("qkm_open: cudaSetDevice", cudaGetErrorString(e));
    cudaDeviceProp prop{};
    if ((e = cudaGetDeviceProperties(&prop, dev)) != cudaSuccess) return bail("qkm_open: cudaGetDeviceProperties", cudaGetErrorString(e));
    if (prop.major != 10) return bail("qkm_open: kernels are built for sm_100a only; device is", prop.name);

    qkm_ctx* c = new (std::nothrow) qkm_ctx();
    if (!c) return bail("qkm_open: out of host memory", nullptr);
    c->cfg = *cfg;
    c->device = dev;
    c->efirst = efirst;
    c->ecount = ecount;
    c->layers.resize(cfg->n_layer);
    const qkm_dims& d = cfg->dims;
    const size_t T = cfg->max_tokens;
    c->route_scratch_bytes = qkm::route_scratch_bytes((uint32_t)T, d.n_expert);
    struct { void** p; size_t bytes; } allocs[] = {
        {(void**)&c->sel, T * sizeof(qkm_sel)},
        {(void**)&c->h, T * (d.n_used + 1) * d.n_ff * sizeof(float)},
        {(void**)&c->route_scratch, qkm::route_scratch_bytes((uint32_t)T, d.n_expert)},
        {(void**)&c->offsets, (d.n_expert + 1) * sizeof(uint32_t)},
        {(void**)&c->pairs, T * (d.n_used + 1) * sizeof(uint32_t)},
        {(void**)&c->y2, T * d.n_embd * sizeof(float)},
        {(void**)&c->x_stage, T * d.n_embd * sizeof(float)},
        {(void**)&c->y_stage, T * d.n_embd * sizeof(float)},
    };
    for (auto& a : allocs) {
        if ((e = cudaMalloc(a.p, a.bytes)) != cudaSuccess) {
            bail("qkm_open: cudaMalloc of scratch", cudaGetErrorString(e));
            qkm_close(c);
            return nullptr;
        }
    }
    c->n_sms = prop.multiProcessorCount;
    // Streaming kernels: column blocks per row must be a power of two in [2,16] (one warp
    // each) and rows must split into whole items.  (The fused decode / prefill sequences
    // also need every expert resident; a sharded context uses the tiles through qkm_ep_*.)
    auto pow2_2_16 = [](uint32_t v) { return v >= 2 && v <= 16 && (v & (v - 1)) == 0; };
    c->shapes_stream_ok = pow2_2_16(d.n_embd / 256) && d.n_embd / 256 <= 8 && pow2_2_16(d.n_ff / 256) && d.n_used <= 15 &&
                          d.n_ff % 128 == 0;
    if (c->shapes_stream_ok) {
        struct { void** p; size_t bytes; } more[] = {
            {(void**)&c->xscale, T * (d.n_embd / 256) * sizeof(float)},
            {(void**)&c->n_items, 4 * sizeof(uint32_t)},
        };
        for (auto& a : more) {
            if ((e = cudaMalloc(a.p, a.bytes)) != cudaSuccess) {
                bail("qkm_open: cudaMalloc of streaming scratch", cudaGetErrorString(e));
                qkm_close(c);
                return nullptr;
            }
        }
        c->dec_ok = decode_gateup_ok(d);
        if (c->dec_ok) {
            if ((e = alloc_decode(c)) != cudaSuccess) {
                bail("qkm_open: cudaMalloc of decode scratch", cudaGetErrorString(e));
                qkm_close(c);
                return nullptr;
            }
            const Launch L0{nullptr, nullptr};
            if ((e = launch_decode_gateup_luts(L0, c->lut_gu)) != cudaSuccess ||
                (e = launch_decode_down_lut(L0, c->lut_dd)) != cudaSuccess ||
                (e = cudaDeviceSynchronize()) != cudaSuccess) {
                bail("qkm_open: decode tables", cudaGetErrorString(e));
                qkm_close(c);
                return nullptr;
            }
        }
    }
    if ((e = cudaMalloc((void**)&c->status, sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMemset(c->status, 0, sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMalloc((void**)&c->route_counter, kDecMaxLayers * kDecCounters * sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMemset(c->route_counter, 0, kDecMaxLayers * kDecCounters * sizeof(uint32_t))) != cudaSuccess ||
        (e = cudaMallocHost((void**)&c->status_host, sizeof(uint32_t))) != cudaSuccess) {
        bail("qkm_open: status word", cudaGetErrorString(e));
        qkm_close(c);
        return nullptr;
    }
    *c->status_host = 0;
    {
        const Launch L0{nullptr, nullptr};
        if ((e = cudaMalloc((void**)&c->lut_pf, wgemm_table_bytes())) != cudaSuccess ||
            (e = launch_wgemm_table(L0, c->lut_pf)) != cudaSuccess || (e = cudaDeviceSynchronize()) != cudaSuccess) {
            bail("qkm_open: prefill tables", cudaGetErrorString(e));
            qkm_close(c);
            return nullptr;
        }
    }
    if (err && err_len) err[0] = 0;
    return c;
}

extern "C" QKM_API void qkm_close(qkm_ctx* c) {
    if (!c) return;
    cudaSetDevice(c->device);
    cudaDeviceSynchronize();
    for (auto& l : c->layers) {
        for (void* p : l.allocs) if (p) cudaFree(p);
        for (void* p : l.tiles) if (p) cudaFree(p);
        if (l.router16) cudaFree(l.router16);
        if (l.w_norm) cudaFree(l.w_norm);
        if (l.router_norm2) cudaFree(l.router_norm2);
    }
    for (auto& dm : c->dense) if (dm.tiles) cudaFree(dm.tiles);
    void* scratch[] = {c->argmax_scratch, c->dense_xb, c->dense_scale, c->sel, c->h, c->route_scratch, c->offsets, c->pairs, c->contrib, c->y2, c->x_stage, c->y_stage,
                       c->stack_x, c->stack_y, c->xscale, c->n_items, c->status, c->route_counter,
                       c->planes8, c->lut_gu, c->lut_dd, c->lut_pf, c->dec_one.mem, c->dec_many.mem,
                       c->xb, c->xnorm, c->hb, c->hscale, c->contrib_p, c->mma_items[0], c->mma_items[1],
                       c->pos_of, c->group_counts, c->ep_counts, c->ep_send_tok, c->ep_send_pos};
    for (void* p : scratch) if (p) cudaFree(p);
    for (auto& o : c->pm_opened) for (void* p : o) if (p) cudaIpcCloseMemHandle(p);
    for (void* p : {(void*)c->pm_xrecv, (void*)c->pm_selrecv, (void*)c->pm_back, (void*)c->pm_partial, (void*)c->pm_xscale}) if (p) cudaFree(p);
    if (c->status_host) cudaFreeHost(c->status_host);
    if (c->ep_counts_host) cudaFreeHost(c->ep_counts_host);
    c->drop_stack_graphs();
    for (cudaEvent_t ev : c->ev_in) if (ev) cudaEventDestroy(ev);
    for (cudaEvent_t ev : c->ev_out) if (ev) cudaEventDestroy(ev);
    if (c->ev_copies) cudaEventDestroy(c->ev_copies);
    if (c->copy_in) cudaStreamDestroy(c->copy_in);
    if (c->copy_out) cudaStreamDestroy(c->copy_out);
    for (cudaEvent_t ev : c->prof_ev) if (ev) cudaEventDestroy(ev);
    delete c;
}

extern "C" QKM_API const char* qkm_last_error(const qkm_ctx* c) { return c ? c->err : "NULL context"; }
extern "C" QKM_API uint32_t qkm_n_embd(const qkm_ctx* c) { return c ? c->cfg.dims.n_embd : 0; }
extern "C" QKM_API uint32_t qkm_n_ff(const qkm_ctx* c) { return c ? c->cfg.dims.n_ff : 0; }
extern "C" QKM_API uint32_t qkm_n_expert(const qkm_ctx* c) { return c ? c->cfg.dims.n_expert : 0; }
extern "C" QKM_API uint32_t qkm_n_used(const qkm_ctx* c) { return c ? c->cfg.dims.n_used : 0; }
extern "C" QKM_API uint32_t qkm_n_layer(const qkm_ctx* c) { return c ? c->cfg.n_layer : 0; }
extern "C" QKM_API uint32_t qkm_max_tokens(const qkm_ctx* c) { return c ? c->cfg.max_tokens : 0; }
extern "C" QKM_API void qkm_expert_range(const qkm_ctx* c, uint32_t* first, uint32_t* count) {
    if (first) *first = c ? c->efirst : 0;
    if (count) *count = c ? c->ecount : 0;
}
extern "C" QKM_API size_t qkm_row_bytes(uint32_t type, uint64_t ne0) {
    const uint32_t be = block_elems(type);
    if (be == 0 || ne0 % be) return 0;
    return row_bytes(type, ne0);
}

extern "C" QKM_API int qkm_set_stream(qkm_ctx* c, void* s) {
    if (!c) return QKM_ERR_ARG;
    c->stream = (cudaStream_t)s;
    return QKM_OK;
}
// Copies the kernels' status word back after a synchronise; a bounded device-side wait
// that gave up (or a broken layout assumption) surfaces here as an error code.
static int check_status(qkm_ctx* c) {
    QKM_CUDA(c, cudaMemcpyAsync(c->status_host, c->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    if (*c->status_host != 0) {
        const uint32_t st = *c->status_host;
        cudaMemsetAsync(c->status, 0, sizeof(uint32_t), c->stream);
        return fail(c, QKM_ERR_TIMEOUT, "a kernel reported status %u (1 = bounded wait gave up, 2 = shared-memory layout)", st);
    }
    return QKM_OK;
}

extern "C" QKM_API int qkm_sync(qkm_ctx* c) {
    if (!c) return QKM_ERR_ARG;
    return check_status(c);
}
extern "C" QKM_API uint64_t qkm_launch_count(const qkm_ctx* c) { return c ? c->launches : 0; }

extern "C" QKM_API void* qkm_dev_alloc(qkm_ctx* c, size_t bytes) {
    if (!c) return nullptr;
    void* p = nullptr;
    cudaSetDevice(c->device);
    cudaError_t e = cudaMalloc(&p, bytes ? bytes : 1);
    if (e != cudaSuccess) { fail(c, QKM_ERR_CUDA, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e)); return nullptr; }
    return p;
}
extern "C" QKM_API int qkm_dev_free(qkm_ctx* c, void* p) {
    if (!c) return QKM_ERR_ARG;
    QKM_CUDA(c, cudaFree(p));
    return QKM_OK;
}
extern "C" QKM_API int qkm_h2d(qkm_ctx* c, void* dst, const void* src, size_t bytes) {
    if (!c || (!dst && bytes) || (!src && bytes)) return QKM_ERR_ARG;
    QKM_CUDA(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    return QKM_OK;
}
extern "C" QKM_API int qkm_d2h(qkm_ctx* c, void* dst, const void* src, size_t bytes) {
    if (!c || (!dst && bytes) || (!src && bytes)) return QKM_ERR_ARG;
    QKM_CUDA(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    return QKM_OK;
}

// ---------------------------------------------------------------- weights

extern "C" QKM_API int qkm_upload_layer(qkm_ctx* c, uint32_t layer, const qkm_layer_weights* w) {
    if (!c || !w) return QKM_ERR_ARG;
    if (layer >= c->cfg.n_layer) return fail(c, QKM_ERR_BOUNDS, "layer %u out of range", layer);
    // the types loadMoeT accepts (src/main.cpp:1283-1291), plus an F16 router
    if (w->router_type != QKM_TYPE_F32 && w->router_type != QKM_TYPE_F16)
        return fail(c, QKM_ERR_TYPE, "router type %u unsupported (F32 or F16)", w->router_type);
    if (w->gateup_type != QKM_TYPE_IQ3_XXS && w->gateup_type != QKM_TYPE_IQ4_XS)
        return fail(c, QKM_ERR_TYPE, "gate/up type %u unsupported (IQ3_XXS or IQ4_XS)", w->gateup_type);
    if (w->down_type != QKM_TYPE_IQ4_XS && w->down_type != QKM_TYPE_Q6_K)
        return fail(c, QKM_ERR_TYPE, "down type %u unsupported (IQ4_XS or Q6_K)", w->down_type);
    const void* src[8] = {w->router, w->gate_inp_shexp, w->gate_exps, w->up_exps, w->down_exps,
                          w->gate_shexp, w->up_shexp, w->down_shexp};
    for (const void* p : src) if (!p) return fail(c, QKM_ERR_ARG, "layer %u: NULL tensor pointer", layer);
    QKM_CUDA(c, cudaSetDevice(c->device));
    c->drop_stack_graphs();
    qkm_layer_dev& l = c->layers[layer];
    for (int i = 0; i < 8; ++i) {
        const size_t bytes = tensor_bytes(c, i, *w);
        if (l.allocs[i]) { QKM_CUDA(c, cudaFree(l.allocs[i])); l.allocs[i] = nullptr; }
        // 256 spare bytes: streaming kernels may read a few bytes past a tensor's end
        QKM_CUDA(c, cudaMalloc(&l.allocs[i], bytes + 256));
        QKM_CUDA(c, cudaMemcpyAsync(l.allocs[i], src[i], bytes, cudaMemcpyHostToDevice, c->stream));
        QKM_CUDA(c, cudaMemsetAsync((uint8_t*)l.allocs[i] + bytes, 0, 256, c->stream));
    }
    // tile-ordered copies for the streaming kernels (same bytes, re-ordered on the device)
    for (void*& p : l.tiles) { if (p) { QKM_CUDA(c, cudaFree(p)); p = nullptr; } }
    for (void** p : {&l.router16, (void**)&l.w_norm, (void**)&l.router_norm2}) { if (*p) { QKM_CUDA(c, cudaFree(*p)); *p = nullptr; } }
    l.tiles_ok = l.fused_ok = false;
    if (c->shapes_stream_ok) {
        const qkm_dims& d = c->cfg.dims;
        struct { int idx; uint32_t type, mats, rows, K; } plan[] = {
            {2, w->gateup_type, c->ecount, d.n_ff, d.n_embd}, {3, w->gateup_type, c->ecount, d.n_ff, d.n_embd},
            {4, w->down_type, c->ecount, d.n_embd, d.n_ff},
            {5, QKM_TYPE_Q8_0, 1, d.n_ff, d.n_embd}, {6, QKM_TYPE_Q8_0, 1, d.n_ff, d.n_embd},
            {7, QKM_TYPE_Q8_0, 1, d.n_embd, d.n_ff},
        };
        for (auto& t : plan) {
            const size_t bytes = tiled_bytes(t.type, t.mats, t.rows, t.K);
            QKM_CUDA(c, cudaMalloc(&l.tiles[t.idx], bytes + 256));
            cudaError_t e = launch_repack(c->L(), t.type, l.allocs[t.idx], l.tiles[t.idx], t.mats, t.rows, t.K);
            if (e != cudaSuccess) return fail(c, QKM_ERR_CUDA, "repack: %s", cudaGetErrorString(e));
        }
        // what the prefill sequence wants beside the tiles: the router in its rows' order, bounds on the hidden values
        const size_t n_norm = 2 * ((size_t)c->ecount + 1);
        QKM_CUDA(c, cudaMalloc(&l.router16, (size_t)d.n_expert * d.n_embd * 2));
        QKM_CUDA(c, cudaMalloc((void**)&l.w_norm, n_norm * sizeof(float)));
        QKM_CUDA(c, cudaMalloc((void**)&l.router_norm2, sizeof(float)));
        QKM_CUDA(c, cudaMemsetAsync(l.router_norm2, 0, sizeof(float), c->stream));
        QKM_CUDA(c, cudaMemsetAsync(l.w_norm, 0, n_norm * sizeof(float), c->stream));
        cudaError_t e = launch_router_f16(c->L(), w->router_type, l.allocs[0], l.router16, (uint64_t)d.n_expert * d.n_embd);
        if (e == cudaSuccess) e = launch_row_norm2(c->L(), d, w->router_type, l.allocs[0], nullptr, l.router_norm2);
        for (int m = 0; m < 2 && e == cudaSuccess; ++m) {
            e = launch_row_norm_max(c->L(), w->gateup_type, l.allocs[2 + m], l.w_norm + m * (c->ecount + 1), c->ecount, d.n_ff, d.n_embd);
            if (e == cudaSuccess) e = launch_row_norm_max(c->L(), QKM_TYPE_Q8_0, l.allocs[5 + m], l.w_norm + m * (c->ecount + 1) + c->ecount, 1, d.n_ff, d.n_embd);
        }
        if (e != cudaSuccess) return fail(c, QKM_ERR_CUDA, "upload: %s", cudaGetErrorString(e));
        l.tiles_ok = true;
        l.fused_ok = c->ecount == c->cfg.dims.n_expert;
    }
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    l.w = *w;
    l.w.router = l.allocs[0];
    l.w.gate_inp_shexp = (const float*)l.allocs[1];
    l.w.gate_exps = l.allocs[2];
    l.w.up_exps = l.allocs[3];
    l.w.down_exps = l.allocs[4];
    l.w.gate_shexp = l.allocs[5];
    l.w.up_shexp = l.allocs[6];
    l.w.down_shexp = l.allocs[7];
    l.uploaded = true;
    return QKM_OK;
}

extern "C" QKM_API int qkm_layer_device_ptrs(const qkm_ctx* c, uint32_t layer, qkm_layer_weights* out) {
    if (!c || !out) return QKM_ERR_ARG;
    if (layer >= c->cfg.n_layer) return QKM_ERR_BOUNDS;
    if (!c->layers[layer].uploaded) return QKM_ERR_BUSY;
    *out = c->layers[layer].w;
    return QKM_OK;
}

// ---------------------------------------------------------------- op-level entry points

#define QKM_LAUNCH(c, call)                                                                          \
    do {                                                                                             \
        cudaError_t e_ = (call);                                                                     \
        if (e_ == cudaErrorInvalidValue) return fail((c), QKM_ERR_TYPE, "%s: unsupported type or shape", #call); \
        if (e_ != cudaSuccess) return fail((c), QKM_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

extern "C" QKM_API int qkm_moe_logits(qkm_ctx* c, uint32_t router_type, const void* router, const float* x,
                                      float* logits, uint32_t n) {
    if (!c || !router || !x || !logits) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_logits(c->L(), c->cfg.dims, router_type, router, x, logits, nullptr, n));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_select(qkm_ctx* c, const float* logits, const float* gis, const float* x,
                                      qkm_sel* sel, uint32_t n) {
    if (!c || !logits || !gis || !x || !sel) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_select(c->L(), c->cfg.dims, logits, gis, x, sel, n));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_route_select(qkm_ctx* c, uint32_t router_type, const void* router,
                                            const float* gis, const float* x, qkm_sel* sel, uint32_t n) {
    if (!c || !router || !gis || !x || !sel) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    if (router_type != QKM_TYPE_F32 && router_type != QKM_TYPE_F16) return fail(c, QKM_ERR_TYPE, "router type %u", router_type);
    QKM_LAUNCH(c, launch_route_select(c->L(), c->cfg.dims, router_type, router, gis, x, sel, n, c->route_scratch, c->route_scratch_bytes));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_group_pairs(qkm_ctx* c, const qkm_sel* sel, uint32_t n, uint32_t* offsets,
                                           uint32_t* pairs) {
    if (!c || !sel || !offsets || !pairs) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_group_pairs(c->L(), c->cfg.dims, sel, n, offsets, pairs, c->efirst, c->ecount));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_gateup(qkm_ctx* c, uint32_t type, const void* gate, const void* up,
                                      const float* x, const qkm_sel* sel, float* h, uint32_t n) {
    if (!c || !gate || !up || !x || !sel || !h) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_gateup_tokens(c->L(), c->cfg.dims, type, gate, up, x, sel, h, n, c->efirst, c->ecount));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_gateup_grouped(qkm_ctx* c, uint32_t type, const void* gate, const void* up,
                                              const float* x, const uint32_t* offsets, const uint32_t* pairs,
                                              float* h, uint32_t n) {
    if (!c || !gate || !up || !x || !offsets || !pairs || !h) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_gateup_pairs(c->L(), c->cfg.dims, type, gate, up, x, offsets, pairs, h, n, c->efirst, c->ecount));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_shared_gateup(qkm_ctx* c, const void* gate, const void* up, const float* x,
                                             float* h, uint32_t n) {
    if (!c || !gate || !up || !x || !h) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_shared_gateup(c->L(), c->cfg.dims, gate, up, x, h, n));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_down(qkm_ctx* c, uint32_t type, const void* down, const float* h,
                                    const qkm_sel* sel, float* y, uint32_t n) {
    if (!c || !down || !h || !sel || !y) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_down_tokens(c->L(), c->cfg.dims, type, down, h, sel, y, n, c->efirst, c->ecount, nullptr));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_down_grouped(qkm_ctx* c, uint32_t type, const void* down, const float* h,
                                            const qkm_sel* sel, const uint32_t* offsets, const uint32_t* pairs,
                                            float* contrib, uint32_t n) {
    if (!c || !down || !h || !sel || !offsets || !pairs || !contrib) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_down_pairs(c->L(), c->cfg.dims, type, down, h, sel, offsets, pairs, contrib, n, c->efirst, c->ecount));
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_shared_down(qkm_ctx* c, const void* down, const float* h, const qkm_sel* sel,
                                           float* y2, uint32_t n) {
    if (!c || !down || !h || !sel || !y2) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_shared_down(c->L(), c->cfg.dims, down, h, sel, y2, n));
    return QKM_OK;
}

extern "C" QKM_API int qkm_gemv(qkm_ctx* c, uint32_t type, const void* W, const float* x, float* y,
                                uint32_t M, uint32_t K, uint32_t n) {
    if (!c || !W || !x || !y) return QKM_ERR_ARG;
    const uint32_t be = block_elems(type);
    if (be == 0) return fail(c, QKM_ERR_TYPE, "qkm_gemv: type %u unsupported", type);
    if (K == 0 || K % be || K % 8) return fail(c, QKM_ERR_ARG, "qkm_gemv: K=%u must be a multiple of the block size %u and of 8", K, be);
    if (n > 65535) return fail(c, QKM_ERR_BOUNDS, "qkm_gemv: n=%u exceeds 65535", n);
    QKM_LAUNCH(c, launch_gemv_stream(c->L(), type, W, x, y, M, K, n, (uint32_t)c->n_sms, c->status));
    return QKM_OK;
}

extern "C" QKM_API int qkm_dequant(qkm_ctx* c, uint32_t type, const void* blocks, float* y, uint64_t n_elems) {
    if (!c || !blocks || !y) return QKM_ERR_ARG;
    const uint32_t be = block_elems(type);
    if (be == 0) return fail(c, QKM_ERR_TYPE, "qkm_dequant: type %u unsupported", type);
    if (n_elems % be || n_elems % 8) return fail(c, QKM_ERR_ARG, "qkm_dequant: n_elems must be whole blocks and a multiple of 8");
    QKM_LAUNCH(c, launch_dequant(c->L(), type, blocks, y, n_elems));
    return QKM_OK;
}

// ---------------------------------------------------------------- fused layer calls

// Three launches (four where the down kernel that groups by expert is followed by a fold) for `count` layers of the same types whose rows are at hand
// together: (1) router logits, selection, the pairs' groups and digit planes; (2) gate/up + SwiGLU of the routed experts and of
// the shared expert; (3) down projections of both and the weighted sum.  The shared expert rides inside (2)
// and (3): no side stream, and nothing runs beside the two persistent kernels that they would have to share
// the SMs with.  At most 64 tokens (the pair grouping's limit).  Rows of layer first + l at x + l * x_stride and y + l * y_stride; sel and h: where the
// last layer's go.
static int decode_fused(qkm_ctx* c, uint32_t first, uint32_t count, const float* x, uint64_t x_stride, uint32_t n, float* y, uint64_t y_stride, qkm_sel* sel, float* h) {
    const qkm_layer_weights& w = c->layers[first].w;
    const qkm_dims& d = c->cfg.dims;
    const uint32_t nb = (uint32_t)c->n_sms;
    // a layer on its own: the blocks of the kernels behind the router group its pairs themselves
    const qkm_ctx::DecScratch& m = count == 1 ? c->dec_one : c->dec_many;
    const DecodeGroups groups{m.counts, m.groups};   // (none for one layer)
    RouteDecodeArgs ra{};
    GateupDecodeArgs ga{};
    DownDecodeArgs da{};
    for (uint32_t l = 0; l < count; ++l) {
        const qkm_layer_dev& ld = c->layers[first + l];
        const uint8_t* t[8];
        for (int i = 0; i < 8; ++i) t[i] = (const uint8_t*)ld.tiles[i];
        ra.layer[l] = {(const uint8_t*)ld.w.router, ld.w.gate_inp_shexp};
        ga.layer[l] = {t[2], t[3], t[5], t[6]};
        da.layer[l] = {t[4], t[7]};
    }
    ra.x = x; ra.x_stride = x_stride; ra.sel = m.sel; ra.sel_last = sel; ra.logits = m.logits; ra.counter = c->route_counter;
    ra.planes = m.planes; ra.xscale = m.xscale; ra.groups = groups; ra.n_tokens = n; ra.n_layers = count; ra.d = d;
    QKM_LAUNCH(c, launch_route_decode(c->Lchain(), w.router_type, ra));
    c->prof_mark("moe.route");
    ga.luts = c->lut_gu; ga.planes = m.planes; ga.xscale = m.xscale; ga.groups = groups; ga.sel = sel; ga.n_tokens = n; ga.n_layers = count;
    ga.gateup_type = w.gateup_type; ga.h = m.h; ga.h_last = h; ga.status = c->status; ga.d = d;
    QKM_LAUNCH(c, launch_decode_gateup(c->Lchain(), ga, nb));
    c->prof_mark("moe.gu");
    da.lut = c->lut_dd; da.h = m.h; da.h_last = h; da.sel = m.sel; da.sel_last = sel; da.y = y; da.y_stride = y_stride;
    da.groups = groups; da.contrib = m.contrib; da.n_tokens = n; da.n_layers = count; da.status = c->status; da.d = d;
    if (c->dec_grouped && decode_down_group_better(d, w.down_type, n)) QKM_LAUNCH(c, launch_decode_down_group(c->Lchain(), da, w.down_type, nb));
    else if (!decode_down_ok(d)) QKM_LAUNCH(c, launch_decode_down_any(c->Lchain(), da, w.down_type, nb));
    else if (w.down_type == QKM_TYPE_IQ4_XS) QKM_LAUNCH(c, launch_decode_down(c->Lchain(), da, nb));
    else QKM_LAUNCH(c, launch_decode_down_q6k(c->Lchain(), da, nb));
    c->prof_mark("moe.dn");
    return QKM_OK;
}

// The fused sequence's limits; the tensors' are in qkm_layer_dev::fused_ok.
static bool decode_fused_ok(const qkm_ctx* c, uint32_t n) {
    const qkm_dims& d = c->cfg.dims;
    return n && c->dec_ok && c->dec_one.mem && route_decode_ok(d) && (decode_down_ok(d) || decode_down_any_ok(d) || c->dec_grouped);
}

// Layers [first, first + count), all ready for the fused sequence, at most 64 tokens at a time: in runs of the same types, as many layers at once
// as the scratch holds.
static int decode_layers(qkm_ctx* c, uint32_t first, uint32_t count, const float* x, uint64_t x_stride, uint32_t n, float* y, uint64_t y_stride) {
    const qkm_dims& d = c->cfg.dims;
    const uint32_t rows = count > 1 && stack_scratch(c) ? c->dec_many.rows : 0;
    for (uint32_t t = 0; t < n; t += 64) {
        const uint32_t nt = n - t < 64 ? n - t : 64, most = rows / nt < kDecMaxLayers ? rows / nt : kDecMaxLayers;
        for (uint32_t l = 0, k = 1; l < count; l += k, k = 1) {
            const qkm_layer_weights& w = c->layers[first + l].w;
            for (; l + k < count && k < most; ++k) {
                const qkm_layer_weights& v = c->layers[first + l + k].w;
                if (v.router_type != w.router_type || v.gateup_type != w.gateup_type || v.down_type != w.down_type) break;
            }
            if (int rc = decode_fused(c, first + l, k, x + l * x_stride + (size_t)t * d.n_embd, x_stride, nt, y + l * y_stride + (size_t)t * d.n_embd, y_stride,
                                      c->sel + t, c->h + (size_t)t * (d.n_used + 1) * d.n_ff)) return rc;
        }
    }
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_decode(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, float* y) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (!x || !y) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    const qkm_layer_dev& ld = c->layers[layer];
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    c->prof_begin();
    if (ld.fused_ok && decode_fused_ok(c, n)) return decode_layers(c, layer, 1, x, 0, n, y, 0);
    // generic kernels on the raw layout
    QKM_LAUNCH(c, launch_route_select(c->L(), d, w.router_type, w.router, w.gate_inp_shexp, x, c->sel, n, c->route_scratch, c->route_scratch_bytes));
    c->prof_mark("moe.route");
    QKM_LAUNCH(c, launch_shared_gateup(c->L(), d, w.gate_shexp, w.up_shexp, x, c->h, n));
    c->prof_mark("moe.shared_gu");
    QKM_LAUNCH(c, launch_gateup_tokens(c->L(), d, w.gateup_type, w.gate_exps, w.up_exps, x, c->sel, c->h, n, c->efirst, c->ecount));
    c->prof_mark("moe.gu");
    QKM_LAUNCH(c, launch_down_tokens(c->L(), d, w.down_type, w.down_exps, c->h, c->sel, y, n, c->efirst, c->ecount, w.down_shexp));
    c->prof_mark("moe.dn");
    return QKM_OK;
}

// Generic prefill sequence on the raw layout (any supported shape and type).
static int prefill_generic(qkm_ctx* c, const qkm_layer_dev& ld, const float* x, uint32_t n, float* y) {
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    if (!c->contrib) {
        QKM_CUDA(c, cudaMalloc((void**)&c->contrib, (size_t)c->cfg.max_tokens * d.n_used * d.n_embd * sizeof(float)));
    }
    QKM_LAUNCH(c, launch_route_select(c->L(), d, w.router_type, w.router, w.gate_inp_shexp, x, c->sel, n, c->route_scratch, c->route_scratch_bytes));
    QKM_LAUNCH(c, launch_group_pairs(c->L(), d, c->sel, n, c->offsets, c->pairs, c->efirst, c->ecount));
    QKM_LAUNCH(c, launch_shared_gateup(c->L(), d, w.gate_shexp, w.up_shexp, x, c->h, n));
    QKM_LAUNCH(c, launch_gateup_pairs(c->L(), d, w.gateup_type, w.gate_exps, w.up_exps, x, c->offsets, c->pairs, c->h, n, c->efirst, c->ecount));
    QKM_CUDA(c, cudaMemsetAsync(c->contrib, 0, (size_t)n * d.n_used * d.n_embd * sizeof(float), c->stream));
    QKM_LAUNCH(c, launch_down_pairs(c->L(), d, w.down_type, w.down_exps, c->h, c->sel, c->offsets, c->pairs, c->contrib, n, c->efirst, c->ecount));
    QKM_LAUNCH(c, launch_shared_down(c->L(), d, w.down_shexp, c->h, c->sel, c->y2, n));
    QKM_LAUNCH(c, launch_fold_contrib(c->L(), d, c->contrib, c->y2, y, n));
    return QKM_OK;
}

// Scratch of the tensor-core (tcgen05) sequences, allocated on first use.
static int ensure_prefill_scratch(qkm_ctx* c) {
    if (c->xb) return QKM_OK;
    const qkm_dims& d = c->cfg.dims;
    const size_t T = c->cfg.max_tokens, rows = T * (d.n_used + 1);
    const uint32_t NT = kWgemmRows;
    const size_t max_tiles = d.n_expert + (T * d.n_used + NT - 1) / NT + (T + NT - 1) / NT;   // the shared expert's last
    const Want want[] = {
        {&c->xb, T * d.n_embd * 2},
        {(void**)&c->xnorm, T * sizeof(float)},
        {&c->hb, rows * d.n_ff * 2},
        {(void**)&c->hscale, rows * sizeof(float)},
        {(void**)&c->contrib_p, rows * d.n_embd * sizeof(float)},
        {(void**)&c->mma_items[0], max_tiles * (d.n_ff / 128) * sizeof(MmaItem)},
        {(void**)&c->mma_items[1], max_tiles * (d.n_embd / 256) * sizeof(MmaItem)},
        {(void**)&c->pos_of, rows * sizeof(uint32_t)},
        {(void**)&c->group_counts, (c->ecount + T * d.n_used) * sizeof(uint32_t)},
    };
    QKM_CUDA(c, dev_alloc_all(want));
    return QKM_OK;
}

// work lists of the GEMMs from c->group_counts; with_routed false: of the shared expert's rows only; picked: see mean_pairs
static int expert_plan(qkm_ctx* c, const qkm_sel* sel, uint32_t n, bool with_routed, uint32_t sh_first, uint32_t sh_count, bool picked = false) {
    const qkm_dims& d = c->cfg.dims;
    GroupPlace g{};
    g.counts = c->group_counts; g.ranks = c->group_counts + c->ecount; g.sel = sel; g.n_tokens = n; g.n_used = d.n_used; g.n_expert = d.n_expert;
    g.expert_first = c->efirst; g.expert_count = with_routed ? c->ecount : 0; g.sh_first = sh_first; g.sh_count = sh_count;
    g.tile = c->unit_rows = with_routed ? wgemm_rows_per_unit(mean_pairs(n, d.n_used, d.n_expert, c->ecount, picked)) : kWgemmRows; g.rt_gu = d.n_ff / 128; g.rt_dn = d.n_embd / 256; g.pairs = c->pairs; g.pos_of = c->pos_of;
    g.items_gu = c->mma_items[0]; g.items_dn = c->mma_items[1]; g.n_items = c->n_items;
    QKM_LAUNCH(c, launch_group_place(c->L(), g));
    return QKM_OK;
}

// The two expert GEMMs over the work lists of expert_plan: c->xb (f16 rows; c->xscale, c->xnorm) -> c->hb -> c->contrib_p.
// n rows; at most np_max routed pairs and sh_max rows of the shared expert.
static int expert_gemms(qkm_ctx* c, const qkm_layer_dev& ld, const qkm_sel* sel, uint32_t n, uint32_t np_max, uint32_t sh_max) {
    const qkm_dims& d = c->cfg.dims;
    const uint32_t NT = c->unit_rows;
    const uint32_t tiles = (c->ecount < np_max ? c->ecount + (np_max + NT - 1) / NT : np_max) + (sh_max + NT - 1) / NT;
    WgemmExperts g{{ld.tiles[2], ld.tiles[3]}, {ld.tiles[5], ld.tiles[6]}, c->mma_items[0], c->n_items, c->n_items + 2, c->pairs, c->lut_pf, c->status, c->ecount, (uint32_t)c->n_sms, NT};
    QKM_LAUNCH(c, launch_wgemm_gateup(c->L(), d, ld.w.gateup_type, g, c->xb, c->xscale, c->xnorm, ld.w_norm, c->hb, c->hscale, tiles * (d.n_ff / 128)));
    c->prof_mark("moe.gu");
    HiddenRows r{};
    r.pairs = c->pairs; r.pos_of = c->pos_of; r.sel = sel; r.xrows = (const __half*)c->xb; r.x_inv_scale = c->xscale; r.x_norm = c->xnorm; r.w_norm = ld.w_norm;
    r.w[0] = (const uint8_t*)ld.w.gate_exps; r.w[1] = (const uint8_t*)ld.w.up_exps; r.sh[0] = (const uint8_t*)ld.w.gate_shexp; r.sh[1] = (const uint8_t*)ld.w.up_shexp;
    r.h = (__half*)c->hb; r.h_inv_scale = c->hscale; r.n_tokens = n; r.n_used = d.n_used; r.n_expert = d.n_expert; r.expert_first = c->efirst;
    r.expert_count = c->ecount; r.n_ff = d.n_ff; r.n_embd = d.n_embd;
    QKM_LAUNCH(c, launch_hidden_rows_check(c->L(), ld.w.gateup_type, r));
    c->prof_mark("moe.h_check");
    WgemmExperts m{{ld.tiles[4], nullptr}, {ld.tiles[7], nullptr}, c->mma_items[1], c->n_items + 1, c->n_items + 3, c->pairs, c->lut_pf, c->status, c->ecount, (uint32_t)c->n_sms, NT};
    QKM_LAUNCH(c, launch_wgemm_down(c->L(), d, ld.w.down_type, m, c->hb, (uint64_t)c->cfg.max_tokens * (d.n_used + 1), c->hscale, sel, c->contrib_p,
                                    tiles * (d.n_embd / 256)));
    c->prof_mark("moe.dn");
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_prefill(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, float* y) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (!x || !y) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    const qkm_layer_dev& ld = c->layers[layer];
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    if (!ld.fused_ok || n == 0) return prefill_generic(c, ld, x, n, y);
    // tensor-core path: tokens grouped by expert, expert GEMMs on tcgen05 with f16 operands; the shared expert's units
    // ride in the same two launches
    if (int rc = ensure_prefill_scratch(c)) return rc;
    c->prof_begin();
    QKM_LAUNCH(c, launch_f16_rows(c->L(), x, c->xb, c->xscale, c->xnorm, n, d.n_embd, c->group_counts, c->ecount));
    RouteExtra ex;
    ex.x_f16 = c->xb; ex.x_f16_inv = c->xscale; ex.router_f16 = ld.router16; ex.router_norm2 = ld.router_norm2; ex.status = c->status;
    ex.counts = c->group_counts; ex.ranks = c->group_counts + c->ecount; ex.expert_first = c->efirst; ex.expert_count = c->ecount;
    QKM_LAUNCH(c, launch_route_select(c->L(), d, w.router_type, w.router, w.gate_inp_shexp, x, c->sel, n, c->route_scratch, c->route_scratch_bytes, ex));
    c->prof_mark("moe.route");
    if (int rc = expert_plan(c, c->sel, n, true, 0, n)) return rc;
    c->prof_mark("moe.pairs");
    if (int rc = expert_gemms(c, ld, c->sel, n, n * d.n_used, n)) return rc;
    QKM_LAUNCH(c, launch_fold_pairs(c->L(), d, c->contrib_p, c->pos_of, y, n));
    c->prof_mark("moe.fold");
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_forward_host(qkm_ctx* c, uint32_t layer, int mode, const float* x_host,
                                            uint32_t n, float* y_host) {
    if (!c || !x_host || !y_host) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    const size_t bytes = (size_t)n * c->cfg.dims.n_embd * sizeof(float);
    QKM_CUDA(c, cudaMemcpyAsync(c->x_stage, x_host, bytes, cudaMemcpyHostToDevice, c->stream));
    const int rc = mode == 0 ? qkm_moe_decode(c, layer, c->x_stage, n, c->y_stage)
                             : qkm_moe_prefill(c, layer, c->x_stage, n, c->y_stage);
    if (rc) return rc;
    QKM_CUDA(c, cudaMemcpyAsync(y_host, c->y_stage, bytes, cudaMemcpyDeviceToHost, c->stream));
    return check_status(c);
}

static int decode_stack_eager(qkm_ctx* c, uint32_t first, uint32_t count, const float* x, uint32_t n, float* y) {
    const size_t stride = (size_t)n * c->cfg.dims.n_embd;
    for (uint32_t l = 0; l < count; ++l)
        if (int rc = qkm_moe_decode(c, first + l, x + l * stride, n, y + l * stride)) return rc;
    return QKM_OK;
}

// Layers of the fused sequence go through each of its stages together: three or four launches for the stack, not for a layer (40 layers of
// 16 tokens 2,740 us as a graph of their launches, 1,870 to 1,990 together; 24 layers of one token 560 and 114).  What is left - an output that
// overlaps a later layer's input, a layer outside the fused sequence - goes layer by layer: the launches are captured into a CUDA graph the
// first time an argument set is seen and replayed afterwards.  Capture needs a real stream: on the legacy default stream, while
// profiling, or after an upload, the launches are issued one by one.
extern "C" QKM_API int qkm_moe_decode_stack(qkm_ctx* c, uint32_t first, uint32_t count, const float* x,
                                            uint32_t n, float* y) {
    if (!c || !x || !y) return QKM_ERR_ARG;
    if ((uint64_t)first + count > c->cfg.n_layer) return fail(c, QKM_ERR_BOUNDS, "layers [%u,%u) out of range", first, first + count);
    if (int rc = check_tokens(c, n)) return rc;
    for (uint32_t l = 0; l < count; ++l)
        if (int rc = layer_ready(c, first + l)) return rc;
    // every layer's rows are at hand: the layers go through each stage together, unless an output overlaps a later layer's input
    const qkm_dims& d = c->cfg.dims;
    const uint64_t stride = (uint64_t)n * d.n_embd, xa = (uint64_t)(uintptr_t)x, ya = (uint64_t)(uintptr_t)y, bytes = count * stride * sizeof(float);
    bool together = decode_fused_ok(c, n) && (xa == ya || xa + bytes <= ya || ya + bytes <= xa);
    for (uint32_t l = 0; l < count && together; ++l) together = c->layers[first + l].fused_ok;
    if (together) {
        c->prof_begin();
        return decode_layers(c, first, count, x, stride, n, y, stride);
    }
    if (c->stream == nullptr || c->profiling || count < 2) return decode_stack_eager(c, first, count, x, n, y);
    qkm_ctx::StackGraph* g = nullptr;
    for (auto& e : c->stack_graphs)
        if (e.exec && e.first == first && e.count == count && e.n == n && e.x == x && e.y == y && e.stream == c->stream) g = &e;
    if (!g) {
        qkm_ctx::StackGraph* slot = &c->stack_graphs[0];
        for (auto& e : c->stack_graphs) {
            if (!e.exec) { slot = &e; break; }
            if (e.used < slot->used) slot = &e;
        }
        if (slot->exec) { cudaGraphExecDestroy(slot->exec); slot->exec = nullptr; }
        const uint64_t before = c->launches;
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            return decode_stack_eager(c, first, count, x, n, y);
        }
        const int rc = decode_stack_eager(c, first, count, x, n, y);
        cudaGraph_t graph = nullptr;
        const cudaError_t e = cudaStreamEndCapture(c->stream, &graph);
        slot->launches = c->launches - before;
        c->launches = before;
        if (rc != QKM_OK || e != cudaSuccess || !graph) {
            if (graph) cudaGraphDestroy(graph);
            cudaGetLastError();
            return rc != QKM_OK ? rc : decode_stack_eager(c, first, count, x, n, y);
        }
        const cudaError_t ei = cudaGraphInstantiate(&slot->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ei != cudaSuccess) {
            slot->exec = nullptr;
            cudaGetLastError();
            return decode_stack_eager(c, first, count, x, n, y);
        }
        slot->first = first; slot->count = count; slot->n = n; slot->x = x; slot->y = y; slot->stream = c->stream;
        g = slot;
    }
    g->used = ++c->stack_clock;
    QKM_CUDA(c, cudaGraphLaunch(g->exec, c->stream));
    c->launches += g->launches;
    return QKM_OK;
}

extern "C" QKM_API int qkm_moe_decode_stack_host(qkm_ctx* c, uint32_t first, uint32_t count,
                                                 const float* x_host, uint32_t n, float* y_host) {
    if (!c || !x_host || !y_host) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    if ((uint64_t)first + count > c->cfg.n_layer) return fail(c, QKM_ERR_BOUNDS, "layers [%u,%u) out of range", first, first + count);
    if (!c->stack_x) {
        const size_t cap = (size_t)c->cfg.n_layer * c->cfg.max_tokens * c->cfg.dims.n_embd * sizeof(float);
        const Want want[] = {{(void**)&c->stack_x, cap}, {(void**)&c->stack_y, cap}};
        QKM_CUDA(c, dev_alloc_all(want));
    }
    const size_t layer_elems = (size_t)n * c->cfg.dims.n_embd;
    const size_t bytes = (size_t)count * layer_elems * sizeof(float);
    if (c->stream == nullptr || c->profiling || bytes < qkm_ctx::kStackChunkBytes || count < 2u * qkm_ctx::kStackChunks) {
        QKM_CUDA(c, cudaMemcpyAsync(c->stack_x, x_host, bytes, cudaMemcpyHostToDevice, c->stream));
        if (int rc = qkm_moe_decode_stack(c, first, count, c->stack_x, n, c->stack_y)) return rc;
        QKM_CUDA(c, cudaMemcpyAsync(y_host, c->stack_y, bytes, cudaMemcpyDeviceToHost, c->stream));
        return check_status(c);
    }
    // Chunks of layers: all input copies are queued on their own stream at once, chunk k computes as soon
    // as its rows are there, and its outputs leave on a third stream while chunk k+1 computes.  Only the
    // first chunk's copy in and the last chunk's copy out are not hidden, so these two chunks are short (a sixteenth: their layers
    // take longer than the copies of the rest).  A chunk more costs about 25 us, since its layers do not go with the others', and a
    // copy that is not hidden 1 us per 55 KB: below 1.5 MB the whole stack is one chunk.
    if (!c->ev_copies) {   // made last; what an earlier try got is kept
        for (cudaStream_t* s : {&c->copy_in, &c->copy_out}) if (!*s) QKM_CUDA(c, cudaStreamCreateWithFlags(s, cudaStreamNonBlocking));
        for (cudaEvent_t& ev : c->ev_in) if (!ev) QKM_CUDA(c, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        for (cudaEvent_t& ev : c->ev_out) if (!ev) QKM_CUDA(c, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        QKM_CUDA(c, cudaEventCreateWithFlags(&c->ev_copies, cudaEventDisableTiming));
    }
    constexpr uint32_t K = qkm_ctx::kStackChunks;
    static_assert(K == 3, "chunk boundaries below are written for three chunks");
    const uint32_t ends = (count + 15u) / 16u, lo[K + 1] = {0u, ends, count - ends, count};
    // whatever the stream still holds (it reads or writes the staging buffers) comes first
    QKM_CUDA(c, cudaEventRecord(c->ev_copies, c->stream));
    QKM_CUDA(c, cudaStreamWaitEvent(c->copy_in, c->ev_copies, 0));
    for (uint32_t k = 0; k < K; ++k) {
        const size_t off = lo[k] * layer_elems, len = (size_t)(lo[k + 1] - lo[k]) * layer_elems * sizeof(float);
        QKM_CUDA(c, cudaMemcpyAsync(c->stack_x + off, x_host + off, len, cudaMemcpyHostToDevice, c->copy_in));
        QKM_CUDA(c, cudaEventRecord(c->ev_in[k], c->copy_in));
    }
    for (uint32_t k = 0; k < K; ++k) {
        const size_t off = lo[k] * layer_elems, len = (size_t)(lo[k + 1] - lo[k]) * layer_elems * sizeof(float);
        QKM_CUDA(c, cudaStreamWaitEvent(c->stream, c->ev_in[k], 0));
        if (int rc = qkm_moe_decode_stack(c, first + lo[k], lo[k + 1] - lo[k], c->stack_x + off, n, c->stack_y + off)) return rc;
        QKM_CUDA(c, cudaEventRecord(c->ev_out[k], c->stream));
        QKM_CUDA(c, cudaStreamWaitEvent(c->copy_out, c->ev_out[k], 0));
        QKM_CUDA(c, cudaMemcpyAsync(y_host + off, c->stack_y + off, len, cudaMemcpyDeviceToHost, c->copy_out));
    }
    QKM_CUDA(c, cudaEventRecord(c->ev_copies, c->copy_out));
    QKM_CUDA(c, cudaStreamWaitEvent(c->stream, c->ev_copies, 0));   // the stream's synchronise below covers the copies
    return check_status(c);
}

extern "C" QKM_API int qkm_profile_enable(qkm_ctx* c, int on) {
    if (!c) return QKM_ERR_ARG;
    if (on && !c->prof_ev[0])
        for (cudaEvent_t& ev : c->prof_ev) QKM_CUDA(c, cudaEventCreate(&ev));
    c->profiling = on != 0;
    c->prof_n = 0;
    return QKM_OK;
}

extern "C" QKM_API int qkm_profile_read(qkm_ctx* c, char* labels, float* ms, uint32_t max_stages) {
    if (!c || !labels || !ms) return QKM_ERR_ARG;
    if (!c->profiling) return fail(c, QKM_ERR_MODE, "profiling is not enabled");
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    const int n = c->prof_n < (int)max_stages ? c->prof_n : (int)max_stages;
    for (int i = 0; i < n; ++i) {
        memcpy(labels + 16 * i, c->prof_label[i], 16);
        QKM_CUDA(c, cudaEventElapsedTime(&ms[i], c->prof_ev[i], c->prof_ev[i + 1]));
    }
    return n;
}

extern "C" QKM_API int qkm_last_sel(qkm_ctx* c, qkm_sel* sel_host, uint32_t n) {
    if (!c || !sel_host) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    return qkm_d2h(c, sel_host, c->sel, (size_t)n * sizeof(qkm_sel));
}
extern "C" QKM_API const qkm_sel* qkm_sel_device(const qkm_ctx* c) { return c ? c->sel : nullptr; }
extern "C" QKM_API const float* qkm_h_device(const qkm_ctx* c) { return c ? c->h : nullptr; }

// ---------------------------------------------------------------- dense quantised GEMM
// The reference's batched-prefill projections (gemm_q8_0*.comp, gemm_iq4_xs.comp; dispatched at
// src/main.cpp:4806-4835): Y[n][M] = X[n][K] . W^T with W a Q8_0 or IQ4_XS matrix.  The matrix is
// uploaded once into a slot (copied and tile-ordered on the device); the GEMM runs on the experts'
// tcgen05 kernel (qkm_wgemm.cu): weights expanded to f16 in tensor memory, x rows as f16 scaled by powers of two.

extern "C" QKM_API int qkm_dense_upload(qkm_ctx* c, uint32_t slot, uint32_t type, const void* w_host, uint32_t M, uint32_t K) {
    if (!c || !w_host) return QKM_ERR_ARG;
    if (slot >= qkm_ctx::kDenseSlots) return fail(c, QKM_ERR_BOUNDS, "dense slot %u out of range", slot);
    if (type != QKM_TYPE_Q8_0 && type != QKM_TYPE_IQ4_XS) return fail(c, QKM_ERR_TYPE, "qkm_dense_upload: type %u (Q8_0 or IQ4_XS)", type);
    if (M == 0 || M % 128 || K == 0 || K % 256) return fail(c, QKM_ERR_ARG, "qkm_dense_upload: M %% 128 and K %% 256 must be 0 (M=%u K=%u)", M, K);
    auto& dm = c->dense[slot];
    if (dm.tiles) { QKM_CUDA(c, cudaFree(dm.tiles)); dm = qkm_ctx::Dense{}; }
    const size_t bytes = (size_t)M * row_bytes(type, K), tbytes = tiled_bytes(type, 1, M, K);
    void* raw = nullptr;
    QKM_CUDA(c, cudaMalloc(&raw, bytes + 256));
    cudaError_t e = cudaMalloc(&dm.tiles, tbytes + 256);
    if (e == cudaSuccess) e = cudaMemcpyAsync(raw, w_host, bytes, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync((uint8_t*)dm.tiles + tbytes, 0, 256, c->stream);
    if (e == cudaSuccess) e = launch_repack(c->L(), type, raw, dm.tiles, 1, M, K);
    // the largest block scale, by way of the spare bytes behind the tiles
    uint32_t* spare = (uint32_t*)((uint8_t*)dm.tiles + tbytes);
    uint32_t d_bits = 0;
    if (e == cudaSuccess) e = launch_scale_max(c->L(), type, raw, spare, M, K);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&d_bits, spare, sizeof d_bits, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    cudaFree(raw);
    if (e != cudaSuccess) {
        if (dm.tiles) cudaFree(dm.tiles);
        dm = qkm_ctx::Dense{};
        return fail(c, QKM_ERR_CUDA, "qkm_dense_upload: %s", cudaGetErrorString(e));
    }
    dm.type = type; dm.M = M; dm.K = K; dm.w_scale = dense_weight_scale(type, d_bits);
    return QKM_OK;
}

extern "C" QKM_API int qkm_dense_gemm(qkm_ctx* c, uint32_t slot, const float* x, uint32_t n, float* y) {
    if (!c || !x || !y) return QKM_ERR_ARG;
    if (slot >= qkm_ctx::kDenseSlots || !c->dense[slot].tiles) return fail(c, QKM_ERR_BUSY, "dense slot %u holds no matrix", slot);
    if (n == 0) return QKM_OK;
    const auto& dm = c->dense[slot];
    const size_t elems = (size_t)n * dm.K;
    if (elems > c->dense_cap_elems) {
        if (c->dense_xb) QKM_CUDA(c, cudaFree(c->dense_xb));
        c->dense_xb = nullptr; c->dense_cap_elems = 0;
        QKM_CUDA(c, cudaMalloc(&c->dense_xb, elems * 2));
        c->dense_cap_elems = elems;
    }
    if (n > c->dense_cap_rows) {
        if (c->dense_scale) QKM_CUDA(c, cudaFree(c->dense_scale));
        c->dense_scale = nullptr; c->dense_cap_rows = 0;
        QKM_CUDA(c, cudaMalloc((void**)&c->dense_scale, (size_t)n * sizeof(float)));
        c->dense_cap_rows = n;
    }
    QKM_LAUNCH(c, launch_dense_gemm(c->L(), dm.type, dm.tiles, dm.w_scale, dm.M, dm.K, x, n, y, c->dense_xb, c->dense_scale, c->lut_pf, (uint32_t)c->n_sms, c->status));
    return QKM_OK;
}

// ---------------------------------------------------------------- layer entry / tail

extern "C" QKM_API int qkm_add_rmsnorm(qkm_ctx* c, const float* a, const float* b, const float* w, float* y, float* xn,
                                       uint32_t n_rows, uint32_t n, float eps) {
    if (!c || !a || !b || !w || !y || !xn) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_add_rms(c->L(), 0, a, b, nullptr, w, y, xn, n_rows, n, 0, eps));
    return QKM_OK;
}

extern "C" QKM_API int qkm_add_rms3(qkm_ctx* c, const float* a, const float* b, const float* c2, const float* w,
                                    float* s, float* xn, uint32_t n_rows, uint32_t n, float eps) {
    if (!c || !a || !b || !c2 || !w || !s || !xn) return QKM_ERR_ARG;
    QKM_LAUNCH(c, launch_add_rms(c->L(), 1, a, b, c2, w, s, xn, n_rows, n, 0, eps));
    return QKM_OK;
}

extern "C" QKM_API int qkm_add_rms3_grouped(qkm_ctx* c, const float* a, const float* routed, const float* c2,
                                            const float* w, float* s, float* xn, uint32_t n_rows, uint32_t n,
                                            uint32_t n_used, float eps) {
    if (!c || !a || !routed || !c2 || !w || !s || !xn) return QKM_ERR_ARG;
    if (n_used == 0 || n_used > 16) return fail(c, QKM_ERR_ARG, "qkm_add_rms3_grouped: n_used %u", n_used);
    QKM_LAUNCH(c, launch_add_rms(c->L(), 2, a, routed, c2, w, s, xn, n_rows, n, n_used, eps));
    return QKM_OK;
}

extern "C" QKM_API int qkm_argmax(qkm_ctx* c, const float* logits, uint32_t n_rows, uint32_t n, uint32_t* tok) {
    if (!c || !logits || !tok) return QKM_ERR_ARG;
    if (n_rows > c->argmax_rows) {
        if (c->argmax_scratch) QKM_CUDA(c, cudaFree(c->argmax_scratch));
        c->argmax_scratch = nullptr; c->argmax_rows = 0;
        QKM_CUDA(c, cudaMalloc(&c->argmax_scratch, argmax_scratch_bytes(n_rows)));
        QKM_CUDA(c, cudaMemsetAsync(c->argmax_scratch, 0, argmax_scratch_bytes(n_rows), c->stream));
        c->argmax_rows = n_rows;
    }
    QKM_LAUNCH(c, launch_argmax(c->L(), logits, n_rows, n, c->argmax_scratch, c->argmax_rows, tok));
    return QKM_OK;
}

// One decoder layer's feed-forward half as the engine runs it (src/main.cpp:4375-4404):
// resid2 = resid + attn_out, xn2 = rmsnorm(resid2) * w_post; y = MoE(xn2);
// resid_out = resid2 + y, xn_next = rmsnorm(resid_out) * w_next.
extern "C" QKM_API int qkm_moe_layer_step(qkm_ctx* c, uint32_t layer, const float* resid, const float* attn_out,
                                          const float* w_post, const float* w_next, uint32_t n, float eps,
                                          float* resid_out, float* xn_next) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (!resid || !attn_out || !w_post || !w_next || !resid_out || !xn_next) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    const qkm_dims& d = c->cfg.dims;
    // x_stage / y_stage double as resid2 / MoE output scratch ([max_tokens][n_embd] each)
    float* xn2 = c->x_stage;
    QKM_LAUNCH(c, launch_add_rms(c->L(), 0, resid, attn_out, nullptr, w_post, resid_out, xn2, n, d.n_embd, 0, eps));
    const int rc = n <= 64 ? qkm_moe_decode(c, layer, xn2, n, c->y_stage) : qkm_moe_prefill(c, layer, xn2, n, c->y_stage);
    if (rc) return rc;
    QKM_LAUNCH(c, launch_add_rms(c->L(), 0, resid_out, c->y_stage, nullptr, w_next, resid_out, xn_next, n, d.n_embd, 0, eps));
    return QKM_OK;
}

// ---------------------------------------------------------------- expert parallel
// One context per GPU, opened with expert_first/expert_count naming its shard.  Per layer:
//   qkm_ep_dispatch  : route the local tokens, decide which rows go to which rank, pack them
//   (host: all-to-all of the rows and their selection records)
//   qkm_ep_shared    : the shared expert of the local tokens (runs while the rows travel)
//   qkm_ep_expert_forward : resident experts over the received rows -> one partial row each
//   (host: all-to-all of the partial rows back)
//   qkm_ep_combine   : y = shared + partials, summed in rank order
// The reference has no multi-GPU path; the sequence keeps its single-GPU arithmetic
// (src/main.cpp:1316-1387) and only changes the order in which a token's slots are summed.

static int ep_check(qkm_ctx* c, uint32_t n_ranks) {
    const qkm_dims& d = c->cfg.dims;
    if (n_ranks == 0 || n_ranks > 64 || d.n_expert % n_ranks) return fail(c, QKM_ERR_ARG, "n_ranks %u does not divide n_expert %u", n_ranks, d.n_expert);
    if (c->ecount != d.n_expert / n_ranks || c->efirst % c->ecount)
        return fail(c, QKM_ERR_MODE, "context holds experts [%u,%u): not one of %u equal shards", c->efirst, c->efirst + c->ecount, n_ranks);
    if (c->ep_ranks != n_ranks) {
        for (void* p : {c->ep_counts, c->ep_send_tok, c->ep_send_pos}) if (p) cudaFree(p);
        if (c->ep_counts_host) cudaFreeHost(c->ep_counts_host);
        c->ep_counts = c->ep_send_tok = c->ep_send_pos = c->ep_counts_host = nullptr;
        c->ep_ranks = 0;
        const size_t T = c->cfg.max_tokens, fan = n_ranks < d.n_used ? n_ranks : d.n_used;
        const Want want[] = {{(void**)&c->ep_counts, (n_ranks + 1) * sizeof(uint32_t)},
                             {(void**)&c->ep_send_tok, T * fan * sizeof(uint32_t)},
                             {(void**)&c->ep_send_pos, T * n_ranks * sizeof(uint32_t)}};
        QKM_CUDA(c, dev_alloc_all(want));
        QKM_CUDA(c, cudaMallocHost((void**)&c->ep_counts_host, (n_ranks + 1) * sizeof(uint32_t)));
        c->ep_ranks = n_ranks;
    }
    return QKM_OK;
}

// the shared expert of so few local tokens runs on the decode kernels
static bool ep_shared_decode(const qkm_ctx* c, const qkm_layer_dev& ld, uint32_t n) { return ld.tiles_ok && n <= 64 && c->dec_ok && decode_down_any_ok(c->cfg.dims); }

// router logits and selection of the n local tokens into c->sel (digit planes / f16 rows as the
// shared-expert kernels of that size want them)
static int ep_route_local(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n) {
    const qkm_layer_dev& ld = c->layers[layer];
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    const bool planes = ep_shared_decode(c, ld, n);   // the decode kernels of the shared expert read digit planes
    const bool tc = ld.tiles_ok && n > 64;        // tensor-core logits from f16 rows
    RouteExtra ex;
    if (planes) { ex.xplanes = c->planes8; ex.xscale = c->xscale; }
    if (tc) {
        if (int rc = ensure_prefill_scratch(c)) return rc;
        QKM_LAUNCH(c, launch_f16_rows(c->L(), x, c->xb, c->xscale, c->xnorm, n, d.n_embd));
        ex.x_f16 = c->xb; ex.x_f16_inv = c->xscale; ex.router_f16 = ld.router16; ex.router_norm2 = ld.router_norm2; ex.status = c->status;
    }
    QKM_LAUNCH(c, launch_route_select(c->L(), d, w.router_type, w.router, w.gate_inp_shexp, x, c->sel, n, c->route_scratch, c->route_scratch_bytes, ex));
    return QKM_OK;
}

static int ep_dispatch_launch(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, uint32_t n_ranks,
                              float* xsend, qkm_sel* selsend) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (!x || !xsend || !selsend) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    if (int rc = ep_check(c, n_ranks)) return rc;
    if (int rc = ep_route_local(c, layer, x, n)) return rc;
    const qkm_dims& d = c->cfg.dims;
    QKM_LAUNCH(c, launch_ep_plan(c->L(), d, c->sel, n, n_ranks, c->ep_counts, c->ep_send_tok, c->ep_send_pos));
    const uint32_t fan = n_ranks < d.n_used ? n_ranks : d.n_used;
    QKM_LAUNCH(c, launch_ep_pack(c->L(), d, x, c->sel, c->ep_send_tok, c->ep_counts + n_ranks, n * fan, xsend, selsend));
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_dispatch(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, uint32_t n_ranks,
                                       float* xsend, qkm_sel* selsend, uint32_t* counts_host) {
    if (!counts_host) return QKM_ERR_ARG;
    if (int rc = ep_dispatch_launch(c, layer, x, n, n_ranks, xsend, selsend)) return rc;
    QKM_CUDA(c, cudaMemcpyAsync(c->ep_counts_host, c->ep_counts, (n_ranks + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
    QKM_CUDA(c, cudaStreamSynchronize(c->stream));
    memcpy(counts_host, c->ep_counts_host, n_ranks * sizeof(uint32_t));
    return QKM_OK;
}

// The same without touching the host: the row counts go to a device buffer of the caller
// (n_ranks 32-bit words), so they can feed the collective that exchanges them directly.
extern "C" QKM_API int qkm_ep_dispatch_dev(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, uint32_t n_ranks,
                                           float* xsend, qkm_sel* selsend, uint32_t* counts_dev) {
    if (!counts_dev) return QKM_ERR_ARG;
    if (int rc = ep_dispatch_launch(c, layer, x, n, n_ranks, xsend, selsend)) return rc;
    QKM_CUDA(c, cudaMemcpyAsync(counts_dev, c->ep_counts, n_ranks * sizeof(uint32_t), cudaMemcpyDeviceToDevice, c->stream));
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_shared(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (!x) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    if (n == 0) return QKM_OK;
    const qkm_layer_dev& ld = c->layers[layer];
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    const bool dec = ep_shared_decode(c, ld, n);
    if (!dec && (!ld.tiles_ok || n <= 64)) {
        QKM_LAUNCH(c, launch_shared_gateup(c->L(), d, w.gate_shexp, w.up_shexp, x, c->h, n));
        QKM_LAUNCH(c, launch_shared_down(c->L(), d, w.down_shexp, c->h, c->sel, c->y2, n));
        return QKM_OK;
    }
    if (dec) {   // the decode kernels without routed experts (digit planes written by qkm_ep_dispatch)
        GateupDecodeArgs ga{};
        ga.layer[0] = {nullptr, nullptr, (const uint8_t*)ld.tiles[5], (const uint8_t*)ld.tiles[6]};   // no groups: the shared expert's only
        ga.luts = c->lut_gu; ga.planes = c->planes8; ga.xscale = c->xscale; ga.n_tokens = n; ga.n_layers = 1; ga.gateup_type = w.gateup_type;
        ga.h_last = c->h; ga.status = c->status; ga.d = d;
        QKM_LAUNCH(c, launch_decode_gateup(c->L(), ga, (uint32_t)c->n_sms));
        DownDecodeArgs da{};
        da.layer[0] = {nullptr, (const uint8_t*)ld.tiles[7]};
        da.h_last = c->h; da.sel_last = c->sel; da.y = c->y2; da.n_tokens = n; da.n_layers = 1; da.status = c->status; da.d = d;
        QKM_LAUNCH(c, launch_decode_down_any(c->L(), da, w.down_type, (uint32_t)c->n_sms));
        return QKM_OK;
    }
    // tensor-core kernels with an empty routed list: only the shared expert's tiles
    if (int rc = ensure_prefill_scratch(c)) return rc;
    if (int rc = expert_plan(c, c->sel, n, false, 0, n)) return rc;
    QKM_LAUNCH(c, launch_f16_rows(c->L(), x, c->xb, c->xscale, c->xnorm, n, d.n_embd));
    if (int rc = expert_gemms(c, ld, c->sel, n, 0, n)) return rc;   // the routed list is empty
    QKM_LAUNCH(c, launch_fold_pairs(c->L(), d, c->contrib_p, c->pos_of, c->y2, n));
    return QKM_OK;
}

// Resident experts over n_recv rows -> partial.  with_shared: rows [sh_first, sh_first + sh_count)
// are this rank's own tokens and also get the shared expert (its units ride in the routed experts'
// launches, as in qkm_moe_prefill), so their partial rows carry shared + routed.
// slot_rows_peer != 0: the rows are slots of the peer-memory form and every live partial row is
// stored into its source rank's return buffer instead of staying in `partial`.
static int ep_expert_forward_impl(qkm_ctx* c, uint32_t layer, const float* xrecv, const qkm_sel* selrecv, uint32_t n_recv,
                                  float* partial, bool with_shared, uint32_t sh_first, uint32_t sh_count,
                                  uint32_t slot_rows_peer = 0, bool rows_f16 = false) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (n_recv == 0) return QKM_OK;
    if (!xrecv || !selrecv || !partial) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n_recv)) return rc;
    const qkm_layer_dev& ld = c->layers[layer];
    const qkm_layer_weights& w = ld.w;
    const qkm_dims& d = c->cfg.dims;
    if (!ld.tiles_ok) {   // generic kernels on the raw layout
        const float* y2 = nullptr;
        if (with_shared && sh_count) {   // shared expert of the own rows first (it uses h too), added by the fold
            const float* xo = xrecv + (size_t)sh_first * d.n_embd;
            QKM_CUDA(c, cudaMemsetAsync(c->y2, 0, (size_t)n_recv * d.n_embd * sizeof(float), c->stream));
            QKM_LAUNCH(c, launch_shared_gateup(c->L(), d, w.gate_shexp, w.up_shexp, xo, c->h, sh_count));
            QKM_LAUNCH(c, launch_shared_down(c->L(), d, w.down_shexp, c->h, selrecv + sh_first, c->y2 + (size_t)sh_first * d.n_embd, sh_count));
            y2 = c->y2;
        }
        QKM_LAUNCH(c, launch_group_pairs(c->L(), d, selrecv, n_recv, c->offsets, c->pairs, c->efirst, c->ecount));
        if (!c->contrib) QKM_CUDA(c, cudaMalloc((void**)&c->contrib, (size_t)c->cfg.max_tokens * d.n_used * d.n_embd * sizeof(float)));
        QKM_LAUNCH(c, launch_gateup_pairs(c->L(), d, w.gateup_type, w.gate_exps, w.up_exps, xrecv, c->offsets, c->pairs, c->h, n_recv, c->efirst, c->ecount));
        QKM_CUDA(c, cudaMemsetAsync(c->contrib, 0, (size_t)n_recv * d.n_used * d.n_embd * sizeof(float), c->stream));
        QKM_LAUNCH(c, launch_down_pairs(c->L(), d, w.down_type, w.down_exps, c->h, selrecv, c->offsets, c->pairs, c->contrib, n_recv, c->efirst, c->ecount));
        QKM_LAUNCH(c, launch_fold_contrib(c->L(), d, c->contrib, y2, partial, n_recv));
        if (slot_rows_peer)
            QKM_LAUNCH(c, launch_ep_return(c->L(), d, partial, selrecv, c->pm_peers, slot_rows_peer, c->pm_rank, c->pm_ranks,
                                           with_shared ? sh_count : 0));
        return QKM_OK;
    }
    if (int rc = ensure_prefill_scratch(c)) return rc;
    QKM_CUDA(c, cudaMemsetAsync(c->group_counts, 0, c->ecount * sizeof(uint32_t), c->stream));
    QKM_LAUNCH(c, launch_group_rank(c->L(), d, selrecv, n_recv, c->efirst, c->ecount, c->group_counts, c->group_counts + c->ecount));
    if (int rc = expert_plan(c, selrecv, n_recv, true, with_shared ? sh_first : 0, with_shared ? sh_count : 0, slot_rows_peer == 0)) return rc;   // (slots: every row of the sources, empty or not)
    // the rows as scaled f16: converted here, or already so on arrival (then their scales and norms are gathered)
    if (rows_f16) {
        QKM_LAUNCH(c, launch_ep_row_scales(c->L(), selrecv, c->xscale, n_recv));
        QKM_LAUNCH(c, launch_f16_rows_in(c->L(), xrecv, c->xscale, c->xb, c->xnorm, n_recv, d.n_embd));
    } else {
        QKM_LAUNCH(c, launch_f16_rows(c->L(), xrecv, c->xb, c->xscale, c->xnorm, n_recv, d.n_embd));
    }
    if (int rc = expert_gemms(c, ld, selrecv, n_recv, n_recv * d.n_used, with_shared ? sh_count : 0)) return rc;
    if (slot_rows_peer)
        QKM_LAUNCH(c, launch_fold_pairs_peer(c->L(), d, c->contrib_p, c->pos_of, c->pm_peers, slot_rows_peer, c->pm_rank, c->pm_ranks));
    else
        QKM_LAUNCH(c, launch_fold_pairs(c->L(), d, c->contrib_p, c->pos_of, partial, n_recv));
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_expert_forward(qkm_ctx* c, uint32_t layer, const float* xrecv, const qkm_sel* selrecv,
                                             uint32_t n_recv, float* partial) {
    return ep_expert_forward_impl(c, layer, xrecv, selrecv, n_recv, partial, false, 0, 0);
}

extern "C" QKM_API int qkm_ep_combine(qkm_ctx* c, uint32_t n, uint32_t n_ranks, const float* back, float* y) {
    if (!c || !y || (!back && n)) return QKM_ERR_ARG;
    if (int rc = check_tokens(c, n)) return rc;
    if (c->ep_ranks != n_ranks || !c->ep_send_pos) return fail(c, QKM_ERR_MODE, "qkm_ep_combine without a matching qkm_ep_dispatch");
    QKM_LAUNCH(c, launch_ep_combine(c->L(), c->cfg.dims, back, c->ep_send_pos, c->y2, y, n, n_ranks));
    return QKM_OK;
}

// ---------------------------------------------------------------- expert parallel over peer memory
// The same layer without an all-to-all.  Every rank keeps three receive buffers of
// n_ranks * slot_cap rows (x rows, selection records, returned partial rows) and maps every peer's:
//   qkm_ep_peer_setup   : allocate this rank's buffers
//   qkm_ep_peer_export / qkm_ep_peer_import : CUDA IPC handles between processes of one node,
//   or qkm_ep_peer_buffers / qkm_ep_peer_set  : raw pointers (one process driving several GPUs)
// and per layer, with slot_rows (>= every rank's token count, the same on all ranks):
//   qkm_ep_push         : route the local tokens, store rows + records into the owners' buffers
//   qkm_ep_shared       : the shared expert (no dependence on the peers)
//   (host: barrier)     : all pushes have landed
//   qkm_ep_forward_slots: resident experts over the n_ranks * slot_rows rows; each partial row is
//                         stored into its source rank's return buffer
//   (host: barrier)     : all partial rows have landed
//   qkm_ep_pull         : y = shared + the partial rows the owners returned
// The two barriers also order the reuse of the buffers by the next layer: a rank pushes layer
// l+1 after the second barrier of layer l, when every rank has finished reading the rows of l,
// and stores partial rows of l+1 after the first barrier of l+1, which every rank enters after
// its pull of l.  Kernels only store to and load from peer memory; none waits.

constexpr size_t kPmFlagBytes = 256;
static uint32_t* pm_flags_of(const qkm_ctx* c, void* selrecv) {
    return (uint32_t*)((char*)selrecv + (size_t)c->pm_ranks * c->pm_cap * sizeof(qkm_sel));
}

static int pm_check(qkm_ctx* c, uint32_t slot_rows) {
    if (!c) return QKM_ERR_ARG;
    if (!c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup has not been called");
    if (slot_rows == 0 || slot_rows > c->pm_cap) return fail(c, QKM_ERR_BOUNDS, "slot_rows %u outside 1..%u", slot_rows, c->pm_cap);
    for (uint32_t r = 0; r < c->pm_ranks; ++r)
        if (!c->pm_peers.x[r] || !c->pm_peers.sel[r] || !c->pm_peers.back[r] || !c->pm_peers.flags[r])
            return fail(c, QKM_ERR_MODE, "buffers of rank %u are not mapped (qkm_ep_peer_import / qkm_ep_peer_set)", r);
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_peer_setup(qkm_ctx* c, uint32_t n_ranks, uint32_t rank, uint32_t slot_cap) {
    if (!c) return QKM_ERR_ARG;
    const qkm_dims& d = c->cfg.dims;
    if (c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup was already called on this context");
    if (n_ranks == 0 || n_ranks > kMaxPeerRanks || d.n_expert % n_ranks || rank >= n_ranks)
        return fail(c, QKM_ERR_ARG, "rank %u of %u ranks (at most %u, dividing n_expert %u)", rank, n_ranks, kMaxPeerRanks, d.n_expert);
    if (c->ecount != d.n_expert / n_ranks || c->efirst != rank * c->ecount)
        return fail(c, QKM_ERR_MODE, "context holds experts [%u,%u): not shard %u of %u", c->efirst, c->efirst + c->ecount, rank, n_ranks);
    if (slot_cap == 0 || (uint64_t)slot_cap * n_ranks > c->cfg.max_tokens)
        return fail(c, QKM_ERR_BOUNDS, "%u ranks x %u rows exceed max_tokens %u", n_ranks, slot_cap, c->cfg.max_tokens);
    const size_t rows = (size_t)n_ranks * slot_cap;
    QKM_CUDA(c, cudaSetDevice(c->device));
    // all five buffers or none: a failure part way frees what was taken, so a retry starts clean
    cudaError_t e = cudaMalloc((void**)&c->pm_xrecv, rows * d.n_embd * sizeof(float));
    // the barrier words of qkm_ep_barrier sit behind the records, so three mappings carry everything
    if (e == cudaSuccess) e = cudaMalloc((void**)&c->pm_selrecv, rows * sizeof(qkm_sel) + kPmFlagBytes);
    if (e == cudaSuccess) e = cudaMemset((char*)c->pm_selrecv + rows * sizeof(qkm_sel), 0, kPmFlagBytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&c->pm_partial, rows * d.n_embd * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void**)&c->pm_back, rows * d.n_embd * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc((void**)&c->pm_xscale, (size_t)slot_cap * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(c->pm_back, 0, rows * d.n_embd * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(c->pm_xrecv, 0, rows * d.n_embd * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(c->pm_selrecv, 0xFF, rows * sizeof(qkm_sel));   // every record empty
    if (e == cudaSuccess) e = cudaMemset(c->pm_partial, 0, rows * d.n_embd * sizeof(float));
    if (e != cudaSuccess) {
        for (void** p : {(void**)&c->pm_xrecv, (void**)&c->pm_selrecv, (void**)&c->pm_partial, (void**)&c->pm_back, (void**)&c->pm_xscale}) {
            if (*p) cudaFree(*p);
            *p = nullptr;
        }
        return fail(c, QKM_ERR_CUDA, "qkm_ep_peer_setup: %s", cudaGetErrorString(e));
    }
    c->pm_ranks = n_ranks; c->pm_rank = rank; c->pm_cap = slot_cap; c->pm_epoch = 0;
    c->pm_peers.x[rank] = c->pm_xrecv; c->pm_peers.sel[rank] = c->pm_selrecv; c->pm_peers.back[rank] = c->pm_back;
    c->pm_peers.flags[rank] = pm_flags_of(c, c->pm_selrecv);
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_peer_buffers(qkm_ctx* c, void** xrecv, void** selrecv, void** back) {
    if (!c || !xrecv || !selrecv || !back) return QKM_ERR_ARG;
    if (!c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup has not been called");
    *xrecv = c->pm_xrecv; *selrecv = c->pm_selrecv; *back = c->pm_back;
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_peer_set(qkm_ctx* c, uint32_t peer, void* xrecv, void* selrecv, void* back) {
    if (!c || !xrecv || !selrecv || !back) return QKM_ERR_ARG;
    if (!c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup has not been called");
    if (peer >= c->pm_ranks || peer == c->pm_rank) return fail(c, QKM_ERR_ARG, "peer %u is not another rank of %u", peer, c->pm_ranks);
    c->pm_peers.x[peer] = (float*)xrecv; c->pm_peers.sel[peer] = (qkm_sel*)selrecv; c->pm_peers.back[peer] = (float*)back;
    c->pm_peers.flags[peer] = pm_flags_of(c, selrecv);   // every rank uses the same slot_cap, hence the same offset
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_peer_export(qkm_ctx* c, void* handles) {
    if (!c || !handles) return QKM_ERR_ARG;
    if (!c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup has not been called");
    static_assert(sizeof(cudaIpcMemHandle_t) == QKM_EP_HANDLE_BYTES / 3, "handle size");
    cudaIpcMemHandle_t h[3];
    QKM_CUDA(c, cudaIpcGetMemHandle(&h[0], c->pm_xrecv));
    QKM_CUDA(c, cudaIpcGetMemHandle(&h[1], c->pm_selrecv));
    QKM_CUDA(c, cudaIpcGetMemHandle(&h[2], c->pm_back));
    memcpy(handles, h, sizeof h);
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_peer_import(qkm_ctx* c, uint32_t peer, const void* handles) {
    if (!c || !handles) return QKM_ERR_ARG;
    if (!c->pm_ranks) return fail(c, QKM_ERR_MODE, "qkm_ep_peer_setup has not been called");
    if (peer >= c->pm_ranks || peer == c->pm_rank) return fail(c, QKM_ERR_ARG, "peer %u is not another rank of %u", peer, c->pm_ranks);
    if (c->pm_opened[peer][0]) return fail(c, QKM_ERR_MODE, "buffers of rank %u are already mapped", peer);
    cudaIpcMemHandle_t h[3];
    memcpy(h, handles, sizeof h);
    QKM_CUDA(c, cudaSetDevice(c->device));   // the mappings belong to this context's device
    void* p[3] = {};
    for (int i = 0; i < 3; ++i) {
        const cudaError_t e = cudaIpcOpenMemHandle(&p[i], h[i], cudaIpcMemLazyEnablePeerAccess);
        if (e != cudaSuccess) {
            for (int j = 0; j < i; ++j) cudaIpcCloseMemHandle(p[j]);
            cudaGetLastError();
            return fail(c, QKM_ERR_CUDA, "mapping buffer %d of rank %u failed: %s", i, peer, cudaGetErrorString(e));
        }
    }
    for (int i = 0; i < 3; ++i) c->pm_opened[peer][i] = p[i];
    return qkm_ep_peer_set(c, peer, p[0], p[1], p[2]);
}

extern "C" QKM_API int qkm_ep_push(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, uint32_t slot_rows) {
    if (int rc = layer_ready(c, layer)) return rc;
    if (int rc = pm_check(c, slot_rows)) return rc;
    if (!x && n) return QKM_ERR_ARG;
    if (n > slot_rows) return fail(c, QKM_ERR_BOUNDS, "%u tokens exceed slot_rows %u", n, slot_rows);
    if (n) if (int rc = ep_route_local(c, layer, x, n)) return rc;
    // Layers whose resident experts run on the tensor cores consume the rows as scaled f16: then those
    // travel (half the bytes; every rank decides the same from the layer's types).  The router above
    // has made them already for more than 64 tokens.
    const qkm_layer_dev& ld = c->layers[layer];
    c->pm_rows_f16 = ld.tiles_ok && c->cfg.dims.n_embd % 8 == 0;
    if (c->pm_rows_f16 && n) {
        const float* inv = c->xscale;
        if (n <= 64) {   // (the router made digit planes, whose scales sit in xscale for the streamed shared expert)
            if (int rc = ensure_prefill_scratch(c)) return rc;
            QKM_LAUNCH(c, launch_f16_rows(c->L(), x, c->xb, c->pm_xscale, nullptr, n, c->cfg.dims.n_embd));
            inv = c->pm_xscale;
        }
        QKM_LAUNCH(c, launch_ep_push(c->L(), c->cfg.dims, x, c->sel, c->pm_peers, n, slot_rows, c->pm_rank, c->pm_ranks, c->xb, inv));
    } else {
        QKM_LAUNCH(c, launch_ep_push(c->L(), c->cfg.dims, x, c->sel, c->pm_peers, n, slot_rows, c->pm_rank, c->pm_ranks));
    }
    return QKM_OK;
}

extern "C" QKM_API int qkm_ep_forward_slots(qkm_ctx* c, uint32_t layer, uint32_t slot_rows, uint32_t n_shared) {
    if (int rc = pm_check(c, slot_rows)) return rc;
    if (n_shared != QKM_EP_NO_SHARED && n_shared > slot_rows) return fail(c, QKM_ERR_BOUNDS, "%u shared rows exceed slot_rows %u", n_shared, slot_rows);
    const bool with_shared = n_shared != QKM_EP_NO_SHARED;
    c->pm_shared_in_partial = with_shared;
    return ep_expert_forward_impl(c, layer, c->pm_xrecv, c->pm_selrecv, c->pm_ranks * slot_rows, c->pm_partial, with_shared,
                                  c->pm_rank * slot_rows, with_shared ? n_shared : 0, slot_rows,
                                  c->pm_rows_f16 && c->layers[layer].tiles_ok);
}

extern "C" QKM_API int qkm_ep_pull(qkm_ctx* c, uint32_t n, uint32_t slot_rows, float* y) {
    if (int rc = pm_check(c, slot_rows)) return rc;
    if (!y && n) return QKM_ERR_ARG;
    if (n > slot_rows) return fail(c, QKM_ERR_BOUNDS, "%u tokens exceed slot_rows %u", n, slot_rows);
    const bool own = c->pm_shared_in_partial;   // the shared expert came with this rank's partial rows
    QKM_LAUNCH(c, launch_ep_pull(c->L(), c->cfg.dims, c->sel, c->pm_peers, own ? nullptr : c->y2, y, n, slot_rows, c->pm_rank, c->pm_ranks, own));
    return QKM_OK;
}

// Barrier of the ranks as a kernel on the context's stream (ep_barrier_kernel): every rank must
// issue the same sequence of barriers, each rank on its own GPU.  timeout_ms bounds the wait on
// the device; a wait that ran out shows as QKM_ERR_TIMEOUT at the next qkm_sync.
extern "C" QKM_API int qkm_ep_barrier(qkm_ctx* c, uint32_t timeout_ms) {
    if (int rc = pm_check(c, 1)) return rc;
    if (timeout_ms == 0) return fail(c, QKM_ERR_ARG, "the barrier needs a time limit");
    QKM_LAUNCH(c, launch_ep_barrier(c->L(), c->pm_peers, c->pm_rank, c->pm_ranks, ++c->pm_epoch, (uint64_t)timeout_ms * 1000000ull, c->status));
    return QKM_OK;
}

// The whole layer in one call: push, barrier, resident + shared experts, barrier, pull.
extern "C" QKM_API int qkm_ep_peer_layer(qkm_ctx* c, uint32_t layer, const float* x, uint32_t n, uint32_t slot_rows, float* y,
                                         uint32_t timeout_ms) {
    if (int rc = qkm_ep_push(c, layer, x, n, slot_rows)) return rc;
    if (int rc = qkm_ep_barrier(c, timeout_ms)) return rc;
    if (int rc = qkm_ep_forward_slots(c, layer, slot_rows, n)) return rc;   // the shared expert rides with the resident ones
    if (int rc = qkm_ep_barrier(c, timeout_ms)) return rc;
    return qkm_ep_pull(c, n, slot_rows, y);
}
