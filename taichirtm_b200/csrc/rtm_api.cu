// Host side of librtm_b200: plans, time loops and the extern "C" entry
// points declared in include/rtm_b200.h.
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/rtm_b200.h"
#include "adjoint_kernels.cuh"
#include "checkpoint_kernels.cuh"
#include "aux_kernels.cuh"
#include "step2_kernels.cuh"
#include "adjoint2_kernels.cuh"
#include "plan_host.h"
#include "resident_kernels.cuh"
#include "step_kernels.cuh"

using namespace rtm;

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define CUDA_TRY(expr)                                                                  \
    do {                                                                                \
        cudaError_t e_ = (expr);                                                        \
        if (e_ != cudaSuccess)                                                          \
            return fail(e_ == cudaErrorMemoryAllocation ? RTM_E_NOMEM : RTM_E_CUDA,     \
                        "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, \
                        __LINE__);                                                      \
    } while (0)

template <typename T>
int dalloc(T **p, size_t n) {
    *p = nullptr;
    if (n == 0) return 0;
    CUDA_TRY(cudaMalloc((void **)p, n * sizeof(T)));
    return 0;
}

// Device buffers that live and die together, in one allocation.  A plan has about
// 45 of them; one by one, making and destroying one took 6.9 and 5.3 ms (395 x 395,
// both wave types), most of a short one-shot run; together 0.9 and 0.6.
struct Slab {
    std::vector<std::pair<void **, size_t>> want;
    void *base = nullptr;
    template <typename T>
    void add(T **p, size_t n) {
        *p = nullptr;
        if (n) want.push_back({reinterpret_cast<void **>(p), n * sizeof(T)});
    }
    int commit() {
#ifdef RTM_BOUNDS_CHECK
        constexpr size_t GAP = 4096;  // an access past a buffer's end must not land in the next one
#else
        constexpr size_t GAP = 0;
#endif
        size_t total = 0;
        for (auto &w : want) total += (w.second + GAP + 511) / 512 * 512;
        if (!total) return 0;
        CUDA_TRY(cudaMalloc(&base, total));
        char *at = static_cast<char *>(base);
        for (auto &w : want) {
            *w.first = at;
            at += (w.second + GAP + 511) / 512 * 512;
        }
        want.clear();
        return 0;
    }
    void release() {
        if (base) cudaFree(base);
        base = nullptr;
        want.clear();
    }
};

// NVTX range around an entry point: the phases show up by name in Nsight
// Systems; without a profiler attached it costs a call that returns.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
};

}  // namespace

struct rtm_plan {
    rtm_grid g{};
    Slab slab;               // every buffer of the plan but the scratch
    int nshots = 0;
    int vec = 4, rows = 32, warps = 4, prefetch = 1;
    int tsteps = 1;  // time steps per launch of the propagation loops (1 or 2)
    int pitch = 0;
    int nstrips = 0;
    std::vector<ShotDev> shots_h;
    ShotDev *d_shots = nullptr;
    int4 *d_work = nullptr;
    int n_work = 0;
    int *d_src_ptr = nullptr, *d_rec_ptr = nullptr;
    int2 *d_src_ent = nullptr, *d_rec_ent = nullptr;
    int nsrc_total = 0, nrec_total = 0;
    size_t n_src_ptr = 0, n_rec_ptr = 0, n_src_ent = 0, n_rec_ent = 0;  // table lengths
    long long rows_total = 0;  // sum of nx over shots
    size_t state_floats = 0;   // per field, per buffer
    float *d_state[2][NFIELD] = {};
    float *d_mat[NMAT] = {};
    float *d_surface = nullptr;
    bool has_surface = false;
    float *d_sponge = nullptr;
    float *d_img[3] = {}, *d_imgc[3] = {};
    float *d_seis_t = nullptr, *d_obs_t = nullptr;
    int *d_flags = nullptr;
    int *d_fail_seq = nullptr;  // per shot: first failing launch of the current loop
    // Scratch of the checkpointed entry points (rtm_adjoint,
    // rtm_backward_checkpointed): kept and reused from call to call, grown
    // when a call needs more, freed with the plan.  A cudaMalloc / cudaFree
    // pair of several GB per call costs a device-wide synchronisation and
    // page mapping on every gradient.
    float *d_scratch = nullptr;
    size_t scratch_floats = 0;
    bool model_set = false;
    long long launches = 0;
    // CUDA-graph replay of time loops (tune.graphs): one cached executable per
    // loop kind, keyed by every pointer and schedule value it bakes in.
    struct GraphCache {
        std::vector<unsigned long long> key;
        cudaGraphExec_t exec = nullptr;
    };
    bool use_graphs = false;
    cudaStream_t gstream = nullptr;
    cudaEvent_t ev_in = nullptr, ev_out = nullptr;
    GraphCache g_fwd, g_bwd, g_ckpt;
    // Host step callback (rtm_plan_set_callback) and the ping-pong buffer that
    // holds the latest state of rtm_forward / rtm_backward (-1: none).
    rtm_step_callback cb = nullptr;
    void *cb_user = nullptr;
    int cb_every = 0;
    int live = -1;
    // fail_seq counts launches: a stopped shot's latest state is in the buffer
    // that the launch of that number wrote, not in `live`
    bool live_seq = false;
    // Resident propagation (resident_kernels.cuh): the tile layout chosen at
    // plan creation, or r == 0 when the plan streams its wavefield.
    struct Resident {
        int layout = -1;        // index into RES_LAYOUTS, -1: streaming
        bool surface = false;   // laid out with room for a topography mask
        int max_src = 0, max_rec_all = 0, max_rec = 0;  // point entries per tile: sources, receivers, owned receivers
        int4 *d_tiles = nullptr, *d_shot_tiles = nullptr;
        unsigned long long *d_sync = nullptr;  // per shot: ResParams::arrive
        uint4 *d_box = nullptr;  // outboxes of the largest launch
        size_t box_bytes = 0;
        int box_stride = 0;
        unsigned tag = 0;        // tags used by the current call
        bool image_fits = false; // every launch fits with its images in shared memory
        std::vector<int2> waves;  // (first tile, tiles) of each launch
        void *base = nullptr;     // their allocation
    } res;
    // The layouts made so far, without and with a mask, kept until the plan is
    // destroyed: a call that a caller captured goes on using its layout's buffers.
    Resident laid[2];
    bool is_laid[2] = {false, false};
    bool auto_shape = false;  // the launch shape is the library's choice
    int wait_limit = RES_SPIN_LIMIT;  // rtm_plan_set_wait_limit (bounds-checking build)
    std::vector<int> src_ptr_h, rec_ptr_h;  // host copies of the row tables
    std::vector<int2> src_ent_h, rec_ent_h;
};

namespace {

bool field_active(int modes, int f) {
    if (f == F_U || f == F_W || f == F_SXX || f == F_SZZ || f == F_SXZ) return modes & RTM_PSV;
    return modes & RTM_SH;
}
bool comp_active(int modes, int c) { return c == 1 ? (modes & RTM_SH) : (modes & RTM_PSV); }

// The plan's scratch, at least n floats (contents undefined).
int plan_scratch(rtm_plan *p, size_t n, float **out) {
    if (p->scratch_floats < n) {
        if (p->d_scratch) cudaFree(p->d_scratch);
        p->d_scratch = nullptr;
        p->scratch_floats = 0;
        if (int rc = dalloc(&p->d_scratch, n)) return rc;
        p->scratch_floats = n;
    }
    *out = p->d_scratch;
    return 0;
}

void plan_free(rtm_plan *p) {
    p->slab.release();
    for (auto &r : p->laid)
        if (r.base) cudaFree(r.base);
    if (p->d_scratch) cudaFree(p->d_scratch);
    for (auto *gc : {&p->g_fwd, &p->g_bwd, &p->g_ckpt})
        if (gc->exec) cudaGraphExecDestroy(gc->exec);
    if (p->ev_in) cudaEventDestroy(p->ev_in);
    if (p->ev_out) cudaEventDestroy(p->ev_out);
    if (p->gstream) cudaStreamDestroy(p->gstream);
}

// Buffers one call may touch, for the bounds-checking build (debug_bounds.cuh):
// the plan's allocations and the caller's buffers, with their sizes.  In the
// normal build every method is empty.
struct BoundsScope {
#ifdef RTM_BOUNDS_CHECK
    std::vector<std::pair<unsigned long long, unsigned long long>> r;
    void add(const void *ptr, size_t bytes) {
        if (ptr && bytes) r.push_back({(unsigned long long)(uintptr_t)ptr, (unsigned long long)(uintptr_t)ptr + bytes});
    }
    int begin(cudaStream_t s) {
        DbgTable t{};
        if (r.size() > (size_t)DBG_MAX_RANGES) return fail(RTM_E_STATE, "bounds check: %zu buffers > %d", r.size(), DBG_MAX_RANGES);
        for (size_t k = 0; k < r.size(); ++k) {
            t.begin[k] = r[k].first;
            t.end[k] = r[k].second;
        }
        t.n = (int)r.size();
        const unsigned long long zero = 0;
        CUDA_TRY(cudaMemcpyToSymbolAsync(g_dbg_table, &t, sizeof t, 0, cudaMemcpyHostToDevice, s));
        CUDA_TRY(cudaMemcpyToSymbolAsync(g_dbg_bad, &zero, sizeof zero, 0, cudaMemcpyHostToDevice, s));
        CUDA_TRY(cudaStreamSynchronize(s));  // the table is a stack object's copy: upload before returning
        return 0;
    }
    int end(cudaStream_t s) {
        unsigned long long bad = 0, first = 0;
        CUDA_TRY(cudaMemcpyFromSymbolAsync(&bad, g_dbg_bad, sizeof bad, 0, cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaMemcpyFromSymbolAsync(&first, g_dbg_first, sizeof first, 0, cudaMemcpyDeviceToHost, s));
        CUDA_TRY(cudaStreamSynchronize(s));
        DbgTable none{};
        CUDA_TRY(cudaMemcpyToSymbol(g_dbg_table, &none, sizeof none));  // later calls of other entry points: unchecked until set
        if (bad) return fail(RTM_E_CUDA, "bounds check: %llu accesses outside every buffer (first at 0x%llx)", bad, first);
        return 0;
    }
#else
    void add(const void *, size_t) {}
    int begin(cudaStream_t) { return 0; }
    int end(cudaStream_t) { return 0; }
#endif
    void add_plan(const rtm_plan *p) {
        const size_t F = sizeof(float);
        add(p->d_shots, p->shots_h.size() * sizeof(ShotDev));
        add(p->d_work, (size_t)p->n_work * sizeof(int4));
        add(p->d_src_ptr, p->n_src_ptr * sizeof(int));
        add(p->d_rec_ptr, p->n_rec_ptr * sizeof(int));
        add(p->d_src_ent, p->n_src_ent * sizeof(int2));
        add(p->d_rec_ent, p->n_rec_ent * sizeof(int2));
        add(p->d_flags, (p->nshots + 2) * sizeof(int));
        add(p->d_fail_seq, p->nshots * sizeof(int));
        add(p->res.d_box, p->res.box_bytes);
        add(p->d_sponge, (size_t)std::max(p->g.absorbing_frame, 1) * F);
        for (int b = 0; b < 2; ++b)
            for (int f = 0; f < NFIELD; ++f) add(p->d_state[b][f], p->state_floats * F);
        const size_t mat = (size_t)(p->g.nx + 2) * p->pitch * F;
        for (int m = 0; m < NMAT; ++m) add(p->d_mat[m], mat);
        add(p->d_surface, mat);
        for (int c = 0; c < 3; ++c) {
            add(p->d_img[c], (size_t)p->rows_total * p->pitch * F);
            add(p->d_imgc[c], (size_t)p->rows_total * p->pitch * F);
        }
        const size_t seis = std::max<size_t>((size_t)3 * p->g.nt * p->nrec_total, 1) * F;
        add(p->d_seis_t, seis);
        add(p->d_obs_t, seis);
    }
};

// Run a time loop: directly on s, or (use_graphs) as a CUDA graph captured on
// the plan's own stream the first time this key is seen and replayed after.
// The caller's stream and the plan stream are ordered by two events.
template <typename Body>
int run_loop(rtm_plan *p, rtm_plan::GraphCache &gc, const std::vector<unsigned long long> &key,
             cudaStream_t s, Body &&body) {
    if (!p->use_graphs) return body(s);
    if (!p->gstream) {
        CUDA_TRY(cudaStreamCreateWithFlags(&p->gstream, cudaStreamNonBlocking));
        CUDA_TRY(cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming));
        CUDA_TRY(cudaEventCreateWithFlags(&p->ev_out, cudaEventDisableTiming));
    }
    if (!gc.exec || gc.key != key) {
        if (gc.exec) {
            cudaGraphExecDestroy(gc.exec);
            gc.exec = nullptr;
        }
        CUDA_TRY(cudaStreamBeginCapture(p->gstream, cudaStreamCaptureModeThreadLocal));
        const int rc = body(p->gstream);
        cudaGraph_t graph = nullptr;
        const cudaError_t e = cudaStreamEndCapture(p->gstream, &graph);
        if (rc || e != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return rc ? rc : fail(RTM_E_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
        }
        const cudaError_t e2 = cudaGraphInstantiate(&gc.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e2 != cudaSuccess) {
            gc.exec = nullptr;
            return fail(RTM_E_CUDA, "graph instantiate failed: %s", cudaGetErrorString(e2));
        }
        gc.key = key;
    }
    CUDA_TRY(cudaEventRecord(p->ev_in, s));
    CUDA_TRY(cudaStreamWaitEvent(p->gstream, p->ev_in, 0));
    CUDA_TRY(cudaGraphLaunch(gc.exec, p->gstream));
    CUDA_TRY(cudaEventRecord(p->ev_out, p->gstream));
    CUDA_TRY(cudaStreamWaitEvent(s, p->ev_out, 0));
    return 0;
}

unsigned long long U(const void *ptr) { return (unsigned long long)(uintptr_t)ptr; }

constexpr size_t kMaxSmem = 227 * 1024;  // dynamic shared memory of a CTA, opt-in limit

template <int DIR, int MODE, int VEC, int PFM>
cudaError_t launch_step(const StepParams &sp, int warps, cudaStream_t s) {
    const int threads = 32 * warps;
    const int blocks = (sp.n_work + warps - 1) / warps;
    size_t smem = 0;
    if constexpr (PFM == 3) {
        smem = (size_t)warps * async_smem_per_warp<MODE, VEC>();
        if (smem > kMaxSmem) return cudaErrorInvalidConfiguration;
        static bool attr_set = false;  // per instantiation; raises the 48 KB default
        if (!attr_set) {
            const size_t want = std::min<size_t>(8 * async_smem_per_warp<MODE, VEC>(), kMaxSmem);
            cudaError_t e = cudaFuncSetAttribute(step_kernel<DIR, MODE, VEC, PFM>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
            if (e != cudaSuccess) return e;
            attr_set = true;
        }
    }
    step_kernel<DIR, MODE, VEC, PFM><<<blocks, threads, smem, s>>>(sp);
    return cudaGetLastError();
}

template <int DIR, int MODE, int VEC>
cudaError_t launch_pf(const StepParams &sp, int pfm, int warps, cudaStream_t s) {
    switch (pfm) {
        case 0: return launch_step<DIR, MODE, VEC, 0>(sp, warps, s);
        case 1: return launch_step<DIR, MODE, VEC, 1>(sp, warps, s);
        case 2: return launch_step<DIR, MODE, VEC, 2>(sp, warps, s);
        default: return launch_step<DIR, MODE, VEC, 3>(sp, warps, s);
    }
}

// vec: columns per lane in bits 0-7, prefetch mode (0/1/2) in bits 8-9
template <int DIR, int MODE>
cudaError_t launch_vec(const StepParams &sp, int vec, int warps, cudaStream_t s) {
    const int pfm = (vec >> 8) & 3;
    switch (vec & 0xff) {
        case 1: return launch_pf<DIR, MODE, 1>(sp, pfm, warps, s);
        case 2: return launch_pf<DIR, MODE, 2>(sp, pfm, warps, s);
        default: return launch_pf<DIR, MODE, 4>(sp, pfm, warps, s);
    }
}

template <int DIR>
cudaError_t launch_mode(const StepParams &sp, int modes, int vec, int warps, cudaStream_t s) {
    switch (modes) {
        case RTM_PSV: return launch_vec<DIR, RTM_PSV>(sp, vec, warps, s);
        case RTM_SH: return launch_vec<DIR, RTM_SH>(sp, vec, warps, s);
        default: return launch_vec<DIR, RTM_BOTH>(sp, vec, warps, s);
    }
}

// May this kernel have as much shared memory as a CTA can?  Once per instantiation.
template <int DIR, int MODE, int VEC, bool STOREA, bool CKPT, bool UNI, bool SR>
cudaError_t ring2_allow_smem() {
    static std::atomic<bool> done{false};
    if (done) return cudaSuccess;
    const size_t want = std::min<size_t>(8 * ring2_smem_per_warp<SR, MODE, VEC>(true), kMaxSmem);
    const cudaError_t e = cudaFuncSetAttribute(step2_kernel<DIR, MODE, VEC, true, STOREA, CKPT, UNI, SR>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
    done = e == cudaSuccess;
    return e;
}

// Enough tasks to be bound by what a task costs rather than by its chain of rows?
bool many_tasks(const StepParams &sp) {
    static std::atomic<int> least{0};
    int n = least.load();
    if (n == 0) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
        least = n = 12 * sms;
    }
    return sp.n_work >= n;
}

// Warps of this kernel that an SM holds, 0 where a CTA's rings do not fit.
template <int MODE, int VEC, bool STOREA, bool CKPT, bool UNI, bool SR>
int ring2_warps_per_sm(int warps, bool surface) {
    const size_t smem = (size_t)warps * ring2_smem_per_warp<SR, MODE, VEC>(surface);
    int ctas = 0;
    if (smem > kMaxSmem || ring2_allow_smem<0, MODE, VEC, STOREA, CKPT, UNI, SR>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, step2_kernel<0, MODE, VEC, true, STOREA, CKPT, UNI, SR>, 32 * warps, smem) != cudaSuccess)
        return 0;
    return ctas * warps;
}

// Does a forward ring launch bring the state through a ring too?  Its time against
// rolling registers, 12 shots of 801 x 801 (2,184 to 8,568 tasks): vec 4, P-SV 0.93
// to 1.04 and both wave types 0.95 to 1.0 where the SM keeps at least 7/8 of its
// warps; 1.10 to 1.18 (P-SV, 4 warps, mask: 8 of 12) and 1.47 (both, 4 of 8) where
// it does not.  With vec 2 a row is short for its copies: P-SV 0.89 to 1.0, with a
// mask 1.08 to 1.20, both wave types 1.20 to 1.25.  Launches of up to 800 tasks, a
// wave or two, are bound by the chain of rows: 1.0 to 1.15.
template <int MODE, int VEC, bool STOREA, bool CKPT, bool UNI>
bool ring2_state_ring(const StepParams &sp, int warps) {
    const bool surface = sp.surface != nullptr;
    if (VEC == 2 && MODE == RTM_PSV && surface) return false;
    if (!many_tasks(sp)) return false;
    static std::atomic<int> keeps[9][2];  // per CTA size and mask: 1 yes, -1 no, 0 not asked yet
    int k = keeps[warps][surface].load();
    if (k == 0) {
        const int with = ring2_warps_per_sm<MODE, VEC, STOREA, CKPT, UNI, true>(warps, surface);
        const int without = ring2_warps_per_sm<MODE, VEC, STOREA, CKPT, UNI, false>(warps, surface);
        k = 8 * with >= 7 * without && with > 0 ? 1 : -1;
        keeps[warps][surface] = k;
    }
    return k > 0;
}

template <int DIR, int MODE, int VEC, bool RING, bool STOREA, bool CKPT, bool UNI, bool SR>
cudaError_t launch_step2_as(const StepParams &sp, int warps, cudaStream_t s) {
    size_t smem = 0;
    if constexpr (RING) {
        smem = (size_t)warps * ring2_smem_per_warp<SR, MODE, VEC>(sp.surface != nullptr);
        if (smem > kMaxSmem) return cudaErrorInvalidConfiguration;
        if (const cudaError_t e = ring2_allow_smem<DIR, MODE, VEC, STOREA, CKPT, UNI, SR>()) return e;
    }
    const int blocks = (sp.n_work + warps - 1) / warps;
    // Many tasks hide the longer chain of packed operations: P-SV, 8,568 tasks 1.01,
    // 800 tasks 0.98 of packed with scalar ones (a gradient of 8 shots of 1201 x 401
    // 79.3 against 78.5 ms)
    if constexpr (MODE == RTM_PSV && VEC == 2 && !RING) {
        if (many_tasks(sp)) {
            step2_kernel<DIR, MODE, VEC, RING, STOREA, CKPT, UNI, SR, 8, true><<<blocks, 32 * warps, smem, s>>>(sp);
            return cudaGetLastError();
        }
    }
    if constexpr (MODE == RTM_SH && VEC == 2 && !RING) {  // 12 shots of 801 x 801, 4 warps: 51.5 -> 44.8 us per step
        if (warps <= 4) {
            step2_kernel<DIR, MODE, VEC, RING, STOREA, CKPT, UNI, SR, 4><<<blocks, 32 * warps, smem, s>>>(sp);
            return cudaGetLastError();
        }
    }
    step2_kernel<DIR, MODE, VEC, RING, STOREA, CKPT, UNI, SR><<<blocks, 32 * warps, smem, s>>>(sp);
    return cudaGetLastError();
}

template <int DIR, int MODE, int VEC, bool RING, bool STOREA = false, bool CKPT = false, bool UNI = false>
cudaError_t launch_step2(const StepParams &sp, int warps, cudaStream_t s) {
    if constexpr (RING && DIR == 0 && !(VEC == 2 && MODE == RTM_BOTH)) {
        if (ring2_state_ring<MODE, VEC, STOREA, CKPT, UNI>(sp, warps))
            return launch_step2_as<DIR, MODE, VEC, RING, STOREA, CKPT, UNI, true>(sp, warps, s);
    }
    return launch_step2_as<DIR, MODE, VEC, RING, STOREA, CKPT, UNI, false>(sp, warps, s);
}

// Checkpoint-storing forward P-SV launches (sp.ck set): one step or two
// steps, the output state also packed into the compressed slot.
template <int VEC, int PFM>
cudaError_t launch_step_ckpt(const StepParams &sp, int warps, cudaStream_t s) {
    const int threads = 32 * warps;
    const int blocks = (sp.n_work + warps - 1) / warps;
    size_t smem = 0;
    if constexpr (PFM == 3) {
        smem = (size_t)warps * async_smem_per_warp<RTM_PSV, VEC>();
        if (smem > kMaxSmem) return cudaErrorInvalidConfiguration;
        static bool attr_set = false;
        if (!attr_set) {
            const size_t want = std::min<size_t>(8 * async_smem_per_warp<RTM_PSV, VEC>(), kMaxSmem);
            cudaError_t e = cudaFuncSetAttribute(step_kernel<0, RTM_PSV, VEC, PFM, true>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
            if (e != cudaSuccess) return e;
            attr_set = true;
        }
    }
    step_kernel<0, RTM_PSV, VEC, PFM, true><<<blocks, threads, smem, s>>>(sp);
    return cudaGetLastError();
}
template <int VEC>
cudaError_t launch_pf_ckpt(const StepParams &sp, int pfm, int warps, cudaStream_t s) {
    switch (pfm) {
        case 0: return launch_step_ckpt<VEC, 0>(sp, warps, s);
        case 1: return launch_step_ckpt<VEC, 1>(sp, warps, s);
        case 2: return launch_step_ckpt<VEC, 2>(sp, warps, s);
        default: return launch_step_ckpt<VEC, 3>(sp, warps, s);
    }
}
cudaError_t launch_ckpt(const StepParams &sp, bool two, int vec, int prefetch, int warps, cudaStream_t s) {
    if (two) {
        const bool ring = prefetch >= 3;
        if (vec == 2)
            return ring ? launch_step2<0, RTM_PSV, 2, true, false, true>(sp, warps, s)
                        : launch_step2<0, RTM_PSV, 2, false, false, true>(sp, warps, s);
        return ring ? launch_step2<0, RTM_PSV, 4, true, false, true>(sp, warps, s)
                    : launch_step2<0, RTM_PSV, 4, false, false, true>(sp, warps, s);
    }
    switch (vec) {
        case 1: return launch_pf_ckpt<1>(sp, prefetch, warps, s);
        case 2: return launch_pf_ckpt<2>(sp, prefetch, warps, s);
        default: return launch_pf_ckpt<4>(sp, prefetch, warps, s);
    }
}

// uni (prefetch 4): the ring kernel with the task taken from blockIdx.x,
// one warp per CTA (the plan forces warps = 1).
template <int DIR, int MODE>
cudaError_t launch_vec2(const StepParams &sp, int vec, bool ring, bool uni, int warps, cudaStream_t s) {
    if (uni) {
        if (warps != 1) return cudaErrorInvalidConfiguration;
        return vec == 2 ? launch_step2<DIR, MODE, 2, true, false, false, true>(sp, 1, s)
                        : launch_step2<DIR, MODE, 4, true, false, false, true>(sp, 1, s);
    }
    if (vec == 2) return ring ? launch_step2<DIR, MODE, 2, true>(sp, warps, s) : launch_step2<DIR, MODE, 2, false>(sp, warps, s);
    // both wave types, vec 4: rolling registers spill (12 shots of 801 x 801, 4 warps:
    // 117 us per step, 85 through the ring), so the ring kernel runs them all
    if constexpr (MODE == RTM_BOTH) return launch_step2<DIR, MODE, 4, true>(sp, warps, s);
    else return ring ? launch_step2<DIR, MODE, 4, true>(sp, warps, s) : launch_step2<DIR, MODE, 4, false>(sp, warps, s);
}

// Forward recompute of the adjoint, P-SV: steps sp.it and sp.it2 in one
// launch, storing the state after each (sp.souta, sp.sout).
cudaError_t launch_recompute2(const StepParams &sp, int vec, int prefetch, int warps, cudaStream_t s) {
    const bool ring = prefetch >= 3;
    if (vec == 2)
        return ring ? launch_step2<0, RTM_PSV, 2, true, true>(sp, warps, s) : launch_step2<0, RTM_PSV, 2, false, true>(sp, warps, s);
    return ring ? launch_step2<0, RTM_PSV, 4, true, true>(sp, warps, s) : launch_step2<0, RTM_PSV, 4, false, true>(sp, warps, s);
}

// Two steps (sp.it, sp.it2) in one launch; vec is 2 or 4 (checked at plan
// creation); prefetch 3 selects the shared-memory material ring.
template <int DIR>
cudaError_t launch_mode2(const StepParams &sp, int modes, int vec, int prefetch, int warps, cudaStream_t s) {
    const bool ring = prefetch >= 3, uni = prefetch == 4;
    switch (modes) {
        case RTM_PSV: return launch_vec2<DIR, RTM_PSV>(sp, vec, ring, uni, warps, s);
        case RTM_SH: return launch_vec2<DIR, RTM_SH>(sp, vec, ring, uni, warps, s);
        default: return launch_vec2<DIR, RTM_BOTH>(sp, vec, ring, uni, warps, s);
    }
}

// The launches of a time loop over loop steps 0 .. nt-1: step `it` alone, or
// steps it and it+1 together when the plan runs two steps per launch and
// step `it` may be the first of a pair (pairable(it): it is not checked and
// its state need not be stored).
struct LoopLaunch {
    int it;
    bool two;
};
template <typename Pairable>
std::vector<LoopLaunch> loop_schedule(int first, int end, int tsteps, Pairable &&pairable) {
    std::vector<LoopLaunch> out;
    for (int it = first; it < end;) {
        const bool two = tsteps == 2 && it + 1 < end && pairable(it);
        out.push_back({it, two});
        it += two ? 2 : 1;
    }
    return out;
}

// The host callback after launch number `seq` (1-based) at step `step`:
// waits for the stream, skips the call once every shot stopped in an earlier
// launch (a failed check ends the reference's loop before its next
// callback), and turns a non-zero return into RTM_E_CALLBACK.
int call_back(rtm_plan *p, int seq, int step, cudaStream_t s) {
    CUDA_TRY(cudaStreamSynchronize(s));
    std::vector<int> fs(p->nshots);
    CUDA_TRY(cudaMemcpy(fs.data(), p->d_fail_seq, p->nshots * sizeof(int), cudaMemcpyDeviceToHost));
    bool alive = false;
    for (int v : fs) alive = alive || v >= seq;
    if (!alive) return 0;
    if (int rc = p->cb(p->cb_user, step))
        return fail(RTM_E_CALLBACK, "the step callback returned %d at step %d", rc, step);
    return 0;
}

void fill_common(const rtm_plan *p, StepParams &sp) {
    std::memset(&sp, 0, sizeof sp);
    const double dt = 1.0 / p->g.fs;
    sp.nz = p->g.nz;
    sp.pitch = p->pitch;
    sp.nt = p->g.nt;
    sp.fw = p->g.absorbing_frame;
    sp.dt = (float)dt;
    sp.inv_dx = (float)(1.0 / p->g.dx);
    sp.inv_dz = (float)(1.0 / p->g.dz);
    sp.src_factor = (float)(dt * p->g.dx * p->g.dz);  // forward_modeling.py:430
    sp.neg_zero = -0.0f;
    sp.sponge = p->d_sponge;
    sp.work = p->d_work;
    sp.n_work = p->n_work;
    sp.shots = p->d_shots;
    for (int m = 0; m < NMAT; ++m) sp.mat[m] = p->d_mat[m];
    sp.surface = p->has_surface ? p->d_surface : nullptr;
    sp.src_ptr = p->d_src_ptr;
    sp.src_ent = p->d_src_ent;
    sp.rec_ptr = p->d_rec_ptr;
    sp.rec_ent = p->d_rec_ent;
    sp.nrec_total = p->nrec_total;
    sp.flags = p->d_flags;
    sp.fail_seq = p->d_fail_seq;
    sp.snap_k = -1;
}

int zero_status(rtm_plan *p, cudaStream_t s) {
    CUDA_TRY(cudaMemsetAsync(p->d_flags, 0, (p->nshots + 1) * sizeof(int), s));  // not the second error word: read_status
    CUDA_TRY(cudaMemsetAsync(p->d_fail_seq, 0x7f, p->nshots * sizeof(int), s));  // 0x7f7f7f7f: none
    return 0;
}
int zero_state(rtm_plan *p, cudaStream_t s) {
    for (int b = 0; b < 2; ++b)
        for (int f = 0; f < NFIELD; ++f)
            if (p->d_state[b][f])
                CUDA_TRY(cudaMemsetAsync(p->d_state[b][f], 0, p->state_floats * sizeof(float), s));
    return zero_status(p, s);
}

// The per-shot status codes to host memory (synchronises), and the second of the
// resident kernel's error words behind them.  That one stays set until it has been
// reported: calls with null flags return before the GPU is done and cannot.
int read_status(rtm_plan *p, int32_t *flags, cudaStream_t s) {
    const int n = p->nshots;
    std::vector<int> h(n + 2);
    CUDA_TRY(cudaMemcpyAsync(h.data(), p->d_flags, h.size() * sizeof(int), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaStreamSynchronize(s));
    if (flags) std::copy(h.begin(), h.begin() + n, flags);
    if (!h[n + 1]) return 0;
    CUDA_TRY(cudaMemsetAsync(p->d_flags + n + 1, 0, sizeof(int), s));
    return fail(RTM_E_CUDA, "resident propagation: a wait between tiles ran out, in this call or in one since the last reported status");
}

// ---- resident propagation (resident_kernels.cuh)

// Tile layouts (rows per lane of the P-SV and of the SH tiles, warps) and the
// time of one step (us, mean of the two directions, 200 to 600 steps of one
// source and a receiver on every row, measured) with 1, 2, ... CTAs on every SM.
// Few rows per lane finish a step soonest; many keep more cells on the chip and
// recompute a smaller share of halo.  Layouts that another one beats at every
// size are not built (P-SV R 4 x 8 warps: 432 CTAs hold 581,000 cells at 3.7 us,
// R 6 x 8: 288 hold 645,000 at 3.3; R 3 x 16 is 5 % behind R 6 x 8; R 7 and 8
// spill so much that they run at 188 / 163 and 139 Gcell/s against 190).  The ones
// built spill a little, too, at these registers (bytes stored, forward / backward):
// P-SV R 2 x 8 60 / 184 and R 6 x 8 256 / 188, SH 0 to 44, both wave types 76 / 300
// and 260 / 220; P-SV R 2 x 12 0 / 72.
struct ResLayout {
    int mode, rp, rs, warps;
    float us[4];
};
constexpr ResLayout RES_LAYOUTS[] = {
    {RTM_PSV, 2, 0, 8, {1.05f, 1.37f, 1.78f, 2.25f}}, {RTM_PSV, 2, 0, 12, {1.31f, 1.90f}}, {RTM_PSV, 6, 0, 8, {2.15f, 3.30f}},
    {RTM_SH, 0, 2, 8, {0.85f, 1.03f, 1.23f, 1.50f}},  {RTM_SH, 0, 4, 8, {1.20f, 1.55f, 1.85f, 2.35f}}, {RTM_SH, 0, 8, 8, {1.53f, 2.17f}},
    {RTM_BOTH, 2, 2, 8, {1.07f, 1.35f, 1.94f, 2.50f}}, {RTM_BOTH, 6, 8, 8, {2.27f, 3.15f}},
};
// Time of one step of the streaming kernels at their tuned shapes (us): the
// launch (one per two steps), the last wave's tail, and the cells at the full
// rate, strips of 120 columns counted whole.  Fits 0.47 to 28 million cells
// within 10 %.
double streaming_us(int modes, long long rows, int nz) {
    const double cells = (double)rows * nz, padded = (double)rows * ((nz + 119) / 120 * 120);
    const double tail = std::min(1.0, cells / 3e6);
    if (modes == RTM_PSV) return 3.5 + 5.83e-6 * padded + 7.0 * tail;
    if (modes == RTM_SH) return 3.5 + 3.7e-6 * padded + 3.5 * tail;
    return 3.5 + 9.5e-6 * padded + 4.0 * tail;
}

// Calls f(kernel, P-SV layout, SH layout) for a tile layout; false if there is none.
template <int DIR, typename F>
bool res_dispatch(const ResLayout &l, F &&f) {
#define RES_ONE(M, RR, NN)                                                                             \
    if (l.mode == M && (M == RTM_PSV ? l.rp : l.rs) == RR && l.warps == NN) {                           \
        f((const void *)resident_kernel<DIR, M, RR, NN>, ResSmem<M, RR, NN>(), ResSmem<M, RR, NN>());   \
        return true;                                                                                   \
    }
#define RES_TWO(RP, RS, NN)                                                                            \
    if (l.mode == RTM_BOTH && l.rp == RP && l.rs == RS && l.warps == NN) {                              \
        f((const void *)resident_both_kernel<DIR, RP, RS, NN>, ResSmem<1, RP, NN>(), ResSmem<2, RS, NN>()); \
        return true;                                                                                   \
    }
    RES_ONE(RTM_PSV, 2, 8) RES_ONE(RTM_PSV, 2, 12) RES_ONE(RTM_PSV, 6, 8)
    RES_ONE(RTM_SH, 2, 8) RES_ONE(RTM_SH, 4, 8) RES_ONE(RTM_SH, 8, 8)
    RES_TWO(2, 2, 8) RES_TWO(6, 8, 8)
#undef RES_ONE
#undef RES_TWO
    return false;
}

// Shared memory of a CTA and the packets of its two outboxes.
size_t resident_smem(const ResLayout &l, int max_inj, int max_rec, bool surface, int *box = nullptr, size_t *image = nullptr) {
    size_t n = 0;
    res_dispatch<0>(l, [&](const void *, auto a, auto b) {
        if (image) *image = std::max(a.image_bytes(), b.image_bytes());
        n = std::max(a.bytes(surface, max_inj, max_rec), b.bytes(surface, max_inj, max_rec));
        if (box) *box = 2 * std::max(a.BOX, b.BOX);
    });
    return n;
}

// Exchange blocks of the loop it0 .. it1-1, as the kernel cuts it.
int resident_blocks(int it0, int it1, int ci) {
    int n = 0;
    for (int it = it0; it < it1; ++n) {
        int k = std::min(RES_HALO, it1 - it);
        if (ci > 0) k = std::min(k, (ci - it % ci) % ci + 1);
        it += k;
    }
    return n;
}

void resident_params(const rtm_plan *p, ResParams &rp, int dir) {
    std::memset(&rp, 0, sizeof rp);
    StepParams sp;
    fill_common(p, sp);
    auto pair = [](float x) {
        unsigned u;
        std::memcpy(&u, &x, 4);
        return ((unsigned long long)u << 32) | u;
    };
    rp.nz = sp.nz;
    rp.pitch = sp.pitch;
    rp.nt = sp.nt;
    rp.fw = sp.fw;
    rp.src_factor = sp.src_factor;
    rp.idx2 = pair(sp.inv_dx);
    rp.idz2 = pair(sp.inv_dz);
    rp.dt2 = pair(sp.dt);
    rp.sdt2 = pair(dir == 0 ? sp.dt : -sp.dt);
    rp.nz2 = pair(-0.0f);
    rp.sponge = sp.sponge;
    rp.shots = sp.shots;
    for (int m = 0; m < NMAT; ++m) rp.mat[m] = sp.mat[m];
    rp.surface = sp.surface;
    rp.src_ptr = sp.src_ptr;
    rp.src_ent = sp.src_ent;
    rp.rec_ptr = sp.rec_ptr;
    rp.rec_ent = sp.rec_ent;
    rp.nrec_total = sp.nrec_total;
    rp.flags = p->d_flags;
    rp.fail_seq = p->d_fail_seq;
    rp.err = p->d_flags + p->nshots;
#ifdef RTM_BOUNDS_CHECK
    rp.polls0 = RES_SPIN_LIMIT - p->wait_limit;
#endif
    for (int f = 0; f < NFIELD; ++f) rp.store[f] = p->d_state[0][f];
    rp.tiles = p->res.d_tiles;
    rp.shot_tiles = p->res.d_shot_tiles;
    rp.outbox = p->res.d_box;
    rp.box_stride = p->res.box_stride;
    rp.arrive = p->res.d_sync;
    rp.max_inj = dir == 0 ? p->res.max_src : p->res.max_rec_all;
    rp.max_rec = dir == 0 ? p->res.max_rec : 0;
}

// Before the first resident_run of a call: no packet carries tag 0, and the tags
// then go on from run to run.
int resident_begin(rtm_plan *p, cudaStream_t s) {
    CUDA_TRY(cudaMemsetAsync(p->res.d_box, 0, p->res.box_bytes, s));
    p->res.tag = 0;
    return 0;
}

// Run the loop of rp for every shot, wave by wave.
int resident_run(rtm_plan *p, ResParams &rp, int dir, cudaStream_t s) {
    if (rp.check_interval > 0) CUDA_TRY(cudaMemsetAsync(p->res.d_sync, 0, 2 * p->nshots * sizeof(*p->res.d_sync), s));
    const ResLayout &lay = RES_LAYOUTS[p->res.layout];
    size_t image = 0, smem = resident_smem(lay, rp.max_inj, rp.max_rec, p->res.surface, nullptr, &image);
    // images stay on the chip where every launch still fits with them: no read and
    // write of the sums per imaging step (301 x 151 RTM, an image at every step, 500
    // steps: 2.40 -> 1.91 ms)
    rp.img_chip = dir == 1 && rp.isnap > 0 && p->res.image_fits;
    if (rp.img_chip) smem += image;
    const unsigned blocks = (unsigned)resident_blocks(rp.it0, rp.it1, rp.check_interval);
    const void *kernel = nullptr;
    auto take = [&](const void *k, auto, auto) { kernel = k; };
    if (dir == 0) res_dispatch<0>(lay, take);
    else res_dispatch<1>(lay, take);
    for (const int2 &w : p->res.waves) {
        rp.tile0 = w.x;
        rp.tag0 = p->res.tag;
        void *args[] = {&rp};
        CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(w.y), dim3(32 * lay.warps), args, smem, s));
        ++p->launches;
        p->res.tag += blocks;
    }
    return 0;
}

// Choose the layout in which every shot's tiles are resident together and the
// estimated step is shortest, and build its tables.  Leaves p->res.layout at -1
// when there is none, when streaming is estimated to be faster, or when the
// device memory left does not hold its buffers.
int resident_setup(rtm_plan *p, bool surface) {
    if (p->is_laid[surface]) {
        p->res = p->laid[surface];
        return 0;
    }
    const std::vector<int> &src_ptr = p->src_ptr_h, &rec_ptr = p->rec_ptr_h;
    const std::vector<int2> &src_ent = p->src_ent_h, &rec_ent = p->rec_ent_h;
    p->res = rtm_plan::Resident();
    p->res.surface = surface;
    int dev = 0, sms = 0, coop = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return 0;
    constexpr int ow = RES_COLS - 2 * RES_HALO;
    const int ntz = (p->g.nz + ow - 1) / ow;
    rtm_plan::Resident best;
    std::vector<int4> tiles, stiles;
    const double stream_us = streaming_us(p->g.modes, p->rows_total, p->g.nz);
    double best_us = stream_us;
    for (int li = 0; li < (int)(sizeof RES_LAYOUTS / sizeof *RES_LAYOUTS); ++li) {
        const ResLayout &lay = RES_LAYOUTS[li];
        if (lay.mode != p->g.modes) continue;
        // per wave type: rows a tile owns, tiles of every shot; point entries of the fullest tile
        const int oh[2] = {lay.warps * lay.rp - 2 * RES_HALO, lay.warps * lay.rs - 2 * RES_HALO};
        std::vector<int4> st((size_t)2 * p->nshots, make_int4(0, 0, ntz, 0));
        int max_src = 0, max_rec_all = 0, max_rec = 0, most = 0;
        for (int s = 0; s < p->nshots; ++s) {
            const ShotDev &d = p->shots_h[s];
            for (int m = 0; m < 2; ++m) {
                if (oh[m] <= 0) continue;
                const int ntx = (d.nx + oh[m] - 1) / oh[m];
                st[2 * s + m].y = ntx;
                auto count = [&](const std::vector<int> &ptr, const std::vector<int2> &ent, int base, int ring) {
                    std::vector<int> n((size_t)ntx * ntz, 0);
                    for (int i = 0; i < d.nx; ++i)
                        for (int e = ptr[base + i]; e < ptr[base + i + 1]; ++e)
                            for (int a = std::max(0, (i - ring) / oh[m]); a <= std::min(ntx - 1, (i + ring) / oh[m]); ++a)
                                for (int b = std::max(0, (ent[e].x - ring) / ow); b <= std::min(ntz - 1, (ent[e].x + ring) / ow); ++b)
                                    ++n[(size_t)a * ntz + b];
                    return *std::max_element(n.begin(), n.end());
                };
                max_src = std::max(max_src, count(src_ptr, src_ent, d.src_row0, RES_HALO));
                max_rec_all = std::max(max_rec_all, count(rec_ptr, rec_ent, d.rec_row0, RES_HALO));
                max_rec = std::max(max_rec, count(rec_ptr, rec_ent, d.rec_row0, 0));
            }
            const int n = (st[2 * s].y + st[2 * s + 1].y) * ntz;
            st[2 * s].x = st[2 * s + 1].x = n;
            most = std::max(most, n);
        }
        // CTAs per SM: the smaller of the two directions'; and backward with images
        int ctas = 0, ctas_image = 0;
        cudaError_t e = cudaSuccess;
        for (int pass = 0; pass < 3; ++pass) {
            const int dir = std::min(pass, 1);
            size_t image = 0, smem = resident_smem(lay, dir == 0 ? max_src : max_rec_all, dir == 0 ? max_rec : 0, surface, nullptr, &image);
            if (pass == 2) smem += image;
            int c = 0;
            auto query = [&](const void *k, auto, auto) {
                // the limit is the kernel's, not the plan's: always the largest
                e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
                if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k, 32 * lay.warps, smem);
            };
            if (smem <= 227 * 1024) {
                if (dir == 0) res_dispatch<0>(lay, query);
                else res_dispatch<1>(lay, query);
            }
            if (e != cudaSuccess) c = 0;
            (pass == 2 ? ctas_image : ctas) = pass == 1 ? std::min(ctas, c) : c;
        }
        if (e != cudaSuccess) cudaGetLastError();
        ctas = std::min(ctas, 4);
        while (ctas > 0 && lay.us[ctas - 1] <= 0.f) --ctas;
        const int capacity = ctas * sms;
        if (most > capacity || max_rec_all > RES_MAX_POINTS) continue;
        // launches: shots by decreasing tile count, each into the first one with room
        std::vector<int> order(p->nshots);
        for (int s = 0; s < p->nshots; ++s) order[s] = s;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return st[2 * a].x > st[2 * b].x; });
        std::vector<std::vector<int>> bins;
        std::vector<int> room;
        for (int s : order) {
            size_t b = 0;
            while (b < bins.size() && room[b] < st[2 * s].x) ++b;
            if (b == bins.size()) {
                bins.push_back({});
                room.push_back(capacity);
            }
            bins[b].push_back(s);
            room[b] -= st[2 * s].x;
        }
        double us = 0;
        for (int left : room) us += lay.us[(capacity - left + sms - 1) / sms - 1];
        // The table holds bare steps.  Imaging and checkpoint segments cost the resident
        // loop more than the streaming one, per launch of tiles, so a P-SV batch in
        // several launches has to look better by that: of 60 batches of 0.2 to 11
        // million cells, those at a ratio up to 0.72 took 0.39 to 0.92 of the best
        // streaming shape's time, those above 0.81 to 1.21.  (SH batches stay below
        // 0.66, both wave types below 0.97 at any ratio.)
        if (us >= best_us || (p->g.modes == RTM_PSV && bins.size() > 1 && us > 0.72 * stream_us)) continue;
        best_us = us;
        best = rtm_plan::Resident();
        tiles.clear();
        for (auto &bin : bins) {
            const int t0 = (int)tiles.size();
            for (int s : bin)
                for (int m = 0; m < 2; ++m)
                    for (int a = 0; a < st[2 * s + m].y; ++a)
                        for (int b = 0; b < ntz; ++b) tiles.push_back(make_int4(s, a * oh[m], b * ow, m));
            best.waves.push_back(make_int2(t0, (int)tiles.size() - t0));
        }
        stiles = std::move(st);
        best.image_fits = true;
        for (const int2 &w : best.waves) best.image_fits = best.image_fits && w.y <= ctas_image * sms;
        best.layout = li;
        best.max_src = max_src;
        best.max_rec_all = max_rec_all;
        best.max_rec = max_rec;
    }
    best.surface = surface;
    if (best.layout < 0) {
        p->laid[surface] = best;
        p->is_laid[surface] = true;
        return 0;
    }
    p->res = best;
    int box = 0;
    resident_smem(RES_LAYOUTS[best.layout], 0, 0, false, &box);
    int wide = 0;
    for (const int2 &w : best.waves) wide = std::max(wide, w.y);
    p->res.box_stride = box;
    p->res.box_bytes = (size_t)box * sizeof(uint4) * wide;
    Slab slab;
    slab.add(&p->res.d_tiles, tiles.size());
    slab.add(&p->res.d_shot_tiles, stiles.size());
    slab.add(&p->res.d_sync, 2 * (size_t)p->nshots);
    slab.add(&p->res.d_box, p->res.box_bytes / sizeof(uint4));
    if (slab.commit()) {
        cudaGetLastError();  // no room: the plan streams, the next set_model tries again
        p->res = rtm_plan::Resident();
        p->res.surface = surface;
        return 0;
    }
    cudaError_t e = cudaMemcpy(p->res.d_tiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(p->res.d_shot_tiles, stiles.data(), stiles.size() * sizeof(int4), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        slab.release();
        p->res = rtm_plan::Resident();
        return fail(RTM_E_CUDA, "upload of the tiles failed: %s", cudaGetErrorString(e));
    }
    p->res.base = slab.base;
    p->laid[surface] = p->res;
    p->is_laid[surface] = true;
    return 0;
}

}  // namespace

extern "C" {

const char *rtm_version(void) {
#ifdef RTM_BOUNDS_CHECK
    return "rtm_b200 1.0 (sm_100a, bounds-checking build)";
#else
    return "rtm_b200 1.0 (sm_100a)";
#endif
}

int rtm_bounds_probe(const rtm_plan *p, const void *buf, size_t buf_bytes, const void *ptr, size_t bytes,
                     int32_t *inside) {
#ifdef RTM_BOUNDS_CHECK
    if (!p || !inside) return fail(RTM_E_ARG, "null argument");
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(buf, buf_bytes);
    if (int rc = bs.begin(0)) return rc;
    bounds_probe_kernel<<<1, 1>>>(ptr, (unsigned)bytes);
    CUDA_TRY(cudaGetLastError());
    int v = 0;
    CUDA_TRY(cudaMemcpyFromSymbol(&v, g_dbg_probe, sizeof v));
    *inside = v;
    const unsigned long long zero = 0;
    CUDA_TRY(cudaMemcpyToSymbol(g_dbg_bad, &zero, sizeof zero));  // the probe's own count
    DbgTable none{};
    CUDA_TRY(cudaMemcpyToSymbol(g_dbg_table, &none, sizeof none));
    return RTM_OK;
#else
    (void)p; (void)buf; (void)buf_bytes; (void)ptr; (void)bytes; (void)inside;
    return fail(RTM_E_STATE, "rtm_bounds_probe needs the bounds-checking build (-DRTM_BOUNDS_CHECK)");
#endif
}
const char *rtm_last_error(void) { return g_err.c_str(); }

int rtm_plan_create(const rtm_grid *grid, int nshots, const rtm_shot *shots, const rtm_tune *tune,
                    rtm_plan **out) {
    if (!grid || !shots || !out || nshots <= 0) return fail(RTM_E_ARG, "null argument or nshots <= 0");
    *out = nullptr;
    const rtm_grid g = *grid;
    if (const char *bad = check_grid(g))
        return fail(RTM_E_ARG, "%s (nx=%d nz=%d nt=%d absorbing_frame=%d)", bad, g.nx, g.nz, g.nt, g.absorbing_frame);
    rtm_plan *p = new rtm_plan();
    p->g = g;
    p->nshots = nshots;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    if (tune) {
        if (tune->vec == 1 || tune->vec == 2 || tune->vec == 4) p->vec = tune->vec;
        if (tune->rows > 0) p->rows = tune->rows;
        if (tune->warps > 0 && tune->warps <= 8) p->warps = tune->warps;
        if (tune->prefetch >= 0 && tune->prefetch <= 4) p->prefetch = tune->prefetch;
        if (p->prefetch == 4) p->warps = 1;  // the uniform-task kernel runs one warp per CTA
        p->use_graphs = tune->graphs == 1;
        if (tune->tsteps == 2) {
            if (p->vec == 1) {
                delete p;
                return fail(RTM_E_ARG, "two steps per launch need vec 2 or 4");
            }
            p->tsteps = 2;
        }
    }
    p->auto_shape = !tune || (tune->vec <= 0 && tune->rows <= 0 && tune->warps <= 0 && tune->tsteps == 0 && tune->prefetch <= 0);
    if (p->auto_shape) {
        // The streaming kernels' shape: two steps per launch, tasks of as many rows
        // as leave 16 warps per SM (a grid of a few hundred thousand cells is bound
        // by the chain of row loads in a task, a large one by the rows a task
        // computes twice).  301 x 151, one shot: 3.9 us per step with 1 row, 49 us
        // with the 32-row, one-step tasks that used to be the default.
        long long rows_all = 0;
        for (int s = 0; s < nshots; ++s) rows_all += std::max(shots[s].nx, 0);
        const long long strips = (g.nz + 59) / 60;
        p->vec = 2;
        p->tsteps = 2;
        p->rows = 24;
        while (p->rows > 1 && rows_all / p->rows * strips < sms * 16) p->rows /= 2;
        p->warps = 4;
        p->prefetch = p->rows >= 12 ? 3 : 1;
        // Long lists of tasks run fastest with 4 columns per lane, one warp per CTA
        // (14 windows of about 800 x 716, both wave types: 71 against 100 us per
        // step).  P-SV plans may be asked for an adjoint, which 2 columns suit.
        if (g.modes != RTM_PSV && rows_all / 24 * ((g.nz + 119) / 120) >= sms * 12) {
            p->vec = 4;
            p->rows = 24;
            p->warps = 1;
            p->prefetch = 4;
        }
    }
    const int W = 30 * p->vec;
    p->nstrips = (g.nz + W - 1) / W;
    p->pitch = layout_pitch(g.nz);

    // shots, row tables, work list
    std::vector<int> src_ptr, rec_ptr;
    std::vector<int2> src_ent, rec_ent;
    std::vector<int4> work;
    long long state_rows = 0;
    for (int s = 0; s < nshots; ++s) {
        const rtm_shot &sh = shots[s];
        if (sh.nx < 3 || sh.x0 < 0 || sh.x0 + sh.nx > g.nx) {
            delete p;
            return fail(RTM_E_ARG, "shot %d window [%d, %d) outside grid nx=%d", s, sh.x0, sh.x0 + sh.nx, g.nx);
        }
        if (g.absorbing_frame > sh.nx) {
            delete p;
            return fail(RTM_E_ARG, "absorbing_frame %d wider than shot %d window (%d rows)", g.absorbing_frame, s, sh.nx);
        }
        if ((sh.nsrc > 0 && !sh.src_ij) || (sh.nrec > 0 && !sh.rec_ij) || sh.nsrc < 0 || sh.nrec < 0) {
            delete p;
            return fail(RTM_E_ARG, "shot %d: bad source/receiver arrays", s);
        }
        ShotDev d{};
        d.nx = sh.nx;
        d.x0 = sh.x0;
        d.state_off = state_rows * p->pitch;
        d.row_off = p->rows_total;
        d.src_row0 = (int)src_ptr.size();
        d.rec_row0 = (int)rec_ptr.size();
        // per-row CSR, stable in the given order (duplicates accumulate in order)
        auto build = [&](int n, const int32_t *ij, int base, std::vector<int> &ptr,
                         std::vector<int2> &ent, const char *what) -> int {
            const int k = append_row_table(sh.nx, g.nz, n, ij, base, ptr, ent);
            if (k >= 0)
                return fail(RTM_E_ARG, "shot %d: %s %d at (%d, %d) outside the %dx%d window", s, what, k, ij[2 * k],
                            ij[2 * k + 1], sh.nx, g.nz);
            return 0;
        };
        if (build(sh.nsrc, sh.src_ij, p->nsrc_total, src_ptr, src_ent, "source") ||
            build(sh.nrec, sh.rec_ij, p->nrec_total, rec_ptr, rec_ent, "receiver")) {
            delete p;
            return RTM_E_ARG;
        }
        p->nsrc_total += sh.nsrc;
        p->nrec_total += sh.nrec;
        p->shots_h.push_back(d);
        state_rows += sh.nx + 2;
        p->rows_total += sh.nx;
        // Per task: bit 20 / 21 of the strip word = no source / no receiver in
        // rows [ia-2, ib+1] (every row a one- or two-step launch updates) and
        // the lanes' columns [j0 - vec, j0 + 31 vec).
        auto none_in = [&](const std::vector<int> &ptr, const std::vector<int2> &ent, int row0, int r0, int r1,
                           int c_lo, int c_hi) {
            for (int r = std::max(r0, 0); r <= std::min(r1, sh.nx - 1); ++r)
                for (int e = ptr[row0 + r]; e < ptr[row0 + r + 1]; ++e)
                    if (ent[e].x >= c_lo && ent[e].x < c_hi) return false;
            return true;
        };
        for (int ia = 0; ia < sh.nx; ia += p->rows)
            for (int st = 0; st < p->nstrips; ++st) {
                const int ib = std::min(ia + p->rows, sh.nx);
                const int j0 = st * W, c_lo = j0 - p->vec, c_hi = j0 + 31 * p->vec;
                int word = st;
                if (none_in(src_ptr, src_ent, d.src_row0, ia - 2, ib + 1, c_lo, c_hi)) word |= 1 << 20;
                if (none_in(rec_ptr, rec_ent, d.rec_row0, ia - 2, ib + 1, c_lo, c_hi)) word |= 1 << 21;
                work.push_back(make_int4(s, word, ia, ib));
            }
    }
    // Order tasks by global row so that concurrently running shots that
    // overlap read the same material rows while they are in L2.
    std::stable_sort(work.begin(), work.end(), [&](const int4 &a, const int4 &b) {
        const int ga = p->shots_h[a.x].x0 + a.z, gb = p->shots_h[b.x].x0 + b.z;
        if (ga != gb) return ga < gb;
        if (a.y != b.y) return a.y < b.y;
        return a.x < b.x;
    });
    // Tail split: the last tasks of the list (the last blocks a launch
    // dispatches) are cut into two halves of rows, so the final wave of a
    // launch is made of short tasks and the SMs run out of work closer
    // together.  Any partition of a shot's rows into tasks gives the same
    // results; a half keeps its parent's no-source / no-receiver flags, which
    // hold for any sub-range of rows.
    split_tail(work, tail_split_tasks(work.size(), sms));
    p->n_work = (int)work.size();
    p->state_floats = (size_t)state_rows * p->pitch;
    const size_t mat_floats = (size_t)(g.nx + 2) * p->pitch;
    const size_t img_floats = (size_t)p->rows_total * p->pitch;
    p->slab.add(&p->d_shots, p->shots_h.size());
    p->slab.add(&p->d_work, work.size());
    p->slab.add(&p->d_src_ptr, src_ptr.size());
    p->slab.add(&p->d_rec_ptr, rec_ptr.size());
    p->slab.add(&p->d_src_ent, std::max<size_t>(src_ent.size(), 1));
    p->slab.add(&p->d_rec_ent, std::max<size_t>(rec_ent.size(), 1));
    p->n_src_ptr = src_ptr.size();
    p->n_rec_ptr = rec_ptr.size();
    p->n_src_ent = std::max<size_t>(src_ent.size(), 1);
    p->n_rec_ent = std::max<size_t>(rec_ent.size(), 1);
    p->slab.add(&p->d_flags, (size_t)nshots + 2);  // the last words: ResParams::err
    p->slab.add(&p->d_fail_seq, nshots);
    p->slab.add(&p->d_sponge, std::max(g.absorbing_frame, 1));
    for (int b = 0; b < 2; ++b)
        for (int f = 0; f < NFIELD; ++f)
            if (field_active(g.modes, f)) p->slab.add(&p->d_state[b][f], p->state_floats);
    for (int m = 0; m < NMAT; ++m) {
        const bool need = (m <= M_MXZ) ? (g.modes & RTM_PSV) : (g.modes & RTM_SH);
        if (need) p->slab.add(&p->d_mat[m], mat_floats);
    }
    p->slab.add(&p->d_surface, mat_floats);
    for (int c = 0; c < 3; ++c)
        if (comp_active(g.modes, c)) {
            p->slab.add(&p->d_img[c], img_floats);
            p->slab.add(&p->d_imgc[c], img_floats);
        }
    p->slab.add(&p->d_seis_t, std::max<size_t>((size_t)3 * g.nt * p->nrec_total, 1));
    p->slab.add(&p->d_obs_t, std::max<size_t>((size_t)3 * g.nt * p->nrec_total, 1));
    const int rc = p->slab.commit();
    if (rc) {
        plan_free(p);
        delete p;
        return rc < 0 ? rc : RTM_E_NOMEM;
    }
    const std::vector<float> prof = sponge_profile(g.absorbing_frame);
    auto H2D = [](void *dst, const void *src, size_t bytes) {
        return bytes ? cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice) : cudaSuccess;
    };
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = H2D(p->d_shots, p->shots_h.data(), p->shots_h.size() * sizeof(ShotDev));
    if (e == cudaSuccess) e = H2D(p->d_work, work.data(), work.size() * sizeof(int4));
    if (e == cudaSuccess) e = H2D(p->d_src_ptr, src_ptr.data(), src_ptr.size() * sizeof(int));
    if (e == cudaSuccess) e = H2D(p->d_rec_ptr, rec_ptr.data(), rec_ptr.size() * sizeof(int));
    if (e == cudaSuccess) e = H2D(p->d_src_ent, src_ent.data(), src_ent.size() * sizeof(int2));
    if (e == cudaSuccess) e = H2D(p->d_rec_ent, rec_ent.data(), rec_ent.size() * sizeof(int2));
    if (e == cudaSuccess) e = H2D(p->d_sponge, prof.data(), prof.size() * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(p->d_flags, 0, ((size_t)nshots + 2) * sizeof(int));
    if (e != cudaSuccess) {
        plan_free(p);
        delete p;
        return fail(RTM_E_CUDA, "plan upload failed: %s", cudaGetErrorString(e));
    }
    if (p->auto_shape) {
        p->src_ptr_h = std::move(src_ptr);
        p->src_ent_h = std::move(src_ent);
        p->rec_ptr_h = std::move(rec_ptr);
        p->rec_ent_h = std::move(rec_ent);
        if (int r2 = resident_setup(p, false)) {
            plan_free(p);
            delete p;
            return r2;
        }
    }
    *out = p;
    return RTM_OK;
}

int rtm_plan_resident(const rtm_plan *p) { return p && p->res.layout >= 0 ? 1 : 0; }

int rtm_plan_resident_layout(const rtm_plan *p, int32_t *layout) {
    if (!p || !layout) return fail(RTM_E_ARG, "null argument");
    if (p->res.layout < 0) return fail(RTM_E_STATE, "the plan streams its wavefield");
    const ResLayout &l = RES_LAYOUTS[p->res.layout];
    const int32_t v[5] = {l.rp, l.rs, l.warps, (int32_t)p->res.waves.size(), p->res.image_fits};
    std::copy(v, v + 5, layout);
    return RTM_OK;
}

int rtm_plan_set_wait_limit(rtm_plan *p, int polls) {
    if (!p) return fail(RTM_E_ARG, "null plan");
#ifdef RTM_BOUNDS_CHECK
    p->wait_limit = polls > 0 ? std::min(polls, RES_SPIN_LIMIT) : RES_SPIN_LIMIT;
    return RTM_OK;
#else
    (void)polls;
    return fail(RTM_E_STATE, "rtm_plan_set_wait_limit needs the bounds-checking build (-DRTM_BOUNDS_CHECK)");
#endif
}

int rtm_plan_status(rtm_plan *p, int32_t *flags, rtm_stream_t stream) {
    if (!p) return fail(RTM_E_ARG, "null plan");
    return read_status(p, flags, (cudaStream_t)stream);
}

int rtm_plan_destroy(rtm_plan *p) {
    if (!p) return RTM_OK;
    plan_free(p);
    delete p;
    return RTM_OK;
}

int rtm_plan_pitch(const rtm_plan *p) { return p ? p->pitch : 0; }

size_t rtm_plan_snapshot_floats(const rtm_plan *p, int nsnap) {
    if (!p || nsnap <= 0) return 0;
    return (size_t)nsnap * (size_t)p->rows_total * (size_t)p->pitch;
}

long long rtm_plan_launch_count(const rtm_plan *p) { return p ? p->launches : 0; }

int rtm_plan_set_callback(rtm_plan *p, int forward_every, rtm_step_callback cb, void *user) {
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (cb && forward_every < 0) return fail(RTM_E_ARG, "forward_every < 0");
    p->cb = cb;
    p->cb_user = cb ? user : nullptr;
    p->cb_every = cb ? forward_every : 0;
    return RTM_OK;
}

int rtm_plan_wavefield(const rtm_plan *p, int shot, float *u, float *v, float *w, rtm_stream_t stream) {
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (shot < 0 || shot >= p->nshots) return fail(RTM_E_ARG, "shot %d outside [0, %d)", shot, p->nshots);
    if (p->live < 0) return fail(RTM_E_STATE, "no wavefield: rtm_forward / rtm_backward has not run");
    cudaStream_t s = (cudaStream_t)stream;
    const ShotDev &d = p->shots_h[shot];
    const int nz = p->g.nz;
    float *dst[3] = {u, v, w};
    const int field[3] = {F_U, F_V, F_W};
    for (int c = 0; c < 3; ++c) {
        if (!dst[c]) continue;
        const float *src = p->d_state[p->live][field[c]];
        if (!src) {  // a mode the plan does not propagate: zero
            CUDA_TRY(cudaMemsetAsync(dst[c], 0, (size_t)d.nx * nz * sizeof(float), s));
            continue;
        }
        wavefield_kernel<<<(int)std::min<long long>(((long long)d.nx * nz + 255) / 256, 148LL * 16), 256, 0, s>>>(
            src, p->d_state[1 - p->live][field[c]], p->live, p->live_seq ? p->d_fail_seq + shot : nullptr,
            d.state_off + p->pitch + COL_OFF, d.nx, nz, p->pitch, dst[c]);
        CUDA_TRY(cudaGetLastError());
    }
    return RTM_OK;
}

int rtm_plan_set_model(rtm_plan *p, const float *mu, const float *lam, const float *rho,
                       const float *surface, rtm_stream_t stream) {
    NvtxRange nvtx_range("rtm_plan_set_model");
    if (!p || !mu || !lam || !rho) return fail(RTM_E_ARG, "null model pointer");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t mat_floats = (size_t)(p->g.nx + 2) * p->pitch;
    for (int m = 0; m < NMAT; ++m)
        if (p->d_mat[m]) CUDA_TRY(cudaMemsetAsync(p->d_mat[m], 0, mat_floats * sizeof(float), s));
    CUDA_TRY(cudaMemsetAsync(p->d_surface, 0, mat_floats * sizeof(float), s));
    const long long n = (long long)p->g.nx * p->g.nz;
    const int blocks = (int)std::min<long long>((n + 255) / 256, 148LL * 16);
    setup_material_kernel<<<blocks, 256, 0, s>>>(
        mu, lam, rho, surface, p->g.nx, p->g.nz, p->pitch, p->d_mat[M_IRU], p->d_mat[M_IRW],
        p->d_mat[M_LAM], p->d_mat[M_MU], p->d_mat[M_MXZ], p->d_mat[M_IR], p->d_mat[M_MYX],
        p->d_mat[M_MYZ], surface ? p->d_surface : nullptr);
    CUDA_TRY(cudaGetLastError());
    p->has_surface = surface != nullptr;
    if (p->auto_shape && (p->has_surface != p->res.surface || !p->is_laid[p->has_surface])) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        CUDA_TRY(cudaStreamIsCapturing(s, &capture));
        if (capture != cudaStreamCaptureStatusNone && !p->is_laid[p->has_surface]) {
            p->res = rtm_plan::Resident();  // nothing can be allocated now: stream until the next set_model
            p->res.surface = p->has_surface;
        } else if (int rc = resident_setup(p, p->has_surface)) {
            return rc;
        }
    }
    p->model_set = true;
    return RTM_OK;
}

static int transpose(const float *in, float *out, int planes, int rows, int cols, cudaStream_t s) {
    if (rows == 0 || cols == 0) return 0;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32, planes);
    transpose_kernel<<<grid, dim3(32, 8), 0, s>>>(in, out, rows, cols);
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int rtm_forward(rtm_plan *p, const float *wavelets, float *seis, int save, int isnap, float *snap_u,
                float *snap_v, float *snap_w, int32_t *isnaps_out, int check_interval,
                int32_t *flags, rtm_stream_t stream) {
    NvtxRange nvtx_range("rtm_forward");
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (!p->model_set) return fail(RTM_E_STATE, "rtm_plan_set_model has not been called");
    if (p->nsrc_total > 0 && !wavelets) return fail(RTM_E_ARG, "null wavelets");
    if (check_interval < 0) return fail(RTM_E_ARG, "check_interval < 0");
    const int nt = p->g.nt;
    int nsnap = 0;
    if (save) {
        if (isnap <= 0) return fail(RTM_E_ARG, "isnap must be positive");
        nsnap = nt / isnap;  // forward_modeling.py:531
        float *sp[3] = {snap_u, snap_v, snap_w};
        for (int c = 0; c < 3; ++c)
            if (comp_active(p->g.modes, c) && nsnap > 0 && !sp[c])
                return fail(RTM_E_ARG, "snapshot buffer %d is null", c);
    }
    cudaStream_t s = (cudaStream_t)stream;
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(wavelets, (size_t)3 * p->nsrc_total * nt * sizeof(float));
    bs.add(seis, (size_t)3 * p->nrec_total * nt * sizeof(float));
    if (save)
        for (float *b : {snap_u, snap_v, snap_w}) bs.add(b, rtm_plan_snapshot_floats(p, nsnap) * sizeof(float));
    if (int rc = bs.begin(s)) return rc;
    const bool resident = p->res.layout >= 0 && !p->cb;
    if (int rc = resident ? zero_status(p, s) : zero_state(p, s)) return rc;
    // Snapshot slots the time loop never reaches ((k+1)*isnap > nt-1) stay
    // zero, like the reference's zero-initialised fields (fm:533-535).
    if (save)
        for (int k = 0; k < nsnap; ++k) {
            if ((long long)(k + 1) * isnap <= nt - 1) continue;
            float *sp3[3] = {snap_u, snap_v, snap_w};
            for (int c = 0; c < 3; ++c) {
                if (!comp_active(p->g.modes, c) || !sp3[c]) continue;
                for (const ShotDev &d : p->shots_h) {
                    const size_t off = ((size_t)nsnap * d.row_off + (size_t)k * d.nx) * p->pitch;
                    CUDA_TRY(cudaMemsetAsync(sp3[c] + off, 0, (size_t)d.nx * p->pitch * sizeof(float), s));
                }
            }
        }
    const size_t nseis = (size_t)3 * nt * p->nrec_total;
    if (nseis) CUDA_TRY(cudaMemsetAsync(p->d_seis_t, 0, nseis * sizeof(float), s));
    StepParams sp;
    fill_common(p, sp);
    sp.code_base = 1;
    const size_t plane = (size_t)nt * p->nrec_total;
    for (int c = 0; c < 3; ++c) {
        sp.wav[c] = wavelets ? wavelets + (size_t)c * p->nsrc_total * nt : nullptr;
        sp.seis[c] = p->d_seis_t + c * plane;
    }
    sp.snap[0] = snap_u;
    sp.snap[1] = snap_v;
    sp.snap[2] = snap_w;
    sp.nsnap = nsnap;
    p->launches = 0;
    auto check_at = [&](int it) { return check_interval > 0 && it % check_interval == 0; };
    auto snap_at = [&](int it) {
        const int k = (save && it % isnap == 0 && it != 0) ? it / isnap - 1 : -1;  // fm:569-570
        return k < nsnap ? k : -1;
    };
    // display_callback steps, it % every == 0 (forward_modeling.py:553-559):
    // a launch ends at each of them
    auto cb_at = [&](int it) { return p->cb && p->cb_every > 0 && it % p->cb_every == 0; };
    const std::vector<LoopLaunch> sched =
        resident ? std::vector<LoopLaunch>() : loop_schedule(0, nt, p->tsteps, [&](int it) { return !check_at(it) && !cb_at(it); });
    auto loop = [&](cudaStream_t ls) -> int {
        for (size_t L = 0; L < sched.size(); ++L) {
            const int it = sched[L].it;
            for (int f = 0; f < NFIELD; ++f) {
                sp.sin[f] = p->d_state[L & 1][f];
                sp.sout[f] = p->d_state[(L + 1) & 1][f];
            }
            sp.it = it;
            sp.seq = (int)L + 1;  // its last bit: the buffer that the launch writes
            sp.snap_k = snap_at(it);
            const int last = sched[L].two ? it + 1 : it;
            if (sched[L].two) {
                sp.it2 = it + 1;
                sp.snap_k2 = snap_at(it + 1);
                sp.check = check_at(it + 1);
                CUDA_TRY((launch_mode2<0>(sp, p->g.modes, p->vec, p->prefetch, p->warps, ls)));
            } else {
                sp.check = check_at(it);
                CUDA_TRY((launch_mode<0>(sp, p->g.modes, p->vec | (std::min(p->prefetch, 3) << 8), p->warps, ls)));
            }
            p->live = (int)((L + 1) & 1);
            p->live_seq = true;
            if (cb_at(last))
                if (int rc = call_back(p, sp.seq, last, ls)) return rc;
        }
        return 0;
    };
    const std::vector<unsigned long long> key = {U(wavelets), U(snap_u), U(snap_v), U(snap_w),
                                                 (unsigned long long)save, (unsigned long long)isnap,
                                                 (unsigned long long)check_interval, U(sp.surface)};
    if (resident) {
        ResParams rp;
        resident_params(p, rp, 0);
        for (int c = 0; c < 3; ++c) {
            rp.wav[c] = sp.wav[c];
            rp.seis[c] = sp.seis[c];
            rp.snap[c] = sp.snap[c];
        }
        rp.code_base = 1;
        rp.nsnap = nsnap;
        rp.it1 = nt;
        rp.check_interval = check_interval;
        if (nsnap > 0) {
            rp.isnap = isnap;
            rp.snap_base = rp.snap_lo = 1;
            rp.snap_hi = nsnap;
        }
        if (int rc = resident_begin(p, s)) return rc;
        if (int rc = resident_run(p, rp, 0, s)) return rc;
        p->live = 0;
        p->live_seq = false;
    } else if (p->cb) {  // host callbacks in the loop: direct launches
        if (int rc = loop(s)) return rc;
    } else if (int rc = run_loop(p, p->g_fwd, key, s, loop)) {
        return rc;
    }
    if (!resident) {  // also when a replayed graph ran the loop
        p->live = (int)(sched.size() & 1);
        p->live_seq = true;
    }
    p->launches += (long long)sched.size();
    if (seis && p->nrec_total) {
        if (int rc = transpose(p->d_seis_t, seis, 3, nt, p->nrec_total, s)) return rc;
        ++p->launches;
    }
    if (isnaps_out)
        for (int k = 0; k < nsnap; ++k) {
            const int it = (k + 1) * isnap;
            isnaps_out[k] = it <= nt - 1 ? it : 0;  // fm:572; slots never reached stay 0
        }
    if (flags)
        if (int rc = read_status(p, flags, s)) return rc;
    if (int rc = bs.end(s)) return rc;
    return RTM_OK;
}

// rtm_backward; norm_eps >= 0 adds the source-illumination normalisation of
// rtm_backward_normalized.
static int backward_impl(rtm_plan *p, const float *obs, const float *snap_u, const float *snap_v,
                         const float *snap_w, const int32_t *isnaps, int num_snaps, int isnap, float *image,
                         double *stack, int check_interval, int32_t *flags, rtm_stream_t stream,
                         double norm_eps) {
    NvtxRange nvtx_range("rtm_backward");
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (!p->model_set) return fail(RTM_E_STATE, "rtm_plan_set_model has not been called");
    if (p->nrec_total > 0 && !obs) return fail(RTM_E_ARG, "null observed data");
    if (check_interval < 0) return fail(RTM_E_ARG, "check_interval < 0");
    if (isnap <= 0) return fail(RTM_E_ARG, "isnap must be positive");
    if (num_snaps < 0 || (num_snaps > 0 && !isnaps)) return fail(RTM_E_ARG, "bad snapshot table");
    if (image && p->nshots != 1) return fail(RTM_E_ARG, "image output needs a single-shot plan; use stack");
    const float *sp3[3] = {snap_u, snap_v, snap_w};
    for (int c = 0; c < 3; ++c)
        if (comp_active(p->g.modes, c) && num_snaps > 0 && !sp3[c])
            return fail(RTM_E_ARG, "snapshot buffer %d is null", c);
    const int nt = p->g.nt;
    cudaStream_t s = (cudaStream_t)stream;
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(obs, (size_t)3 * p->nrec_total * nt * sizeof(float));
    for (const float *b : sp3) bs.add(b, rtm_plan_snapshot_floats(p, num_snaps) * sizeof(float));
    bs.add(image, (size_t)3 * p->g.nx * p->g.nz * sizeof(float));
    bs.add(stack, (size_t)3 * p->g.nx * p->g.nz * sizeof(double));
    if (int rc = bs.begin(s)) return rc;
    // the resident kernel images at every multiple of isnap that has a slot
    bool resident = p->res.layout >= 0 && !p->cb;
    for (int k = 0; k < num_snaps; ++k)
        if ((long long)(k + 1) * isnap <= nt - 1 && isnaps[k] != (k + 1) * isnap) resident = false;
    if (int rc = resident ? zero_status(p, s) : zero_state(p, s)) return rc;
    const size_t img_floats = (size_t)p->rows_total * p->pitch;
    for (int c = 0; c < 3; ++c)
        if (p->d_img[c]) {
            CUDA_TRY(cudaMemsetAsync(p->d_img[c], 0, img_floats * sizeof(float), s));
            CUDA_TRY(cudaMemsetAsync(p->d_imgc[c], 0, img_floats * sizeof(float), s));
        }
    if (p->nrec_total) {
        if (int rc = transpose(obs, p->d_obs_t, 3, p->nrec_total, nt, s)) return rc;
    }
    StepParams sp;
    fill_common(p, sp);
    sp.code_base = 4;
    const size_t plane = (size_t)nt * p->nrec_total;
    for (int c = 0; c < 3; ++c) {
        sp.obs[c] = p->d_obs_t + c * plane;
        sp.snap[c] = const_cast<float *>(sp3[c]);
        sp.img[c] = p->d_img[c];
        sp.imgc[c] = p->d_imgc[c];
    }
    sp.nsnap = num_snaps;
    p->launches = 1;
    // imaging schedule, known on the host (replaces _check_isnap_match, bm:490-496)
    std::vector<int> snap_of(nt, -1);
    for (int it = 0; it < nt; ++it) {
        const int t = (nt - 1) - it;
        if (t > 0 && t % isnap == 0) {  // backward_modeling.py:558-564
            const int k = t / isnap - 1;
            if (k >= 0 && k < num_snaps && isnaps[k] == t) snap_of[it] = k;
        }
    }
    auto check_at = [&](int it) { return check_interval > 0 && it % check_interval == 0; };
    // display_callback at every imaging step, after the correlation
    // (backward_modeling.py:565-569): a launch ends at each of them
    auto cb_at = [&](int it) { return p->cb && snap_of[it] >= 0; };
    const std::vector<LoopLaunch> sched =
        resident ? std::vector<LoopLaunch>() : loop_schedule(0, nt, p->tsteps, [&](int it) { return !check_at(it) && !cb_at(it); });
    auto loop = [&](cudaStream_t ls) -> int {
        for (size_t L = 0; L < sched.size(); ++L) {
            const int it = sched[L].it;
            for (int f = 0; f < NFIELD; ++f) {
                sp.sin[f] = p->d_state[L & 1][f];
                sp.sout[f] = p->d_state[(L + 1) & 1][f];
            }
            sp.it = (nt - 1) - it;  // backward_modeling.py:549
            sp.seq = (int)L + 1;
            sp.snap_k = snap_of[it];
            const int last = sched[L].two ? it + 1 : it;
            if (sched[L].two) {
                sp.it2 = (nt - 1) - (it + 1);
                sp.snap_k2 = snap_of[it + 1];
                sp.check = check_at(it + 1);
                CUDA_TRY((launch_mode2<1>(sp, p->g.modes, p->vec, p->prefetch, p->warps, ls)));
            } else {
                sp.check = check_at(it);
                CUDA_TRY((launch_mode<1>(sp, p->g.modes, p->vec | (std::min(p->prefetch, 3) << 8), p->warps, ls)));
            }
            p->live = (int)((L + 1) & 1);
            p->live_seq = true;
            if (cb_at(last))
                if (int rc = call_back(p, sp.seq, (nt - 1) - last, ls)) return rc;
        }
        return 0;
    };
    std::vector<unsigned long long> key = {U(snap_u), U(snap_v), U(snap_w), (unsigned long long)num_snaps,
                                           (unsigned long long)isnap, (unsigned long long)check_interval, U(sp.surface)};
    for (int it = 0; it < nt; ++it)
        if (snap_of[it] >= 0) key.push_back(((unsigned long long)it << 32) | (unsigned)snap_of[it]);
    if (resident) {
        ResParams rp;
        resident_params(p, rp, 1);
        for (int c = 0; c < 3; ++c) {
            rp.obs[c] = sp.obs[c];
            rp.snap[c] = sp.snap[c];
            rp.img[c] = sp.img[c];
            rp.imgc[c] = sp.imgc[c];
        }
        rp.code_base = 4;
        rp.nsnap = num_snaps;
        rp.it1 = nt;
        rp.check_interval = check_interval;
        if (num_snaps > 0) {
            rp.isnap = isnap;
            rp.snap_base = rp.snap_lo = 1;
            rp.snap_hi = num_snaps;
        }
        if (int rc = resident_begin(p, s)) return rc;
        if (int rc = resident_run(p, rp, 1, s)) return rc;
        p->live = 0;
        p->live_seq = false;
    } else if (p->cb) {  // host callbacks in the loop: direct launches
        if (int rc = loop(s)) return rc;
    } else if (int rc = run_loop(p, p->g_bwd, key, s, loop)) {
        return rc;
    }
    if (!resident) {  // also when a replayed graph ran the loop
        p->live = (int)(sched.size() & 1);
        p->live_seq = true;
    }
    p->launches += (long long)sched.size();
    const int blocks = 148 * 8;
    const size_t n = (size_t)p->g.nx * p->g.nz;
    // source illumination (rtm_backward_normalized): FP64 per cell, one
    // component at a time, over the snapshot slots the correlation used; in the
    // plan's scratch (allocated for each call, it took 2 to 10 ms of it)
    struct {
        double *illum = nullptr;
        unsigned long long *imax = nullptr;
        int *slots = nullptr;
    } sc;
    std::vector<int> slots;
    const bool norm = norm_eps >= 0.0;
    if (norm) {
        for (int it = 0; it < nt; ++it)
            if (snap_of[it] >= 0) slots.push_back(snap_of[it]);
        float *scratch = nullptr;
        if (int rc = plan_scratch(p, 2 * (img_floats + (size_t)p->nshots) + slots.size(), &scratch)) return rc;
        sc.illum = reinterpret_cast<double *>(scratch);
        sc.imax = reinterpret_cast<unsigned long long *>(sc.illum + img_floats);
        sc.slots = reinterpret_cast<int *>(sc.imax + p->nshots);
        if (!slots.empty())
            CUDA_TRY(cudaMemcpyAsync(sc.slots, slots.data(), slots.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    }
    for (int c = 0; c < 3; ++c) {
        IllumNorm nm;
        if (norm && p->d_img[c]) {
            CUDA_TRY(cudaMemsetAsync(sc.imax, 0, (size_t)p->nshots * sizeof(unsigned long long), s));
            illum_kernel<<<dim3(64, p->nshots), 256, 0, s>>>(sp3[c], sc.slots, (int)slots.size(), num_snaps,
                                                             p->d_shots, p->g.nz, p->pitch, sc.illum, sc.imax);
            CUDA_TRY(cudaGetLastError());
            ++p->launches;
            nm.illum = sc.illum;
            nm.imax = sc.imax;
            nm.eps = norm_eps;
        }
        if (image) {
            float *dst = image + c * n;
            if (p->d_img[c]) {
                image_out_kernel<<<blocks, 256, 0, s>>>(p->d_img[c], p->d_imgc[c], dst, 0, p->shots_h[0].nx,
                                                        p->g.nz, p->pitch, nm);
                CUDA_TRY(cudaGetLastError());
                ++p->launches;
            } else {
                CUDA_TRY(cudaMemsetAsync(dst, 0, n * sizeof(float), s));
            }
        }
        if (stack && p->d_img[c]) {
            stack_kernel<<<blocks, 256, 0, s>>>(p->d_img[c], p->d_imgc[c], stack + c * n, p->d_shots, p->nshots,
                                                p->g.nx, p->g.nz, p->pitch, nm);
            CUDA_TRY(cudaGetLastError());
            ++p->launches;
        }
    }
    if (flags || norm)  // norm: the slot table is host memory of this call
        if (int rc = read_status(p, flags, s)) return rc;
    if (int rc = bs.end(s)) return rc;
    return RTM_OK;
}

int rtm_backward(rtm_plan *p, const float *obs, const float *snap_u, const float *snap_v,
                 const float *snap_w, const int32_t *isnaps, int num_snaps, int isnap, float *image,
                 double *stack, int check_interval, int32_t *flags, rtm_stream_t stream) {
    return backward_impl(p, obs, snap_u, snap_v, snap_w, isnaps, num_snaps, isnap, image, stack, check_interval,
                         flags, stream, -1.0);
}

int rtm_backward_normalized(rtm_plan *p, const float *obs, const float *snap_u, const float *snap_v,
                            const float *snap_w, const int32_t *isnaps, int num_snaps, int isnap, float eps,
                            float *image, double *stack, int check_interval, int32_t *flags,
                            rtm_stream_t stream) {
    if (!(eps >= 0.0f) || !std::isfinite(eps)) return fail(RTM_E_ARG, "eps must be finite and >= 0");
    return backward_impl(p, obs, snap_u, snap_v, snap_w, isnaps, num_snaps, isnap, image, stack, check_interval,
                         flags, stream, (double)eps);
}

size_t rtm_plan_state_floats(const rtm_plan *p) { return p ? p->state_floats : 0; }

int rtm_plan_num_checkpoints(const rtm_plan *p, int ckpt_every) {
    if (!p || ckpt_every <= 0) return 0;
    const int nseg = (p->g.nt + ckpt_every - 1) / ckpt_every;
    return nseg - 1;
}

static bool ckpt_dtype_ok(int dtype) { return dtype >= RTM_CKPT_F32 && dtype <= RTM_CKPT_I16; }
static size_t ckpt_elem(int dtype) { return dtype == RTM_CKPT_F32 ? 4 : 2; }
static size_t ckpt_data_bytes(const rtm_plan *p, int dtype) {
    return ((size_t)NADJ * p->state_floats * ckpt_elem(dtype) + 255) & ~size_t(255);
}
// Block exponents of a compressed slot: one int32 per (field, padded state
// row, block of ckpt_block_cols(vec) columns).
static int ckpt_blocks_per_row(const rtm_plan *p) { return p->nstrips * 30 * p->vec / ckpt_block_cols(p->vec); }
static long long ckpt_shifts_per_field(const rtm_plan *p) {
    return (long long)(p->state_floats / (size_t)p->pitch) * ckpt_blocks_per_row(p);
}
static size_t ckpt_shift_bytes(const rtm_plan *p) {
    return ((size_t)NADJ * (size_t)ckpt_shifts_per_field(p) * sizeof(int) + 255) & ~size_t(255);
}
static size_t ckpt_slot_total(const rtm_plan *p, int dtype) {
    return ckpt_data_bytes(p, dtype) + (dtype == RTM_CKPT_F32 ? 0 : ckpt_shift_bytes(p));
}

size_t rtm_plan_checkpoint_bytes(const rtm_plan *p, int ckpt_every, int ckpt_dtype) {
    const int n = rtm_plan_num_checkpoints(p, ckpt_every);
    if (n <= 0 || !ckpt_dtype_ok(ckpt_dtype)) return 0;
    return (size_t)n * ckpt_slot_total(p, ckpt_dtype);
}

namespace {

// Checkpoint slot c: data, then (compressed dtypes) its block-exponent table.
unsigned char *ckpt_slot(const rtm_plan *p, void *ckpt, int dtype, int c) {
    return static_cast<unsigned char *>(ckpt) + (size_t)c * ckpt_slot_total(p, dtype);
}

// The compressed slot c as the storing step launch writes it.
CkptOut ckpt_out(const rtm_plan *p, void *ckpt, int dtype, int c) {
    unsigned char *slot = ckpt_slot(p, ckpt, dtype, c);
    CkptOut o{};
    o.data = slot;
    o.shift = reinterpret_cast<int *>(slot + ckpt_data_bytes(p, dtype));
    o.field_elems = (long long)p->state_floats;
    o.shift_per_field = ckpt_shifts_per_field(p);
    o.dtype = dtype;
    o.nblk = ckpt_blocks_per_row(p);
    return o;
}

// Restore compressed slot c into the 5 FP32 fields `dst`: the interior rows, in the
// columns that the strips cover (an even number, nz or more).  Pad rows and the left
// pad columns are left as they are: callers whose streaming launches read them clear
// them before; a resident launch reads only rows of the window and pairs of columns
// that begin below nz.
int ckpt_load(rtm_plan *p, const void *ckpt, int dtype, int c, float *const *dst, cudaStream_t s) {
    const CkptOut o = ckpt_out(p, const_cast<void *>(ckpt), dtype, c);
    CkptIn ci{};
    ci.data = o.data;
    ci.shift = o.shift;
    for (int f = 0; f < NADJ; ++f) ci.dst[f] = dst[f];
    ci.field_elems = o.field_elems;
    ci.shift_per_field = o.shift_per_field;
    ci.shots = p->d_shots;
    ci.pitch = p->pitch;
    ci.ncols = p->nstrips * 30 * p->vec;
    ci.nblk = ckpt_blocks_per_row(p);
    ci.block_w = ckpt_block_cols(p->vec);
    ci.dtype = dtype;
    ckpt_unpack_kernel<<<dim3(64, p->nshots, NADJ), 256, 0, s>>>(ci);
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// Pack the FP32 state src[] (after step seq - 1) into compressed slot c.
int ckpt_store(rtm_plan *p, void *ckpt, int dtype, int c, float *const *src, int seq, cudaStream_t s) {
    CkptFrom from{};
    for (int f = 0; f < NADJ; ++f) from.src[f] = src[f];
    from.shots = p->d_shots;
    from.fail_seq = p->d_fail_seq;
    from.pitch = p->pitch;
    from.nz = p->g.nz;
    from.seq = seq;
    ckpt_pack_kernel<<<dim3(64, p->nshots, NADJ), 256, 0, s>>>(ckpt_out(p, ckpt, dtype, c), from);
    CUDA_TRY(cudaGetLastError());
    ++p->launches;
    return 0;
}

// Where segment sgi's start state (after step sgi*K - 1) lives: the zero
// state for sgi = 0, the FP32 slot itself, or `stage` after unpacking.
int segment_start(rtm_plan *p, const void *ckpt, int dtype, int sgi, float *zero, float *stage,
                  float **out, cudaStream_t s) {
    if (sgi == 0) {
        *out = zero;
        return 0;
    }
    if (dtype == RTM_CKPT_F32) {
        *out = reinterpret_cast<float *>(ckpt_slot(p, const_cast<void *>(ckpt), dtype, sgi - 1));
        return 0;
    }
    float *dst[NADJ];
    for (int f = 0; f < NADJ; ++f) dst[f] = stage + (size_t)f * p->state_floats;
    if (int rc = ckpt_load(p, ckpt, dtype, sgi - 1, dst, s)) return rc;
    *out = stage;
    return 0;
}

}  // namespace

int rtm_forward_checkpointed(rtm_plan *p, const float *wavelets, float *seis, int ckpt_every, int ckpt_dtype,
                             void *ckpt, int check_interval, int32_t *flags, rtm_stream_t stream) {
    NvtxRange nvtx_range("rtm_forward_checkpointed");
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (!p->model_set) return fail(RTM_E_STATE, "rtm_plan_set_model has not been called");
    if (p->g.modes != RTM_PSV) return fail(RTM_E_ARG, "checkpointed propagation supports the P-SV mode");
    if (ckpt_every <= 0) return fail(RTM_E_ARG, "ckpt_every must be positive");
    if (!ckpt_dtype_ok(ckpt_dtype)) return fail(RTM_E_ARG, "bad ckpt_dtype");
    if (p->nsrc_total > 0 && !wavelets) return fail(RTM_E_ARG, "null wavelets");
    const int nt = p->g.nt;
    const int nck = rtm_plan_num_checkpoints(p, ckpt_every);
    if (nck > 0 && !ckpt) return fail(RTM_E_ARG, "null checkpoint buffer");
    cudaStream_t s = (cudaStream_t)stream;
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(wavelets, (size_t)3 * p->nsrc_total * nt * sizeof(float));
    bs.add(seis, (size_t)3 * p->nrec_total * nt * sizeof(float));
    bs.add(ckpt, rtm_plan_checkpoint_bytes(p, ckpt_every, ckpt_dtype));
    if (int rc = bs.begin(s)) return rc;
    const bool resident = p->res.layout >= 0;
    if (int rc = resident ? zero_status(p, s) : zero_state(p, s)) return rc;
    // every slot starts at zero: pad rows / columns of FP32 slots, and the
    // slots of a shot that stops before reaching them
    if (nck > 0) CUDA_TRY(cudaMemsetAsync(ckpt, 0, rtm_plan_checkpoint_bytes(p, ckpt_every, ckpt_dtype), s));
    const size_t nseis = (size_t)3 * nt * p->nrec_total;
    if (nseis) CUDA_TRY(cudaMemsetAsync(p->d_seis_t, 0, nseis * sizeof(float), s));
    StepParams sp;
    fill_common(p, sp);
    sp.code_base = 1;
    const size_t plane = (size_t)nt * p->nrec_total;
    for (int c = 0; c < 3; ++c) {
        sp.wav[c] = wavelets ? wavelets + (size_t)c * p->nsrc_total * nt : nullptr;
        sp.seis[c] = p->d_seis_t + c * plane;
    }
    float *in[NFIELD] = {}, *out[NFIELD] = {};
    for (int f = 0; f < NADJ; ++f) in[f] = p->d_state[0][f];
    p->launches = 0;
    p->live = -1;
    auto check_at = [&](int it) { return check_interval > 0 && it % check_interval == 0; };
    auto save_at = [&](int it) { return (it + 1) % ckpt_every == 0 && it + 1 < nt; };
    if (resident) {
        // FP32 slots are written by one launch over all steps (201 x 101, 18 segments:
        // 0.1 ms less than a launch each).  16-bit ones are packed from a state buffer,
        // one segment between checkpoints at a time.
        const bool f32 = ckpt_dtype == RTM_CKPT_F32;
        const int len = f32 ? nt : ckpt_every;
        ResParams rp;
        resident_params(p, rp, 0);
        for (int c = 0; c < 3; ++c) {
            rp.wav[c] = sp.wav[c];
            rp.seis[c] = sp.seis[c];
        }
        rp.code_base = 1;
        rp.check_interval = check_interval;
        rp.segment = !f32;
        rp.keep_every = f32 ? ckpt_every : 0;
        rp.keep = (long long)(ckpt_slot_total(p, RTM_CKPT_F32) / sizeof(float));
        if (int rc = resident_begin(p, s)) return rc;
        for (int start = 0, seg = 0; start < nt; start += len, ++seg) {
            const int end = std::min(start + len, nt);
            const bool save = !f32 && end < nt;
            float *dst[NADJ];
            for (int f = 0; f < NADJ; ++f) {
                dst[f] = f32 && ckpt ? static_cast<float *>(ckpt) + (size_t)f * p->state_floats : p->d_state[seg & 1][f];
                rp.store[f] = save || f32 ? dst[f] : nullptr;
            }
            rp.it0 = start;
            rp.it1 = end;
            if (int rc = resident_run(p, rp, 0, s)) return rc;
            if (save) {
                if (int rc = ckpt_store(p, ckpt, ckpt_dtype, seg, dst, end, s)) return rc;
            }
            for (int f = 0; f < NADJ; ++f) rp.load[f] = dst[f];
        }
    }
    const std::vector<LoopLaunch> sched =
        resident ? std::vector<LoopLaunch>() : loop_schedule(0, nt, p->tsteps, [&](int it) { return !check_at(it) && !save_at(it); });
    for (const LoopLaunch &ln : sched) {
        const int last = ln.two ? ln.it + 1 : ln.it;  // the step whose state the launch writes
        const bool save = save_at(last);
        const int c = (last + 1) / ckpt_every - 1;
        for (int f = 0; f < NADJ; ++f) {
            if (save && ckpt_dtype == RTM_CKPT_F32)  // the step writes its output into the slot
                out[f] = reinterpret_cast<float *>(ckpt_slot(p, ckpt, ckpt_dtype, c)) + (size_t)f * p->state_floats;
            else
                out[f] = (in[f] == p->d_state[0][f]) ? p->d_state[1][f] : p->d_state[0][f];
            sp.sin[f] = in[f];
            sp.sout[f] = out[f];
        }
        sp.it = ln.it;
        sp.seq = ln.it + 1;
        sp.check = check_at(last);
        if (ln.two) {
            sp.it2 = last;
            sp.snap_k2 = -1;
        }
        if (save && ckpt_dtype != RTM_CKPT_F32) {
            // the launch also packs its output state into compressed slot c
            sp.ck = ckpt_out(p, ckpt, ckpt_dtype, c);
            CUDA_TRY(launch_ckpt(sp, ln.two, p->vec, p->prefetch, p->warps, s));
            sp.ck = CkptOut{};
        } else if (ln.two) {
            CUDA_TRY((launch_mode2<0>(sp, p->g.modes, p->vec, p->prefetch, p->warps, s)));
        } else {
            CUDA_TRY((launch_mode<0>(sp, p->g.modes, p->vec | (std::min(p->prefetch, 3) << 8), p->warps, s)));
        }
        ++p->launches;
        for (int f = 0; f < NADJ; ++f) in[f] = out[f];
    }
    if (seis && p->nrec_total) {
        if (int rc = transpose(p->d_seis_t, seis, 3, nt, p->nrec_total, s)) return rc;
        ++p->launches;
    }
    if (flags)
        if (int rc = read_status(p, flags, s)) return rc;
    if (int rc = bs.end(s)) return rc;
    return RTM_OK;
}

int rtm_adjoint(rtm_plan *p, const float *wavelets, const float *resid, int ckpt_every, int ckpt_dtype,
                const void *ckpt, double *grad, float *grad_wavelet, rtm_stream_t stream) {
    NvtxRange nvtx_range("rtm_adjoint");
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (!p->model_set) return fail(RTM_E_STATE, "rtm_plan_set_model has not been called");
    if (p->g.modes != RTM_PSV) return fail(RTM_E_ARG, "the adjoint supports the P-SV mode");
    if (ckpt_every <= 0) return fail(RTM_E_ARG, "ckpt_every must be positive");
    if (!ckpt_dtype_ok(ckpt_dtype)) return fail(RTM_E_ARG, "bad ckpt_dtype");
    if (!grad) return fail(RTM_E_ARG, "null gradient output");
    if (p->nrec_total > 0 && !resid) return fail(RTM_E_ARG, "null residual");
    if (p->nsrc_total > 0 && !wavelets) return fail(RTM_E_ARG, "null wavelets");
    const int nt = p->g.nt;
    const int K = ckpt_every;
    const int nseg = (nt + K - 1) / K;
    if (nseg > 1 && !ckpt) return fail(RTM_E_ARG, "null checkpoint buffer");
    cudaStream_t s = (cudaStream_t)stream;
    const size_t sf = p->state_floats;
    const size_t slot = (size_t)NADJ * sf;
    const size_t gfl = (size_t)p->rows_total * p->pitch;
    // scratch: K-1 recompute slots, zero state, 2 adjoint states, unpack stage;
    // Kahan gradients; wavelet gradient
    // (the plan's scratch, subdivided; every piece starts on a 128-byte
    // boundary since state_floats and gfl are multiples of the pitch)
    const size_t nrec_slots = (size_t)std::max(K - 1, 1);
    const size_t nslots = nrec_slots + 1 + 2 + (ckpt_dtype == RTM_CKPT_F32 ? 0 : 1);
    const size_t n_gsum = (size_t)3 * NGRAD * gfl;  // Kahan sums, compensations, partials
    const size_t n_gwt = grad_wavelet && p->nsrc_total ? (size_t)3 * nt * p->nsrc_total : 0;
    float *scratch = nullptr;
    if (int rc = plan_scratch(p, nslots * slot + n_gsum + n_gwt, &scratch)) return rc;
    float *seg = scratch, *gsum = seg + nslots * slot, *gwt = n_gwt ? gsum + n_gsum : nullptr;
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(wavelets, (size_t)3 * p->nsrc_total * nt * sizeof(float));
    bs.add(ckpt, rtm_plan_checkpoint_bytes(p, ckpt_every, ckpt_dtype));
    bs.add(seg, nslots * slot * sizeof(float));
    bs.add(gsum, (size_t)3 * NGRAD * gfl * sizeof(float));
    bs.add(gwt, (size_t)3 * nt * p->nsrc_total * sizeof(float));
    p->live = -1;
    auto body = [&]() -> int {
        if (int r = bs.begin(s)) return r;
        if (int r = zero_status(p, s)) return r;
        CUDA_TRY(cudaMemsetAsync(seg, 0, nslots * slot * sizeof(float), s));
        CUDA_TRY(cudaMemsetAsync(gsum, 0, (size_t)3 * NGRAD * gfl * sizeof(float), s));
        if (gwt) CUDA_TRY(cudaMemsetAsync(gwt, 0, (size_t)3 * nt * p->nsrc_total * sizeof(float), s));
        if (p->nrec_total) {
            if (int r = transpose(resid, p->d_obs_t, 3, p->nrec_total, nt, s)) return r;
        }
        float *zero = seg + nrec_slots * slot;
        float *adj[2] = {zero + slot, zero + 2 * slot};
        float *stage = zero + 3 * slot;
        auto fld = [&](float *base, int f) { return base + (size_t)f * sf; };
        // a_{nt-1} = R^T g_{nt-1}
        if (p->nrec_total) {
            int max_nx = 1;
            for (const ShotDev &d : p->shots_h) max_nx = std::max(max_nx, d.nx);
            inject_last_resid_kernel<<<dim3((max_nx + 127) / 128, p->nshots), 128, 0, s>>>(
                p->d_shots, p->nshots, p->d_rec_ptr, p->d_rec_ent, p->d_obs_t, nt, p->nrec_total,
                p->g.nz, p->pitch, fld(adj[0], A_U), fld(adj[0], A_W));
            CUDA_TRY(cudaGetLastError());
        }
        StepParams sp;
        fill_common(p, sp);
        sp.check = 0;
        const size_t plane = (size_t)nt * p->nrec_total;
        for (int c = 0; c < 3; ++c) {
            sp.wav[c] = wavelets ? wavelets + (size_t)c * p->nsrc_total * nt : nullptr;
            sp.seis[c] = p->d_seis_t + c * plane;  // recompute records here; not returned
        }
        AdjParams ap;
        std::memset(&ap, 0, sizeof ap);
        ap.nz = p->g.nz;
        ap.pitch = p->pitch;
        ap.nt = nt;
        ap.fw = p->g.absorbing_frame;
        ap.dt = sp.dt;
        ap.inv_dx = sp.inv_dx;
        ap.inv_dz = sp.inv_dz;
        ap.src_factor = sp.src_factor;
        ap.sponge = p->d_sponge;
        ap.work = p->d_work;
        ap.n_work = p->n_work;
        ap.shots = p->d_shots;
        for (int m = 0; m < NMAT; ++m) ap.mat[m] = p->d_mat[m];
        ap.surface = p->has_surface ? p->d_surface : nullptr;
        ap.src_ptr = p->d_src_ptr;
        ap.src_ent = p->d_src_ent;
        ap.rec_ptr = p->d_rec_ptr;
        ap.rec_ent = p->d_rec_ent;
        ap.nrec_total = p->nrec_total;
        ap.nsrc_total = p->nsrc_total;
        for (int c = 0; c < 3; ++c) {
            ap.wav[c] = sp.wav[c];
            ap.resid[c] = p->d_obs_t + c * plane;
            ap.gwav[c] = gwt ? gwt + (size_t)c * nt * p->nsrc_total : nullptr;
        }
        GradFold fold;
        fold.n = (long long)gfl;
        for (int g = 0; g < NGRAD; ++g) {
            fold.sum[g] = gsum + (size_t)g * gfl;
            fold.comp[g] = gsum + (size_t)(NGRAD + g) * gfl;
            fold.part[g] = gsum + (size_t)(2 * NGRAD + g) * gfl;
            ap.gpart[g] = fold.part[g];
        }
        // A resident plan recomputes on the chip (its streaming launches are bound by
        // their row chains: gradient of 201 x 101, 300 steps, 4.6 -> 3.9 ms).
        const bool resident = p->res.layout >= 0;
        ResParams rp;
        if (resident) {
            resident_params(p, rp, 0);
            for (int c = 0; c < 3; ++c) {
                rp.wav[c] = sp.wav[c];
                rp.seis[c] = sp.seis[c];
            }
            rp.keep_every = 1;
            rp.keep = (long long)slot;
            if (int r = resident_begin(p, s)) return r;
        }
        int cur = 0;
        const int warps = p->warps;
        const int blocks = (p->n_work + warps - 1) / warps;
        p->launches = 1;
        for (int sgi = nseg - 1; sgi >= 0; --sgi) {
            const int start = sgi * K, end = std::min(start + K, nt);
            float *s0 = nullptr;
            if (int r = segment_start(p, ckpt, ckpt_dtype, sgi, zero, stage, &s0, s)) return r;
            // recompute forward states start .. end-2 into seg slots 0 .. len-2: in one
            // resident launch that stores the state of every step, or two steps
            // per launch (each state stored) where the plan runs two
            if (resident && end - start >= 2) {
                for (int f = 0; f < NADJ; ++f) {
                    rp.load[f] = fld(s0, f);
                    rp.store[f] = fld(seg, f);
                }
                rp.it0 = start;
                rp.it1 = end - 1;
                if (int r = resident_run(p, rp, 0, s)) return r;
            }
            for (int it = start; !resident && it <= end - 2;) {
                float *src = it == start ? s0 : seg + (size_t)(it - 1 - start) * slot;
                float *dst = seg + (size_t)(it - start) * slot;
                const bool two = p->tsteps == 2 && p->vec >= 2 && it + 1 <= end - 2;
                for (int f = 0; f < NADJ; ++f) {
                    sp.sin[f] = fld(src, f);
                    sp.souta[f] = two ? fld(dst, f) : nullptr;
                    sp.sout[f] = two ? fld(dst + slot, f) : fld(dst, f);
                }
                sp.it = it;
                sp.seq = it + 1;
                if (two) {
                    sp.it2 = it + 1;
                    sp.snap_k2 = -1;
                    CUDA_TRY(launch_recompute2(sp, p->vec, p->prefetch, warps, s));
                    it += 2;
                } else {
                    CUDA_TRY((launch_mode<0>(sp, RTM_PSV, p->vec | (std::min(p->prefetch, 3) << 8), warps, s)));
                    it += 1;
                }
                ++p->launches;
            }
            // reverse steps end-1 .. start; with two steps per launch, steps n and
            // n-1 together unless the partials are folded after step n
            auto fwd_state = [&](int m) { return m == start ? s0 : seg + (size_t)(m - 1 - start) * slot; };
            for (int n = end - 1; n >= start;) {
                float *fs = fwd_state(n);
                for (int f = 0; f < NADJ; ++f) {
                    ap.fwd[f] = fld(fs, f);
                    ap.ain[f] = fld(adj[cur], f);
                    ap.aout[f] = fld(adj[1 - cur], f);
                }
                ap.n = n;
                if (p->tsteps == 2 && p->vec >= 2 && n - 1 >= start && n % GRAD_FOLD_STEPS != 0) {
                    float *fs2 = fwd_state(n - 1);
                    for (int f = 0; f < NADJ; ++f) ap.fwd2[f] = fld(fs2, f);
                    // one warp per CTA: the uniform-task instantiation (same task, same arithmetic)
                    if (p->vec == 2) {
                        if (warps == 1) adjoint2_kernel<2, true><<<blocks, 32, 0, s>>>(ap);
                        else adjoint2_kernel<2><<<blocks, 32 * warps, 0, s>>>(ap);
                    } else {
                        adjoint2_kernel<4><<<blocks, 32 * warps, 0, s>>>(ap);
                    }
                    CUDA_TRY(cudaGetLastError());
                    ++p->launches;
                    cur = 1 - cur;
                    n -= 2;
                    if ((n + 1) % GRAD_FOLD_STEPS == 0) {  // after step n+1 (the pair's second)
                        grad_fold_kernel<<<148 * 8, 256, 0, s>>>(fold);
                        CUDA_TRY(cudaGetLastError());
                        ++p->launches;
                    }
                    continue;
                }
                switch (p->vec) {
                    case 1: adjoint_step_kernel<1><<<blocks, 32 * warps, 0, s>>>(ap); break;
                    case 2:
                        if (warps == 1) adjoint_step_kernel<2, true><<<blocks, 32, 0, s>>>(ap);
                        else adjoint_step_kernel<2><<<blocks, 32 * warps, 0, s>>>(ap);
                        break;
                    default: adjoint_step_kernel<4><<<blocks, 32 * warps, 0, s>>>(ap); break;
                }
                CUDA_TRY(cudaGetLastError());
                ++p->launches;
                cur = 1 - cur;
                if (n % GRAD_FOLD_STEPS == 0) {  // n = 0 is the last step: everything is folded
                    grad_fold_kernel<<<148 * 8, 256, 0, s>>>(fold);
                    CUDA_TRY(cudaGetLastError());
                    ++p->launches;
                }
                --n;
            }
        }
        const size_t n2 = (size_t)p->g.nx * p->g.nz;
        for (int g = 0; g < NGRAD; ++g) {
            stack_kernel<<<148 * 8, 256, 0, s>>>(fold.sum[g], fold.comp[g], grad + g * n2, p->d_shots, p->nshots,
                                                 p->g.nx, p->g.nz, p->pitch);
            CUDA_TRY(cudaGetLastError());
        }
        if (gwt) {
            if (int r = transpose(gwt, grad_wavelet, 3, nt, p->nsrc_total, s)) return r;
        }
        if (int r = read_status(p, nullptr, s)) return r;
        if (int r = bs.end(s)) return r;
        return RTM_OK;
    };
    return body();
}

int rtm_backward_checkpointed(rtm_plan *p, const float *wavelets, const float *obs, int ckpt_every,
                              int ckpt_dtype, const void *ckpt, int isnap, float *image, double *stack,
                              int check_interval, int32_t *flags, rtm_stream_t stream) {
    NvtxRange nvtx_range("rtm_backward_checkpointed");
    if (!p) return fail(RTM_E_ARG, "null plan");
    if (!p->model_set) return fail(RTM_E_STATE, "rtm_plan_set_model has not been called");
    if (p->g.modes != RTM_PSV) return fail(RTM_E_ARG, "checkpointed RTM supports the P-SV mode");
    if (ckpt_every <= 0 || isnap <= 0) return fail(RTM_E_ARG, "ckpt_every and isnap must be positive");
    if (!ckpt_dtype_ok(ckpt_dtype)) return fail(RTM_E_ARG, "bad ckpt_dtype");
    if (p->nrec_total > 0 && !obs) return fail(RTM_E_ARG, "null observed data");
    if (p->nsrc_total > 0 && !wavelets) return fail(RTM_E_ARG, "null wavelets");
    if (image && p->nshots != 1) return fail(RTM_E_ARG, "image output needs a single-shot plan; use stack");
    const int nt = p->g.nt;
    const int K = ckpt_every;
    const int nseg = (nt + K - 1) / K;
    if (nseg > 1 && !ckpt) return fail(RTM_E_ARG, "null checkpoint buffer");
    const int num_snaps = nt / isnap;  // the snapshot slots the reference would allocate (fm:531)
    cudaStream_t s = (cudaStream_t)stream;
    const size_t sf = p->state_floats;
    const size_t slot = (size_t)NADJ * sf;
    const int seg_snaps = K / isnap + 1;
    const size_t snap_comp = (size_t)seg_snaps * p->rows_total * p->pitch;
    // scratch: recompute ping-pong (2 states), zero state, unpack stage, segment snapshots (u, w)
    float *buf = nullptr;
    const size_t nbuf = 4 * slot + 2 * snap_comp;
    if (int rc = plan_scratch(p, nbuf, &buf)) return rc;
    BoundsScope bs;
    bs.add_plan(p);
    bs.add(wavelets, (size_t)3 * p->nsrc_total * nt * sizeof(float));
    bs.add(obs, (size_t)3 * p->nrec_total * nt * sizeof(float));
    bs.add(ckpt, rtm_plan_checkpoint_bytes(p, ckpt_every, ckpt_dtype));
    bs.add(image, (size_t)3 * p->g.nx * p->g.nz * sizeof(float));
    bs.add(stack, (size_t)3 * p->g.nx * p->g.nz * sizeof(double));
    bs.add(buf, nbuf * sizeof(float));
    p->live = -1;
    auto body = [&]() -> int {
        if (int rc = bs.begin(s)) return rc;
        const bool resident = p->res.layout >= 0;
        if (int rc = resident ? zero_status(p, s) : zero_state(p, s)) return rc;
        if (!resident) CUDA_TRY(cudaMemsetAsync(buf, 0, nbuf * sizeof(float), s));
        else if (int rc = resident_begin(p, s)) return rc;
        const size_t img_floats = (size_t)p->rows_total * p->pitch;
        for (int c = 0; c < 3; ++c)
            if (p->d_img[c]) {
                CUDA_TRY(cudaMemsetAsync(p->d_img[c], 0, img_floats * sizeof(float), s));
                CUDA_TRY(cudaMemsetAsync(p->d_imgc[c], 0, img_floats * sizeof(float), s));
            }
        if (p->nrec_total) {
            if (int r = transpose(obs, p->d_obs_t, 3, p->nrec_total, nt, s)) return r;
        }
        float *rec[2] = {buf, buf + slot};
        float *zero = buf + 2 * slot, *stage = buf + 3 * slot;
        float *snapu = buf + 4 * slot, *snapw = snapu + snap_comp;
        const size_t plane = (size_t)nt * p->nrec_total;
        StepParams fp;  // forward recompute
        fill_common(p, fp);
        fp.check = 0;
        fp.nsnap = seg_snaps;
        fp.snap[0] = snapu;
        fp.snap[2] = snapw;
        for (int c = 0; c < 3; ++c) {
            fp.wav[c] = wavelets ? wavelets + (size_t)c * p->nsrc_total * nt : nullptr;
            fp.seis[c] = p->d_seis_t + c * plane;  // not returned
        }
        StepParams bp;  // backward with imaging
        fill_common(p, bp);
        bp.code_base = 4;
        bp.nsnap = seg_snaps;
        bp.snap[0] = snapu;
        bp.snap[2] = snapw;
        for (int c = 0; c < 3; ++c) {
            bp.obs[c] = p->d_obs_t + c * plane;
            bp.img[c] = p->d_img[c];
            bp.imgc[c] = p->d_imgc[c];
        }
        // imaging at t > 0, t % isnap == 0 with a snapshot slot t/isnap - 1 < nt/isnap
        // that the forward fills (t <= nt-1): backward_modeling.py:556-564, fm:569-572
        auto images_at = [&](int t) { return t > 0 && t % isnap == 0 && t / isnap - 1 < num_snaps && t <= nt - 1; };
        auto check_at = [&](int it) { return check_interval > 0 && it % check_interval == 0; };
        p->launches = 1;
        long long nb = 0;  // backward launches so far: the ping-pong parity
        for (int sgi = nseg - 1; sgi >= 0; --sgi) {
            const int start = sgi * K, end = std::min(start + K, nt);
            float *s0 = nullptr;
            if (int r = segment_start(p, ckpt, ckpt_dtype, sgi, zero, stage, &s0, s)) return r;
            // recompute forward steps start .. end-1, keeping u, w at imaging steps
            const int first = ((start + isnap - 1) / isnap) * isnap;  // first multiple of isnap >= start
            auto slot_at = [&](int t) { return images_at(t) ? (t - first) / isnap : -1; };
            if (resident) {
                ResParams rp;
                resident_params(p, rp, 0);
                for (int c = 0; c < 3; ++c) rp.wav[c] = fp.wav[c];
                rp.nsnap = seg_snaps;
                rp.snap[0] = snapu;
                rp.snap[2] = snapw;
                rp.isnap = isnap;
                rp.snap_base = first / isnap;
                rp.snap_lo = 1;
                rp.snap_hi = num_snaps;
                rp.it0 = start;
                rp.it1 = end;
                for (int f = 0; f < NADJ; ++f) {
                    rp.load[f] = sgi == 0 ? nullptr : s0 + (size_t)f * sf;
                    rp.store[f] = nullptr;
                }
                if (int r = resident_run(p, rp, 0, s)) return r;
                resident_params(p, rp, 1);
                for (int c = 0; c < 3; ++c) {
                    rp.obs[c] = bp.obs[c];
                    rp.img[c] = bp.img[c];
                    rp.imgc[c] = bp.imgc[c];
                }
                rp.nsnap = seg_snaps;
                rp.snap[0] = snapu;
                rp.snap[2] = snapw;
                rp.isnap = isnap;
                rp.snap_base = first / isnap;
                rp.snap_lo = 1;
                rp.snap_hi = num_snaps;
                rp.code_base = 4;
                rp.check_interval = check_interval;
                rp.segment = true;
                rp.it0 = nt - end;
                rp.it1 = nt - start;
                for (int f = 0; f < NADJ; ++f) {
                    rp.load[f] = nb == 0 ? nullptr : p->d_state[nb & 1][f];
                    rp.store[f] = p->d_state[(nb + 1) & 1][f];
                }
                if (int r = resident_run(p, rp, 1, s)) return r;
                ++nb;
                continue;
            }
            const std::vector<LoopLaunch> fsched = loop_schedule(start, end, p->tsteps, [](int) { return true; });
            for (size_t L = 0; L < fsched.size(); ++L) {
                const int it = fsched[L].it;
                float *src = L == 0 ? s0 : rec[(L - 1) & 1];
                float *dst = rec[L & 1];
                for (int f = 0; f < NADJ; ++f) {
                    fp.sin[f] = src + (size_t)f * sf;
                    fp.sout[f] = dst + (size_t)f * sf;
                }
                fp.it = it;
                fp.seq = it + 1;
                fp.snap_k = slot_at(it);
                if (fsched[L].two) {
                    fp.it2 = it + 1;
                    fp.snap_k2 = slot_at(it + 1);
                    CUDA_TRY((launch_mode2<0>(fp, RTM_PSV, p->vec, p->prefetch, p->warps, s)));
                } else {
                    CUDA_TRY((launch_mode<0>(fp, RTM_PSV, p->vec | (std::min(p->prefetch, 3) << 8), p->warps, s)));
                }
                ++p->launches;
            }
            // backward iterations it whose reversed time t = nt-1-it falls in [start, end)
            const std::vector<LoopLaunch> bsched =
                loop_schedule(nt - end, nt - start, p->tsteps, [&](int it) { return !check_at(it); });
            for (const LoopLaunch &ln : bsched) {
                const int it = ln.it, t = (nt - 1) - it;
                for (int f = 0; f < NFIELD; ++f) {
                    bp.sin[f] = p->d_state[nb & 1][f];
                    bp.sout[f] = p->d_state[(nb + 1) & 1][f];
                }
                bp.it = t;
                bp.seq = it + 1;
                bp.snap_k = slot_at(t);
                if (ln.two) {
                    bp.it2 = t - 1;
                    bp.snap_k2 = slot_at(t - 1);
                    bp.check = check_at(it + 1);
                    CUDA_TRY((launch_mode2<1>(bp, RTM_PSV, p->vec, p->prefetch, p->warps, s)));
                } else {
                    bp.check = check_at(it);
                    CUDA_TRY((launch_mode<1>(bp, RTM_PSV, p->vec | (std::min(p->prefetch, 3) << 8), p->warps, s)));
                }
                ++p->launches;
                ++nb;
            }
        }
        const int blocks = 148 * 8;
        if (image) {
            const size_t n = (size_t)p->g.nx * p->g.nz;
            for (int c = 0; c < 3; ++c) {
                float *dst = image + c * n;
                if (p->d_img[c]) {
                    image_out_kernel<<<blocks, 256, 0, s>>>(p->d_img[c], p->d_imgc[c], dst, 0, p->shots_h[0].nx,
                                                            p->g.nz, p->pitch);
                    CUDA_TRY(cudaGetLastError());
                } else {
                    CUDA_TRY(cudaMemsetAsync(dst, 0, n * sizeof(float), s));
                }
            }
        }
        if (stack) {
            const size_t n = (size_t)p->g.nx * p->g.nz;
            for (int c = 0; c < 3; ++c)
                if (p->d_img[c]) {
                    stack_kernel<<<blocks, 256, 0, s>>>(p->d_img[c], p->d_imgc[c], stack + c * n, p->d_shots,
                                                        p->nshots, p->g.nx, p->g.nz, p->pitch);
                    CUDA_TRY(cudaGetLastError());
                }
        }
        if (int rc = read_status(p, flags, s)) return rc;  // the call waits for its results in any case
        if (int rc = bs.end(s)) return rc;
        return RTM_OK;
    };
    return body();
}

}  // extern "C"
