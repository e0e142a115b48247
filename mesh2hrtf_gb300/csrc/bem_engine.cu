// bem_engine.cu - host side of the batched Krylov engine: launch table,
// work-item lists, graph capture and replay.
#include <cuda_runtime.h>

#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>

#include <cudaTypedefs.h>

#include "bem_engine.h"

namespace bem {

namespace {
// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// TMA map of a complex64 matrix viewed as n rows of 2 n floats (row pitch
// 2 lda floats): boxes of 32 floats x kUmRows rows with the 128-byte swizzle,
// zeros outside the matrix
bool encode_group_map(CUtensorMap *map, const void *A, int n, long long lda) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)(2 * (long long)n), (cuuint64_t)n};
    cuuint64_t strides[1] = {(cuuint64_t)(2 * lda * 4)};
    cuuint32_t box[2] = {32, (cuuint32_t)kUmRows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(A), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// BEM_GB300_TEST_WAIT_CYCLES: a bound (clock cycles) for the products'
// mbarrier waits in place of the default of about 2 s.  Only for tests that
// make a wait run out; read whenever a batch is set up.
// BEM_GB300_TEST_WAIT_KINDS: the product kinds the bound applies to (bit k:
// kind k; 0 Krylov products, 1 first refinement residuals, 2 residual
// updates); all by default.
int test_wait_kinds() {
    const char *v = std::getenv("BEM_GB300_TEST_WAIT_KINDS");
    return (v && *v) ? std::atoi(v) : 7;
}

long long test_wait_cycles() {
    const char *v = std::getenv("BEM_GB300_TEST_WAIT_CYCLES");
    if (!v || !*v) return 0;
    const long long c = std::atoll(v);
    return c > 0 ? c : 0;
}
}  // namespace

Engine::~Engine() {
    if (st_) cudaStreamSynchronize(st_);
    for (auto &part : exec_)
        for (auto &x : part)
            if (x) cudaGraphExecDestroy(x);
    for (auto &e : ev_)
        if (e) cudaEventDestroy(e);
    if (side_.fork) cudaEventDestroy(side_.fork);
    if (side_.join) cudaEventDestroy(side_.join);
    if (side_.st) cudaStreamDestroy(side_.st);
    cudaFree(d_tab_);
    cudaFree(d_st_);
    cudaFree(d_items_);
    if (h_tab_) cudaFreeHost(h_tab_);
    if (h_st_) cudaFreeHost(h_st_);
}

cudaError_t Engine::ensure_init() {
    if (d_tab_) return cudaSuccess;
    cudaError_t e = krylov_prepare();
    if (e == cudaSuccess) e = cudaMalloc(&d_tab_, sizeof(KTable));
    if (e == cudaSuccess) e = cudaMalloc(&d_st_, sizeof(KState) * kMaxSys);
    if (e == cudaSuccess) e = cudaMallocHost(&h_tab_, sizeof(KTable));
    if (e == cudaSuccess) e = cudaMallocHost(&h_st_, sizeof(KState) * kMaxSys);
    for (auto &ev : ev_)
        if (e == cudaSuccess) e = cudaEventCreate(&ev);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&side_.st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&side_.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&side_.join, cudaEventDisableTiming);
    if (e == cudaSuccess) {
        std::memset(h_tab_, 0, sizeof(KTable));
        std::memset(h_st_, 0, sizeof(KState) * kMaxSys);
        e = cudaMemcpyAsync(d_tab_, h_tab_, sizeof(KTable), cudaMemcpyHostToDevice, st_);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    return e;
}

cudaError_t Engine::set_batch(const std::vector<KSys> &sys, const std::vector<KState> &init) {
    if (sys.size() != init.size() || sys.size() > (size_t)kMaxSys) return cudaErrorInvalidValue;
    cudaError_t e = ensure_init();
    if (e != cudaSuccess) return e;
    // the previous replay (if any) has completed: run_body synchronizes
    const int B = (int)sys.size();
    items_.clear();
    int vb_total = 0;
    for (int b = 0; b < B; ++b) vb_total += sys[b].nvb;
    items_.reserve((size_t)vb_total);
    for (int b = 0; b < B; ++b)
        for (int q = 0; q < sys[b].nvb; ++q) items_.push_back(make_int2(b, q));
    if (items_.size() > items_cap_) {
        cudaFree(d_items_);
        d_items_ = nullptr;
        items_cap_ = 0;
        const size_t cap = items_.size() + items_.size() / 4 + 1024;
        e = cudaMalloc(&d_items_, cap * sizeof(int2));
        if (e != cudaSuccess) return e;
        items_cap_ = cap;
    }
    if (!items_.empty())
        e = cudaMemcpyAsync(d_items_, items_.data(), items_.size() * sizeof(int2), cudaMemcpyHostToDevice, st_);
    if (e != cudaSuccess) return e;
    std::memset(h_tab_, 0, sizeof(KTable));   // plans are rebuilt on the device below
    h_tab_->B = B;
    h_tab_->prec = prec_;
    h_tab_->vb_total = vb_total;
    h_tab_->vb_items = d_items_;
    h_tab_->wait_cycles = test_wait_cycles();
    h_tab_->wait_kinds = test_wait_kinds();
    for (int b = 0; b < B; ++b) {
        h_tab_->sys[b] = sys[b];
        h_tab_->sys[b].st = d_st_ + b;
        h_tab_->sys[b].shared = 0;
        h_tab_->pcw_any |= sys[b].pcw;
        h_st_[b] = init[b];
    }
    // complex64 systems next to each other on the same matrix (the right-hand
    // sides of one solver) form groups whose products share each read of A
    int ng = 0;
    for (int b = 0; b < B && prec_ == 1;) {
        int e = b + 1;
        while (e < B && e - b < kMaxGroup && sys[e].A == sys[b].A) ++e;
        if (e - b >= 2) {
            h_tab_->grp[ng].first = b;
            h_tab_->grp[ng].count = e - b;
            ++ng;
            for (int q = b; q < e; ++q) {
                h_tab_->sys[q].shared = 1;
                h_tab_->sys[q].nchunk = 1;   // the group product writes full rows
            }
        }
        b = e;
    }
    h_tab_->n_groups = ng;
    groups_ = ng;
    blr_ = 0;
    dense_ = 0;
    for (int b = 0; b < B; ++b) {
        if (h_tab_->sys[b].shared) continue;
        if (h_tab_->sys[b].blr_nb > 0) ++blr_;
        else ++dense_;
    }
    // the groups' Krylov products on the 5th-generation tensor cores need a
    // TMA map of each group's matrix; without them the warp-level kernel runs
    bool umma = ng > 0 && group_product_umma();
    for (int q = 0; q < ng && umma; ++q) {
        const KSys &g0 = h_tab_->sys[h_tab_->grp[q].first];
        umma = encode_group_map(&h_tab_->gmap[q], g0.A, g0.n, g0.lda);
    }
    h_tab_->grp_umma = umma ? 1 : 0;
    e = cudaMemcpyAsync(d_tab_, h_tab_, sizeof(KTable), cudaMemcpyHostToDevice, st_);
    if (e == cudaSuccess && B > 0)
        e = cudaMemcpyAsync(d_st_, h_st_, sizeof(KState) * B, cudaMemcpyHostToDevice, st_);
    // systems may be in the middle of a cycle: their next products need plans
    if (e == cudaSuccess) e = launch_plans(d_tab_, st_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    B_ = B;
    rate_.assign(B, 0.0);
    bodies_ = 0;
    return e;
}

cudaError_t Engine::time_product(const KSys &sys, float *ms) {
    cudaError_t e = ensure_init();
    if (e != cudaSuccess) return e;
    std::memset(h_tab_, 0, sizeof(KTable));
    h_tab_->B = 1;
    h_tab_->prec = prec_;
    h_tab_->vb_total = sys.nvb;
    h_tab_->wait_cycles = test_wait_cycles();
    h_tab_->wait_kinds = test_wait_kinds();
    h_tab_->sys[0] = sys;
    h_tab_->sys[0].st = d_st_;
    h_tab_->sys[0].shared = 0;
    const int strip = sys.strip > 0 ? sys.strip : kTmaStrip;
    KPlan &p = h_tab_->plan[0];
    p.n = 1;
    p.sys[0] = 0;
    p.off[0] = 0;
    p.off[1] = sys.A16 ? mv_items16(sys.n, strip) : mv_items_of(sys.n, prec_, strip);
    e = cudaMemcpyAsync(d_tab_, h_tab_, sizeof(KTable), cudaMemcpyHostToDevice, st_);
    float best = 1e30f;
    for (int rep = 0; rep < 3 && e == cudaSuccess; ++rep) {
        e = cudaEventRecord(ev_[0], st_);
        if (e == cudaSuccess) e = launch_product(d_tab_, prec_, st_);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[1], st_);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev_[1]);
        float t = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t, ev_[0], ev_[1]);
        if (e == cudaSuccess && rep > 0 && t < best) best = t;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h_tab_->err, &d_tab_->err, sizeof(int), cudaMemcpyDeviceToHost, st_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    if (e == cudaSuccess && h_tab_->err) e = cudaErrorLaunchTimeout;
    count_launches(3);
    *ms = best;
    B_ = 0;   // the table no longer holds a batch
    return e;
}

cudaError_t Engine::capture(int part, int v) {
    if (exec_[part][v]) return cudaSuccess;
    const bool groups = v & 1, blr = v & 2, dense = v & 4;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    const cudaError_t le =
        part == 0 ? launch_krylov_step(prec_, d_tab_, st_, &launches_[0][v], groups, blr, dense, side_)
                  : launch_krylov_cycle_end(prec_, d_tab_, st_, &launches_[1][v], groups, blr, dense);
    e = cudaStreamEndCapture(st_, &g);
    if (le != cudaSuccess) e = le;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec_[part][v], g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) exec_[part][v] = nullptr;
    return e;
}

// Arnoldi steps of the next body: what the system furthest from the end of its
// cycle is expected to need (at the rate of its cycle so far, or of its last
// one; kSteps without either), at most kSteps, none before the first residual.
// A step too many is some ten empty launches (1280 triangles: 16 us), one too
// few an empty end of cycle and a wait for the host (40 us), hence the half
// step on top.  The number changes when a cycle's end is seen, not its result.
int Engine::steps_ahead() const {
    int most = 0;
    for (int b = 0; b < B_; ++b) {
        const KState &q = h_st_[b];
        if (q.phase != kPhaseArnoldi) continue;
        const double from = q.k > 0 ? q.res : q.beta, rate = q.k > 0 ? std::log(q.beta / q.res) / q.k : rate_[b];
        const double need = std::log(from / q.thr) / rate + 0.5;
        int s = kSteps;
        if (rate > 0.0 && need < kSteps) s = need > 1.0 ? (int)std::ceil(need) : 1;
        most = std::max(most, std::min(s, q.m - q.k));
    }
    return std::min(most, kSteps);
}

cudaError_t Engine::run_body() {
    cudaError_t e = ensure_init();
    if (e != cudaSuccess) return e;
    const int v = (groups_ > 0 ? 1 : 0) | (blr_ > 0 ? 2 : 0) | (dense_ > 0 ? 4 : 0);
    const int steps = steps_ahead();
    if (steps > 0) e = capture(0, v);
    if (e == cudaSuccess) e = capture(1, v);
    for (int q = 0; q < steps && e == cudaSuccess; ++q) e = cudaGraphLaunch(exec_[0][v], st_);
    if (e == cudaSuccess) e = cudaGraphLaunch(exec_[1][v], st_);
    std::vector<KState> was(h_st_, h_st_ + B_);
    if (e == cudaSuccess && B_ > 0)
        e = cudaMemcpyAsync(h_st_, d_st_, sizeof(KState) * B_, cudaMemcpyDeviceToHost, st_);
    if (e == cudaSuccess)   // err and mv_ns
        e = cudaMemcpyAsync(&h_tab_->err, &d_tab_->err, offsetof(KTable, mv_t0) - offsetof(KTable, err),
                            cudaMemcpyDeviceToHost, st_);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    if (e != cudaSuccess) return e;
    if (h_tab_->err) return cudaErrorLaunchTimeout;   // a bounded wait in the product gave up
    count_launches(steps * launches_[0][v] + launches_[1][v]);
    for (int b = 0; b < B_; ++b) {   // the rate of a cycle that ended
        const KState &q = h_st_[b];
        const int len = q.iters - (was[b].iters - was[b].k);
        if (q.cycles > was[b].cycles && len > 0) rate_[b] = std::log(q.prev_beta / q.res) / len;
    }
    ++bodies_;
    return cudaSuccess;
}

}  // namespace bem
