// Host side of the cuda MPS backend: the C ABI of include/wqc_cuda.h.
//
// A gate list is expanded into the reference's MpsState operations (one-qubit
// applies and adjacent two-site splits, with SWAP routing and the CCNOT
// decomposition of src/tn/mps.rs:353-375, 657-677), scheduled into levels so
// that splits on disjoint sites share a wave, and enqueued on the state's
// stream without waiting for the device.  Bond dimensions live on the device;
// the host only tracks upper bounds to size launches.
#include <cuda_runtime.h>

#include <sys/stat.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/wqc_cuda.h"
#include "common.cuh"
#include "scratch.h"
#include "split_kernels.cuh"
#include "tc_gemm.cuh"
#include "tile_gemm.cuh"

using namespace wqc;

namespace {

thread_local std::string g_err;
// Byte counts of the last WQC_ERR_OOM on this thread, for
// EngineError::InsufficientMemory { required, available } (src/engine.rs:72).
thread_local uint64_t g_oom_required = 0, g_oom_available = 0;

wqc_status fail(wqc_status code, const std::string& msg) {
    g_err = msg;
    return code;
}

wqc_status fail_oom(uint64_t required, uint64_t available) {
    g_oom_required = required;
    g_oom_available = available;
    return fail(WQC_ERR_OOM, "Insufficient memory: need " + std::to_string(required) + " bytes, only " +
                                 std::to_string(available) + " bytes free on the device");
}

// The error state of the thread, put back by a call that made do without what
// it was refused.
struct ErrorState {
    std::string err = g_err;
    uint64_t required = g_oom_required, available = g_oom_available;
    void restore() const {
        g_err = err;
        g_oom_required = required;
        g_oom_available = available;
    }
};

#define CUDA_TRY(expr)                                                                                    \
    do {                                                                                                  \
        cudaError_t e_ = (expr);                                                                          \
        if (e_ != cudaSuccess) return fail(WQC_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

constexpr int kMaxSweeps = 60;
constexpr int kOzAutoBond = 192;  // default merges take int8 digit slices above this bond
constexpr int kDenseMaxQubits = 28;  // 2^28 complex128 = 4 GiB on the host
constexpr size_t kSlotBudget = size_t(1) << 30;  // split workspace per chi_max bucket
constexpr size_t kSmemLimit = 232448 - 1024;  // 227 KB opt-in per block, minus static shared memory

struct Mat2 {
    double2 u[4];  // row-major
};
struct Mat4 {
    double2 u[16];  // [c_out][t_out][c_in][t_in] flattened: ((co*2+to)*2+ci)*2+ti
};

double2 C(double r, double i = 0.0) { return make_double2(r, i); }

// src/tn/gates.rs:10-66 and mps.rs:1173-1180.
Mat2 unary_matrix(int kind, double theta) {
    const double r2 = 0.70710678118654752440;
    switch (kind) {
        case WQC_GATE_H: {
            const double k = 1.0 / std::sqrt(2.0);
            return {{C(k), C(k), C(k), C(-k)}};
        }
        case WQC_GATE_X: return {{C(0), C(1), C(1), C(0)}};
        case WQC_GATE_Y: return {{C(0), C(0, -1), C(0, 1), C(0)}};
        case WQC_GATE_Z: return {{C(1), C(0), C(0), C(-1)}};
        case WQC_GATE_S: return {{C(1), C(0), C(0), C(0, 1)}};
        case WQC_GATE_T: return {{C(1), C(0), C(0), C(r2, r2)}};
        case WQC_GATE_RX: {
            const double s = std::sin(theta / 2.0), c = std::cos(theta / 2.0);
            return {{C(c), C(0, -s), C(0, -s), C(c)}};
        }
        case WQC_GATE_RY: {
            const double s = std::sin(theta / 2.0), c = std::cos(theta / 2.0);
            return {{C(c), C(-s), C(s), C(c)}};
        }
        default: {  // RZ
            const double s = std::sin(theta / 2.0), c = std::cos(theta / 2.0);
            return {{C(c, -s), C(0), C(0), C(c, s)}};
        }
    }
}
Mat2 tdg_matrix() {
    const double r2 = 0.70710678118654752440;
    return {{C(1), C(0), C(0), C(r2, -r2)}};
}
int i4(int co, int to, int ci, int ti) { return ((co * 2 + to) * 2 + ci) * 2 + ti; }
Mat4 cnot_matrix() {
    Mat4 m{};
    m.u[i4(0, 0, 0, 0)] = C(1);
    m.u[i4(0, 1, 0, 1)] = C(1);
    m.u[i4(1, 0, 1, 1)] = C(1);
    m.u[i4(1, 1, 1, 0)] = C(1);
    return m;
}
Mat4 cz_matrix() {
    Mat4 m{};
    m.u[i4(0, 0, 0, 0)] = C(1);
    m.u[i4(0, 1, 0, 1)] = C(1);
    m.u[i4(1, 0, 1, 0)] = C(1);
    m.u[i4(1, 1, 1, 1)] = C(-1);
    return m;
}
Mat4 swap_matrix() {
    Mat4 m{};
    m.u[i4(0, 0, 0, 0)] = C(1);
    m.u[i4(0, 1, 1, 0)] = C(1);
    m.u[i4(1, 0, 0, 1)] = C(1);
    m.u[i4(1, 1, 1, 1)] = C(1);
    return m;
}
Mat2 adjoint2(const Mat2& a) {
    return {{make_double2(a.u[0].x, -a.u[0].y), make_double2(a.u[2].x, -a.u[2].y),
             make_double2(a.u[1].x, -a.u[1].y), make_double2(a.u[3].x, -a.u[3].y)}};
}
Mat4 adjoint4(const Mat4& a) {
    Mat4 o{};
    for (int co = 0; co < 2; ++co)
        for (int to = 0; to < 2; ++to)
            for (int ci = 0; ci < 2; ++ci)
                for (int ti = 0; ti < 2; ++ti) {
                    const double2 v = a.u[i4(ci, ti, co, to)];
                    o.u[i4(co, to, ci, ti)] = make_double2(v.x, -v.y);
                }
    return o;
}

// Effective 4x4 acting on theta[a][s][t][b] (mps.rs:396-421, split.rs:808-831).
void effective(const Mat4& u, bool ctrl_is_first, double2* out) {
    for (int so = 0; so < 2; ++so)
        for (int to = 0; to < 2; ++to)
            for (int si = 0; si < 2; ++si)
                for (int ti = 0; ti < 2; ++ti) {
                    const int co = ctrl_is_first ? so : to, tgo = ctrl_is_first ? to : so;
                    const int ci = ctrl_is_first ? si : ti, tgi = ctrl_is_first ? ti : si;
                    out[(so * 2 + to) * 4 + si * 2 + ti] = u.u[i4(co, tgo, ci, tgi)];
                }
}

struct Op {
    bool two;
    int site;        // 1q: site; 2q: left site (global site index)
    int slice = 0;   // batch slice the operation belongs to
    int gate = -1;   // index of the gate (in the caller's list) this operation comes from
    Mat2 m2;
    double2 ueff[16];
};

// Launch shape of one Jacobi phase for a group of jobs.
struct PhaseCfg {
    int C = 0;            // cluster size (the largest of the group's tasks)
    size_t smem = 0;
    int threads = 0;      // one warp per column of a block
    bool staged = false;  // jacobi_staged_kernel with blocks of b columns
    int kr = 0;           // row groups of the cluster Jacobi's instance
    int b = 0;
    int idx_off = 0;      // task list
};

// Jobs of one wave whose SVDs share launch shapes: one phase in the plain
// form; the complex64 first phase and the FP64 finish in the precision form.
struct Group {
    int mode, count;
    int nph = 1;
    int qr_kr = 0, qr_C = 0;  // QR before the first phase (0: none of the tasks takes one)
    PhaseCfg ph[2];
};

struct Wave {
    int oq_off = 0, oq_count = 0;  // OneQubitOp entries
    int jobs_off = 0, njobs = 0;   // SplitJob entries
    int max_dl = 1, max_dr = 1, max_rows = 2, max_cols = 2, max_ell = 1;
    bool any_rsvd = false;
    std::vector<Group> groups;
};

struct Arena {
    void* d = nullptr;
    size_t cap = 0;
};

}  // namespace

struct wqc_cuda_ctx {
    int device = 0;
    int sm_count = 0;
    int max_cluster = 8;
    std::mutex mu;
    // Jacobi cluster sizes measured by wqc_cuda_autotune, by working-matrix
    // shape (M x N, rows stored per column, bytes per complex entry) and by
    // kind of wave (one latency-bound split, or a throughput-bound batch).
    struct Tuned {
        int M, N, len, elem, throughput, C;
    };
    std::vector<Tuned> tuned;
    int force_C = 0;  // set by the tuner while it measures one cluster size
};

struct wqc_mps {
    wqc_cuda_ctx* ctx = nullptr;
    int n = 0, chi = 0;
    bool reject = false;
    bool exact_only = false;  // WQC_SPLIT_RULE_EXACT
    // No QR before the Jacobi (set while an adjoint runs): the derivative
    // divides by differences of squared singular values, and on a graded theta
    // the vectors of the small ones are more exact from a Jacobi on theta
    // itself (gradient of the 32-qubit ansatz against 64-bit autograd: 3.7e-7
    // with the QR where 4.7e-8 without).
    bool direct_svd = false;
    bool fp32 = false;        // WQC_PRECISION_FP32 or _TF32X3: complex64 Jacobi columns
    // WQC_PRECISION_TF32X3: merges on the tensor cores (tc_gemm.cu), their
    // operands staged per wave job as TF32 hi/lo planes under two tensor maps
    bool tc = false;
    float* tc_a = nullptr;
    float* tc_b = nullptr;
    int tc_rpad = 0, tc_npad = 0, tc_kpad = 0;
    CUtensorMap tc_map_a{}, tc_map_b{};
    // WQC_MERGE_TC_INT8 (wqc_mps_set_merge): merges from int8 digit slices
    // on the tensor cores (tc_ozaki.cu), staged per wave job
    bool oz = false;
    bool oz_auto = false;  // the default: by size, until wqc_mps_set_merge says which
    void* oz_pool = nullptr;
    size_t oz_bytes = 0;
    OzPlanes oz_planes;
    bool batch = false;       // made by wqc_batch_create: Jacobi clusters sized for throughput
    cudaStream_t stream = nullptr;
    // Second stream of a wave: the exact-path SVDs run there while the range
    // finder runs on `stream`; fork after the merge, join before the absorb.
    cudaStream_t side = nullptr;
    cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
    // device state
    double2* site_pool = nullptr;
    std::vector<double2*> site_ptr;  // device address of every site (capacity chi_slice * 2 * chi_slice)
    DeviceMps dev{};
    double2** d_site_ptr = nullptr;
    int* d_dl = nullptr;
    int* d_dr = nullptr;
    int* d_status = nullptr;
    volatile int* h_cancel = nullptr;  // mapped pinned
    int* d_cancel = nullptr;
    // split workspace
    int nslots = 0;
    // Slots come in buckets, one per distinct chi_max of the slices, each
    // slot sized for its bucket's largest two-site matrix (R = 2 chi_max).
    std::vector<int> bucket_chi, bucket_base, bucket_cap;
    std::vector<int> slot_R, slot_E;
    int bucket_of(int chi) const {
        for (size_t b = 0; b < bucket_chi.size(); ++b)
            if (bucket_chi[b] == chi) return int(b);
        return 0;
    }
    char* slot_pool = nullptr;
    SlotBuffers* d_slots = nullptr;
    SplitState* d_state = nullptr;
    // per-call plan
    char* h_stage = nullptr;
    size_t h_stage_cap = 0;
    cudaEvent_t stage_done = nullptr;
    Arena d_stage;
    wqc_split_info* d_records = nullptr;
    size_t rec_cap = 0;
    uint32_t rec_count = 0;
    double2* d_small = nullptr;  // results of amplitude / site kernels
    unsigned long long* d_counters = nullptr;  // Jacobi tasks, Jacobi sweeps
    // host bounds: ub[i] = upper bound of the bond between sites i and i+1
    std::vector<int> ub;
    // slices: a single state is one slice; a batch concatenates its slices'
    // sites, and no split ever crosses a slice boundary
    std::vector<int> seg_first, seg_n, seg_chi;
    std::vector<int> site_chi, site_slice;
    int* d_seg = nullptr;  // (first, count) per slice for the amplitude kernel
    // per-slice completion times of the last call (batch, profiling on)
    std::vector<int> slice_last_wave;
    std::vector<cudaEvent_t> wave_done;
    cudaEvent_t call_start = nullptr;
    // Cached environments of the trace feeders (single states): L_0..L_lvalid
    // and R_rvalid..R_{n-1} are current; an operation on sites [a, b] leaves
    // lvalid <= a and rvalid >= b.
    double2* d_envL = nullptr;
    double2* d_envR = nullptr;
    int* d_targets = nullptr;     // targets of one wqc_mps_site_amplitudes_many call
    double2* d_env_out = nullptr; // its (a0, a1) pairs
    int lvalid = 0, rvalid = 0;
    void touch(int a, int b) {
        lvalid = std::min(lvalid, a);
        rvalid = std::max(rvalid, b);
    }
    // Set by wqc_mps_upload_site: the bonds of the chain are checked once
    // before the next call that computes on it.
    bool uploaded = false;
    // accounting
    uint64_t bytes_now = 0, bytes_peak = 0;
    uint64_t bytes_limit = ~uint64_t(0);  // wqc_mps_debug_limit_bytes
    int device = -1;                      // counted among its states (scratch.h); the context may close first
    bool profiling = false;
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> events;
    std::vector<cudaEvent_t> event_pool;
    wqc_kernel_stats stats{};

    int left_bond(int site) const { return site == 0 ? 1 : ub[site - 1]; }
    int right_bond(int site) const { return site + 1 >= n ? 1 : ub[site]; }
};

namespace {

wqc_status dmalloc(wqc_mps* m, void** p, size_t bytes);

// Digit planes of the int8-slice merges for every split slot of the state.
size_t oz_state_bytes(const wqc_mps* m) {
    return oz_planes_bytes(m->nslots, oz_rpad(2 * m->chi), oz_npad(2 * m->chi), oz_kpad(m->chi));
}

}  // namespace

// Merges from int8 digit slices from now on: allocate the digit planes of
// every split slot the first time (WQC_ERR_OOM if they do not fit).
static wqc_status oz_enable(wqc_mps* m) {
    if (!m->oz_pool) {
        const int rpad = oz_rpad(2 * m->chi), npad = oz_npad(2 * m->chi), kpad = oz_kpad(m->chi);
        const size_t bytes = oz_state_bytes(m);
        size_t fr = 0;
        if (device_room(bytes, &fr) != cudaSuccess) return fail(WQC_ERR_CUDA, "cudaMemGetInfo");
        if (bytes > fr) return fail_oom(bytes, fr);
        void* p = nullptr;
        if (wqc_status st = dmalloc(m, &p, bytes)) return st;
        if (!oz_planes_init(&m->oz_planes, p, m->nslots, rpad, npad, kpad)) {
            cudaFree(p);
            m->bytes_now -= bytes;
            return fail(WQC_ERR_CUDA, "cuTensorMapEncodeTiled refused the merge digit planes");
        }
        m->oz_pool = p;
        m->oz_bytes = bytes;
    }
    m->oz = true;
    return WQC_OK;
}

namespace {

wqc_status dmalloc(wqc_mps* m, void** p, size_t bytes) {
    if (m->bytes_now + bytes > m->bytes_limit)
        return fail_oom(bytes, m->bytes_limit > m->bytes_now ? m->bytes_limit - m->bytes_now : 0);
    cudaError_t e = device_malloc(p, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        return fail_oom(bytes, fr);
    }
    m->bytes_now += bytes;
    m->bytes_peak = std::max(m->bytes_peak, m->bytes_now);
    return WQC_OK;
}
void dfree(wqc_mps* m, void* p, size_t bytes) {
    if (!p) return;
    cudaFree(p);
    m->bytes_now -= bytes;
}

// Device memory of one read, from the device's pool; back there once the
// state's stream has drained, whichever way the call ends.
struct Scratch {
    wqc_mps* m;
    void* p = nullptr;
    size_t cap = 0;
    bool drained = false;  // set by a call that has synchronised after its last use
    explicit Scratch(wqc_mps* mm) : m(mm) {}
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch() {
        if (!p) return;
        if (!drained) cudaStreamSynchronize(m->stream);
        m->bytes_now -= cap;
        scratch_give(m->device, p, cap);
    }
    wqc_status get(size_t bytes) {
        if (m->bytes_now + bytes <= m->bytes_limit) p = scratch_take(m->device, bytes, &cap);
        if (!p) {
            void* q = nullptr;
            if (wqc_status s = dmalloc(m, &q, bytes)) return s;
            p = q;
            cap = bytes;
            return WQC_OK;
        }
        m->bytes_now += cap;
        m->bytes_peak = std::max(m->bytes_peak, m->bytes_now);
        return WQC_OK;
    }
};

std::once_flag g_attr_once;
cudaError_t g_attr_err = cudaSuccess;

void set_kernel_attributes() {
    std::vector<const void*> jacobi = jacobi_ring_kernels();
    jacobi.push_back(jacobi_staged(false));
    jacobi.push_back(jacobi_staged(true));
    for (const void* f : jacobi) {
        if (g_attr_err == cudaSuccess)
            g_attr_err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit));
        if (g_attr_err == cudaSuccess)
            g_attr_err = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    if (g_attr_err == cudaSuccess) g_attr_err = jacobi_qr_attributes();
    for (const void* f : {qr_cluster(false), qr_cluster(true)}) {
        if (g_attr_err == cudaSuccess)
            g_attr_err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit));
        if (g_attr_err == cudaSuccess)
            g_attr_err = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    if (g_attr_err == cudaSuccess)
        g_attr_err = cudaFuncSetAttribute(amplitude_zero_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
}

// Launch shape of a cluster Jacobi task: C CTAs (a power of two), blocks of b
// columns, kr row groups.
struct RingShape {
    int C = 0, b = 0, kr = 0, warps = 0;
    size_t smem = 0;
};

// The shape of an M x N working matrix (with vrows rows of V under it) on C
// CTAs; false when it does not fit.  A block of odd width takes one warp more,
// for the pairs inside the blocks.
bool ring_shape(int M, int N, int vrows, size_t elem, int C, RingShape* out) {
    const bool fp32 = elem == sizeof(float2);
    RingShape s;
    s.C = C;
    s.b = (N + 2 * C - 1) / (2 * C);
    s.kr = jacobi_ring_kr(fp32, M, vrows);
    if (s.kr == 0) return false;
    s.warps = s.b + (s.b & 1);
    s.smem = jacobi_ring_smem(s.b, s.kr, elem);
    if (s.warps > jacobi_ring_warps(s.kr, int(elem)) || s.smem > kSmemLimit) return false;
    *out = s;
    return true;
}

// Cluster size of a Jacobi task.  A sweep is (2C - 1) b + b rounds of rotation
// (about N whatever C is) and 2C - 1 block moves with a cluster barrier.  A
// round costs its dependent chain (850 cycles) and, as the block's warps go
// through it in step, the FP64 pipe's time for all of them (50 instructions a
// column and 20 per row group) and their shared-memory traffic; constants
// fitted to single SVDs of 8 to 384 columns on every cluster size (64
// columns: 1080 cycles a round at b = 4, 1222 at 8, 1620 at 16).  A single
// state is latency-bound (a few splits per level) and takes the shortest
// sweep, until the wave's clusters would fill the GPU, from where SM time
// counts.  A batch fills the GPU, so SM time decides, with as many CTAs on an
// SM as fit it, but never less than the FP64 work; that choice depends on the
// shape alone, so a slice's results do not depend on the other slices of its
// batch.  `most_warps` bounds the CTA of a task that shares a launch with
// longer columns, whose instance is compiled for fewer warps.  0: no cluster
// size fits.
int choose_cluster(const wqc_cuda_ctx* ctx, int M, int N, int max_c, int njobs, int sm_count, size_t elem,
                   bool throughput, int vrows = 0, int most_warps = 32) {
    RingShape s;
    auto shaped = [&](int Cc) { return ring_shape(M, N, vrows, elem, Cc, &s) && s.warps <= most_warps; };
    if (ctx) {
        auto fits = [&](int Cc) { return Cc >= 1 && Cc <= max_c && !(Cc & (Cc - 1)) && shaped(Cc); };
        if (ctx->force_C > 0 && fits(ctx->force_C)) return ctx->force_C;
        for (const auto& t : ctx->tuned)
            if (t.M == M && t.N == N && t.len == M + vrows && t.elem == int(elem) &&
                t.throughput == int(throughput) && fits(t.C))
                return t.C;
    }
    int best = 0;
    double best_cost = 1e300;
    for (int Cc = 1; Cc <= std::min(max_c, kJacobiRingMaxCluster); Cc *= 2) {
        if (!shaped(Cc)) continue;
        const double kr = s.kr * double(elem) / sizeof(double2);
        const double work = s.b * (25.0 + 10.0 * kr);  // FP64 pipe cycles of a round
        const double round = 850.0 + work + 0.6 * kr * kr * s.b;
        const double rounds = 2.0 * Cc * s.b;
        const double moves = Cc > 1 ? (2 * Cc - 1) * 700.0 + 2500.0 : 0.0;
        double cost = rounds * round + moves;
        if (throughput) {
            const int by_threads = 2048 / (32 * s.warps), by_smem = int(kSmemLimit / s.smem);
            const int by_regs = 65536 / (32 * s.warps * std::min(255, 2 * s.kr * int(elem) / 4 + 48));
            const int ctas = std::max(1, std::min(std::min(by_threads, by_smem), by_regs));
            cost = Cc * std::max(cost / ctas, rounds * work);
        } else if (double(njobs) * Cc >= 1.5 * sm_count) {
            cost *= Cc;
        }
        if (cost < best_cost) {
            best_cost = cost;
            best = Cc;
        }
    }
    return best;
}

cudaEvent_t get_event(wqc_mps* m) {
    if (!m->event_pool.empty()) {
        cudaEvent_t e = m->event_pool.back();
        m->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

struct Timed {
    wqc_mps* m;
    int kind;
    cudaEvent_t a = nullptr, b = nullptr;
    cudaStream_t s;
    Timed(wqc_mps* mm, int k, cudaStream_t on = nullptr) : m(mm), kind(k), s(on ? on : mm->stream) {
        if (m->profiling) {
            a = get_event(m);
            b = get_event(m);
            cudaEventRecord(a, s);
        }
    }
    ~Timed() {
        if (m->profiling) {
            cudaEventRecord(b, s);
            m->events.push_back({kind, {a, b}});
        }
    }
};

void count_launch(wqc_mps* m, int kind) {
    m->stats.total_launches++;
    if (kind >= 0) m->stats.launches[kind]++;
}

// ---------------------------------------------------------------------------
// Expansion of gates into MpsState operations.
// ---------------------------------------------------------------------------
struct Expander {
    std::vector<Op> ops;
    int cur = -1;  // gate being expanded
    void one(int q, const Mat2& u) {
        Op o{};
        o.two = false;
        o.site = q;
        o.m2 = u;
        o.gate = cur;
        ops.push_back(o);
    }
    void two_at(int p, const Mat4& u, bool cf) {
        Op o{};
        o.two = true;
        o.site = p;
        o.gate = cur;
        effective(u, cf, o.ueff);
        ops.push_back(o);
    }
    void two_routed(int ctrl, int tgt, const Mat4& u) {  // mps.rs:353-375
        const int left = std::min(ctrl, tgt), right = std::max(ctrl, tgt);
        const int span = right - left;
        const Mat4 sw = swap_matrix();
        if (span > 1)
            for (int pos = right - 1; pos >= left + 1; --pos) two_at(pos, sw, true);
        two_at(left, u, ctrl < tgt);
        if (span > 1)
            for (int pos = left + 1; pos < right; ++pos) two_at(pos, sw, true);
    }
    void ccnot(int c1, int c2, int t) {  // mps.rs:657-677
        const Mat2 tdg = tdg_matrix(), h = unary_matrix(WQC_GATE_H, 0), tt = unary_matrix(WQC_GATE_T, 0);
        const Mat4 cx = cnot_matrix();
        one(t, h);
        two_routed(c2, t, cx);
        one(t, tdg);
        two_routed(c1, t, cx);
        one(t, tt);
        two_routed(c2, t, cx);
        one(t, tdg);
        two_routed(c1, t, cx);
        one(t, tt);
        one(t, h);
        one(c2, tt);
        two_routed(c1, c2, cx);
        one(c1, tt);
        one(c2, tdg);
        two_routed(c1, c2, cx);
    }
};

wqc_status check_gate(int n, const wqc_gate& g) {
    auto chk = [&](int q) -> wqc_status {
        if (q < 0 || q >= n)
            return fail(WQC_ERR_QUBIT_OUT_OF_RANGE,
                        "Qubit index " + std::to_string(q) + " out of bounds (limit: " + std::to_string(n) + ")");
        return WQC_OK;
    };
    wqc_status s = WQC_OK;
    switch (g.kind) {
        case WQC_GATE_H: case WQC_GATE_X: case WQC_GATE_Y: case WQC_GATE_Z: case WQC_GATE_S: case WQC_GATE_T:
        case WQC_GATE_RX: case WQC_GATE_RY: case WQC_GATE_RZ:
            return chk(g.q0);
        case WQC_GATE_CNOT: case WQC_GATE_CZ:
            if ((s = chk(g.q0)) || (s = chk(g.q1))) return s;
            if (g.q0 == g.q1) return fail(WQC_ERR_INVALID, "two-qubit gate on one qubit");
            return WQC_OK;
        case WQC_GATE_CCNOT:
            if ((s = chk(g.q0)) || (s = chk(g.q1)) || (s = chk(g.q2))) return s;
            if (g.q0 == g.q1 || g.q0 == g.q2 || g.q1 == g.q2) return fail(WQC_ERR_INVALID, "CCNOT needs three qubits");
            return WQC_OK;
        case WQC_GATE_MEASURE: case WQC_GATE_RESET: case WQC_GATE_IF:
            return WQC_OK;
        default:
            return fail(WQC_ERR_INVALID, "unknown gate kind " + std::to_string(g.kind));
    }
}

wqc_status expand(int n, const wqc_gate* gates, uint32_t count, bool adjoint, Expander& ex) {
    for (uint32_t i = 0; i < count; ++i) {
        const wqc_gate& g = gates[adjoint ? count - 1 - i : i];
        ex.cur = int(adjoint ? count - 1 - i : i);
        if (wqc_status s = check_gate(n, g)) return s;
        switch (g.kind) {
            case WQC_GATE_CNOT:
                ex.two_routed(g.q0, g.q1, adjoint ? adjoint4(cnot_matrix()) : cnot_matrix());
                break;
            case WQC_GATE_CZ:
                ex.two_routed(g.q0, g.q1, adjoint ? adjoint4(cz_matrix()) : cz_matrix());
                break;
            case WQC_GATE_CCNOT:
                ex.ccnot(g.q0, g.q1, g.q2);
                break;
            case WQC_GATE_MEASURE: case WQC_GATE_RESET: case WQC_GATE_IF:
                if (adjoint) return fail(WQC_ERR_INVALID, "time-split overlap does not apply measurement or reset");
                break;
            default: {
                const Mat2 u = unary_matrix(g.kind, g.angle);
                ex.one(g.q0, adjoint ? adjoint2(u) : u);
                break;
            }
        }
    }
    return WQC_OK;
}

// ---------------------------------------------------------------------------
// Plan: levels -> waves, staged in one pinned buffer and copied once.
// ---------------------------------------------------------------------------
struct Plan {
    std::vector<Wave> waves;
    std::vector<OneQubitOp> oq;
    std::vector<double2> mats;
    std::vector<SplitJob> jobs;
    std::vector<int> idx;
    std::vector<int> slice_last_wave;  // last wave holding an operation of each slice
    uint32_t first_seq = 0, nsplits = 0;
};

// Level of every operation: a split on (p, p+1) goes one level after the last
// split that touched p or p+1; a one-qubit gate goes one level after the last
// split on its site and runs before that level's splits.  Each site therefore
// sees its operations in program order, and the splits of one level touch
// disjoint sites.
void assign_levels(int n, const std::vector<Op>& ops, std::vector<int>& level_of) {
    std::vector<int> last2q(n, -1);
    level_of.resize(ops.size());
    for (size_t i = 0; i < ops.size(); ++i) {
        const Op& o = ops[i];
        if (!o.two) {
            level_of[i] = last2q[o.site] + 1;
        } else {
            const int L = std::max(last2q[o.site], last2q[o.site + 1]) + 1;
            level_of[i] = L;
            last2q[o.site] = last2q[o.site + 1] = L;
        }
    }
}

void build_plan(wqc_mps* m, const std::vector<Op>& ops, Plan& plan) {
    struct LevelBuild {
        std::vector<std::pair<int, std::vector<Mat2>>> oq;  // site -> matrices in order
        std::vector<int> oq_index;                          // site -> entry in oq (built lazily)
        std::vector<SplitJob> jobs;
        std::vector<std::pair<int, int>> bounds;  // (ub left of p, ub right of p+1) at the job
        std::vector<int> job_slice;
        std::vector<int> oq_slices;
    };
    std::vector<LevelBuild> levels;
    std::vector<int> level_of;
    assign_levels(m->n, ops, level_of);
    auto level = [&](int L) -> LevelBuild& {
        while (int(levels.size()) <= L) levels.emplace_back();
        return levels[L];
    };
    uint32_t seq = m->rec_count;
    plan.first_seq = seq;
    for (size_t oi = 0; oi < ops.size(); ++oi) {
        const Op& o = ops[oi];
        m->touch(o.site, o.two ? o.site + 1 : o.site);
        if (!o.two) {
            LevelBuild& lb = level(level_of[oi]);
            if (lb.oq_index.empty()) lb.oq_index.assign(m->n, -1);
            int& e = lb.oq_index[o.site];
            if (e < 0) {
                e = int(lb.oq.size());
                lb.oq.push_back({o.site, {}});
                lb.oq_slices.push_back(o.slice);
            }
            lb.oq[e].second.push_back(o.m2);
        } else {
            const int p = o.site;
            LevelBuild& lb = level(level_of[oi]);
            SplitJob J{};
            J.p = p;
            J.seq = int(seq++);
            J.reject = m->reject ? 1 : 0;
            J.exact_only = m->exact_only ? 1 : 0;
            J.chi_max = m->site_chi[p];
            std::memcpy(J.u, o.ueff, sizeof(J.u));
            const int bl = m->left_bond(p), br = m->right_bond(p + 1);
            lb.jobs.push_back(J);
            lb.bounds.push_back({bl, br});
            lb.job_slice.push_back(o.slice);
            m->ub[p] = std::min(std::min(2 * bl, 2 * br), J.chi_max);
        }
    }
    plan.nsplits = seq - plan.first_seq;
    plan.slice_last_wave.assign(m->seg_first.size(), -1);
    struct WaveTask {
        int mode, M, N, local;
    };
    std::vector<WaveTask> wave_tasks;
    std::vector<std::array<int, 2>> sizes;
    // A plan holds few shapes many times over: the cluster sizes last worked
    // out, by shape and (outside batches, where it counts) the wave's splits.
    // M, N and V's rows are at most 512, warps 32 and splits 2^24.
    struct KnownCluster {
        uint64_t key = 0;
        int C = 0;
    };
    std::array<KnownCluster, 256> known_clusters;
    for (LevelBuild& lb : levels) {
        // one-qubit ops run first, in one wave with no splits when needed
        std::vector<char> taken(lb.jobs.size(), 0);
        size_t remaining = lb.jobs.size();
        bool first = true;
        do {
            Wave w;
            const int wave_index = int(plan.waves.size());
            if (first) {
                w.oq_off = int(plan.oq.size());
                for (auto& e : lb.oq) {
                    OneQubitOp op;
                    op.site = e.first;
                    op.first = int(plan.mats.size() / 4);
                    op.count = int(e.second.size());
                    for (const Mat2& u : e.second)
                        for (int k = 0; k < 4; ++k) plan.mats.push_back(u.u[k]);
                    plan.oq.push_back(op);
                }
                for (int sl : lb.oq_slices) plan.slice_last_wave[sl] = std::max(plan.slice_last_wave[sl], wave_index);
                w.oq_count = int(lb.oq.size());
                first = false;
            }
            // Jacobi groups: the tasks of a mode that run in one launch (one
            // per phase).  Launches of a stream follow one another, so a
            // latency-bound wave puts all of a mode's cluster tasks into one
            // launch: it lasts as long as its longest task.  The launch runs
            // the instance of its longest columns, so the wave's other tasks
            // take cluster sizes whose CTAs that instance allows
            // (`most_warps`); one with none gets a launch with its like.  A
            // batch keeps tasks of unlike column length apart, whose registers
            // and shared memory would be those of the longest.
            struct GKey {
                int mode, k1, k2;
            };
            struct Task {
                int local, c1, c2;  // job of the wave, cluster size per phase
            };
            std::vector<std::pair<GKey, std::vector<Task>>> groups;
            auto add = [&](int mode, int k1, int k2, const Task& t) {
                for (auto& g : groups)
                    if (g.first.mode == mode && g.first.k1 == k1 && g.first.k2 == k2) {
                        g.second.push_back(t);
                        return;
                    }
                groups.push_back({{mode, k1, k2}, {t}});
            };
            auto shape = [&](size_t k, int& rows, int& cols, int& ell) {
                rows = 2 * lb.bounds[k].first;
                cols = 2 * lb.bounds[k].second;
                ell = std::min(std::min(lb.jobs[k].chi_max + kRsvdOversample, rows), cols);
            };
            // Working matrix of a job in a mode: M x N, M >= N; and the matrix
            // its Jacobi runs on, R^H where a QR comes first.  Both are upper
            // bounds, and the choice of a QR is made from them alone, so the
            // device takes it from the job.
            auto dims = [&](size_t k, int mode, int& M, int& N) {
                int rows, cols, ell;
                shape(k, rows, cols, ell);
                M = mode != kJacobiRsvd ? std::max(rows, cols) : cols;
                N = mode != kJacobiRsvd ? std::min(rows, cols) : ell;
            };
            auto takes_qr = [&](size_t k, int mode) {
                int M, N;
                dims(k, mode, M, N);
                return !m->direct_svd && jacobi_qr_takes(M, N);
            };
            auto jacobi_dims = [&](size_t k, int mode, int& M, int& N) {
                dims(k, mode, M, N);
                if (takes_qr(k, mode)) M = N;
            };
            // The wave takes the level's next jobs while their bucket has a
            // free slot (every job of a level is independent of the others).
            std::vector<size_t> sel;
            std::vector<int> sel_slot;
            {
                std::vector<int> used(m->bucket_chi.size(), 0);
                for (size_t k = 0; k < lb.jobs.size(); ++k) {
                    if (taken[k]) continue;
                    const int bk = m->bucket_of(lb.jobs[k].chi_max);
                    if (used[bk] >= m->bucket_cap[bk]) continue;
                    taken[k] = 1;
                    sel.push_back(k);
                    sel_slot.push_back(m->bucket_base[bk] + used[bk]++);
                }
                remaining -= sel.size();
            }
            const int nj_wave = int(sel.size());
            auto cluster_of = [&](int M, int N, size_t elem, int vrows, int most_warps) {
                const uint64_t shape_key = (uint64_t(M) << 20 | uint64_t(N) << 10 | uint64_t(vrows)) << 7 |
                                           uint64_t(most_warps) << 1 | (elem == sizeof(float2) ? 1 : 0);
                const uint64_t key = uint64_t(m->batch ? 0 : nj_wave) << 37 | shape_key;
                KnownCluster& known = known_clusters[(key * 0x9E3779B97F4A7C15ull) >> 56];
                if (known.key != key)
                    known = {key, choose_cluster(m->ctx, M, N, m->ctx->max_cluster, nj_wave, m->ctx->sm_count, elem,
                                                 m->batch, vrows, most_warps)};
                return known.C;
            };
            wave_tasks.clear();
            auto add_task = [&](int mode, int M, int N, int local) { wave_tasks.push_back({mode, M, N, local}); };
            w.jobs_off = int(plan.jobs.size());
            w.njobs = nj_wave;
            for (int local = 0; local < nj_wave; ++local) {
                const size_t k = sel[local];
                SplitJob J = lb.jobs[k];
                J.slot = sel_slot[local];
                J.pre = (takes_qr(k, kJacobiExact) ? 1 : 0) | (takes_qr(k, kJacobiRsvd) ? 2 : 0);
                plan.jobs.push_back(J);
                plan.slice_last_wave[lb.job_slice[k]] = std::max(plan.slice_last_wave[lb.job_slice[k]], wave_index);
                int rows, cols, ell;
                shape(k, rows, cols, ell);
                const unsigned long long f = (unsigned long long)rows * cols * ell;
                const bool rs = !m->reject && !m->exact_only && ell < std::min(rows, cols) &&
                                f >= (unsigned long long)kRsvdMinSide * kRsvdMinSide * kRsvdMinSide;
                w.max_dl = std::max(w.max_dl, lb.bounds[k].first);
                w.max_dr = std::max(w.max_dr, lb.bounds[k].second);
                w.max_rows = std::max(w.max_rows, rows);
                w.max_cols = std::max(w.max_cols, cols);
                w.max_ell = std::max(w.max_ell, ell);
                int M, N;
                jacobi_dims(k, kJacobiExact, M, N);
                add_task(kJacobiExact, M, N, local);
                if (rs) {
                    w.any_rsvd = true;
                    add_task(kJacobiFallback, M, N, local);
                    jacobi_dims(k, kJacobiRsvd, M, N);
                    add_task(kJacobiRsvd, M, N, local);
                }
            }
            // Cluster sizes, and the warps of the instance that the cluster
            // tasks of a mode share, per phase.
            const int phases = m->fp32 ? 2 : 1;
            auto elem_of = [&](int ph) { return m->fp32 && ph == 0 ? sizeof(float2) : sizeof(double2); };
            auto vrows_of = [&](const WaveTask& t, int ph) { return m->fp32 && ph == 0 ? t.N : 0; };
            auto kr_of = [&](const WaveTask& t, int ph) {
                return jacobi_ring_kr(m->fp32 && ph == 0, t.M, vrows_of(t, ph));
            };
            sizes.resize(wave_tasks.size());
            int most_warps[3][2] = {{32, 32}, {32, 32}, {32, 32}};
            for (size_t i = 0; i < wave_tasks.size(); ++i)
                for (int ph = 0; ph < phases; ++ph) {
                    const WaveTask& t = wave_tasks[i];
                    sizes[i][ph] = cluster_of(t.M, t.N, elem_of(ph), vrows_of(t, ph), 32);
                    if (!m->batch && sizes[i][ph] >= 1)
                        most_warps[t.mode][ph] =
                            std::min(most_warps[t.mode][ph], jacobi_ring_warps(kr_of(t, ph), int(elem_of(ph))));
                }
            // A shape beyond every cluster goes to the staged kernel: its key
            // is -b, the width of its blocks (0: no kernel takes it).
            auto key_of = [&](const WaveTask& t, int ph, int& c) {
                if (c < 1) return -jacobi_staged_b(t.M + vrows_of(t, ph), t.N, elem_of(ph), kSmemLimit, nullptr);
                if (m->batch) return kr_of(t, ph);
                RingShape s;
                ring_shape(t.M, t.N, vrows_of(t, ph), elem_of(ph), c, &s);
                if (s.warps <= most_warps[t.mode][ph]) return 1;
                const int shared = cluster_of(t.M, t.N, elem_of(ph), vrows_of(t, ph), most_warps[t.mode][ph]);
                if (shared < 1) return 1 + kr_of(t, ph);
                c = shared;
                return 1;
            };
            for (size_t i = 0; i < wave_tasks.size(); ++i) {
                const WaveTask& t = wave_tasks[i];
                Task out{t.local, sizes[i][0], sizes[i][1]};
                const int k1 = key_of(t, 0, out.c1);
                add(t.mode, k1, m->fp32 ? key_of(t, 1, out.c2) : 0, out);
            }
            // Launch shape of one phase for the tasks of a group.
            auto fill = [&](PhaseCfg& pc, int key, bool first, int mode, const std::vector<Task>& tasks, size_t elem,
                            bool with_v) {
                pc.idx_off = int(plan.idx.size());
                if (key <= 0) {
                    pc.staged = true;
                    pc.b = -key;
                    pc.C = m->ctx->max_cluster;
                    for (const Task& t : tasks) {
                        int M, N;
                        jacobi_dims(sel[t.local], mode, M, N);
                        pc.smem = std::max(pc.smem, size_t(2) * pc.b * size_t(with_v ? M + N : M) * elem);
                        plan.idx.push_back(jacobi_entry(t.local, 0));
                    }
                    pc.threads = 32 * std::min(kJacobiStagedThreads / 32, std::max(4, pc.b));
                    return;
                }
                int warps = 1, b = 1;
                for (const Task& t : tasks) {
                    int M, N;
                    jacobi_dims(sel[t.local], mode, M, N);
                    RingShape s;
                    const int c = first ? t.c1 : t.c2;
                    ring_shape(M, N, with_v ? N : 0, elem, c, &s);
                    pc.C = std::max(pc.C, c);
                    pc.kr = std::max(pc.kr, s.kr);
                    warps = std::max(warps, s.warps);
                    b = std::max(b, s.b);
                    int log2_c = 0;
                    while ((1 << log2_c) < c) ++log2_c;
                    plan.idx.push_back(jacobi_entry(t.local, log2_c));
                }
                pc.threads = 32 * warps;
                pc.smem = jacobi_ring_smem(b, pc.kr, elem);
            };
            for (auto& g : groups) {
                Group gr;
                gr.mode = g.first.mode;
                gr.count = int(g.second.size());
                for (const Task& t : g.second) {
                    if (!takes_qr(sel[t.local], gr.mode)) continue;
                    int M, N;
                    dims(sel[t.local], gr.mode, M, N);
                    gr.qr_kr = std::max(gr.qr_kr, jacobi_qr_kr(M));
                    gr.qr_C = std::max(gr.qr_C, std::min(m->ctx->max_cluster, (N + kJacobiQrPerCta - 1) / kJacobiQrPerCta));
                }
                if (m->fp32) {
                    gr.nph = 2;
                    fill(gr.ph[0], g.first.k1, true, gr.mode, g.second, sizeof(float2), true);
                    fill(gr.ph[1], g.first.k2, false, gr.mode, g.second, sizeof(double2), false);
                } else {
                    gr.nph = 1;
                    fill(gr.ph[0], g.first.k1, true, gr.mode, g.second, sizeof(double2), false);
                }
                w.groups.push_back(gr);
            }
            plan.waves.push_back(std::move(w));
        } while (remaining > 0);
    }
}

template <class T>
size_t stage_section(size_t& off, const std::vector<T>& v) {
    off = (off + 255) & ~size_t(255);
    const size_t at = off;
    off += v.size() * sizeof(T);
    return at;
}

wqc_status ensure_records(wqc_mps* m, size_t need) {
    if (need <= m->rec_cap) return WQC_OK;
    size_t cap = std::max<size_t>(need, m->rec_cap * 2 + 1024);
    void* p = nullptr;
    if (wqc_status s = dmalloc(m, &p, cap * sizeof(wqc_split_info))) return s;
    if (m->d_records) {
        CUDA_TRY(cudaStreamSynchronize(m->stream));
        CUDA_TRY(cudaMemcpy(p, m->d_records, m->rec_cap * sizeof(wqc_split_info), cudaMemcpyDeviceToDevice));
        dfree(m, m->d_records, m->rec_cap * sizeof(wqc_split_info));
    }
    m->d_records = static_cast<wqc_split_info*>(p);
    m->rec_cap = cap;
    return WQC_OK;
}

// Threads a CTA of the phase's kernel may have.
int phase_thread_limit(const PhaseCfg& pc, bool fp32) {
    return pc.staged ? kJacobiStagedThreads
                     : 32 * jacobi_ring_warps(pc.kr, int(fp32 ? sizeof(float2) : sizeof(double2)));
}

// Every SVD launch of a plan against the limits of its kernel, before any of
// the plan is enqueued.
wqc_status check_plan(const Plan& plan) {
    for (const Wave& w : plan.waves)
        for (const Group& g : w.groups)
            for (int ph = 0; ph < g.nph; ++ph) {
                const PhaseCfg& pc = g.ph[ph];
                if (pc.C < 1 || (pc.staged && pc.b < 1))
                    return fail(WQC_ERR_INVALID, "two-site matrix too large for the cluster-resident Jacobi SVD");
                if (pc.threads > phase_thread_limit(pc, g.nph == 2 && ph == 0) || pc.smem > kSmemLimit)
                    return fail(WQC_ERR_INVALID, "a Jacobi launch of " + std::to_string(pc.threads) + " threads and " +
                                                     std::to_string(pc.smem) + " bytes does not fit its kernel");
            }
    return WQC_OK;
}

wqc_status launch_plan(wqc_mps* m, Plan& plan) {
    if (plan.waves.empty()) return WQC_OK;
    if (wqc_status s = check_plan(plan)) return s;
    if (wqc_status s = ensure_records(m, size_t(plan.first_seq) + plan.nsplits)) return s;
    size_t off = 0;
    const size_t o_oq = stage_section(off, plan.oq);
    const size_t o_mats = stage_section(off, plan.mats);
    const size_t o_jobs = stage_section(off, plan.jobs);
    const size_t o_idx = stage_section(off, plan.idx);
    const size_t bytes = std::max<size_t>(off, 256);
    // host staging: wait for the previous copy out of it
    CUDA_TRY(cudaEventSynchronize(m->stage_done));
    if (bytes > m->h_stage_cap) {
        if (m->h_stage) cudaFreeHost(m->h_stage);
        m->h_stage = nullptr;
        CUDA_TRY(cudaHostAlloc(reinterpret_cast<void**>(&m->h_stage), bytes * 2, cudaHostAllocDefault));
        m->h_stage_cap = bytes * 2;
    }
    if (bytes > m->d_stage.cap) {
        CUDA_TRY(cudaStreamSynchronize(m->stream));
        dfree(m, m->d_stage.d, m->d_stage.cap);
        m->d_stage.d = nullptr;
        m->d_stage.cap = 0;
        if (wqc_status s = dmalloc(m, &m->d_stage.d, bytes * 2)) return s;
        m->d_stage.cap = bytes * 2;
    }
    std::memcpy(m->h_stage + o_oq, plan.oq.data(), plan.oq.size() * sizeof(OneQubitOp));
    std::memcpy(m->h_stage + o_mats, plan.mats.data(), plan.mats.size() * sizeof(double2));
    std::memcpy(m->h_stage + o_jobs, plan.jobs.data(), plan.jobs.size() * sizeof(SplitJob));
    std::memcpy(m->h_stage + o_idx, plan.idx.data(), plan.idx.size() * sizeof(int));
    CUDA_TRY(cudaMemcpyAsync(m->d_stage.d, m->h_stage, bytes, cudaMemcpyHostToDevice, m->stream));
    m->stats.h2d_bytes += bytes;
    CUDA_TRY(cudaEventRecord(m->stage_done, m->stream));
    char* dbase = static_cast<char*>(m->d_stage.d);
    const OneQubitOp* d_oq = reinterpret_cast<const OneQubitOp*>(dbase + o_oq);
    const double2* d_mats = reinterpret_cast<const double2*>(dbase + o_mats);
    const SplitJob* d_jobs_all = reinterpret_cast<const SplitJob*>(dbase + o_jobs);
    const int* d_idx = reinterpret_cast<const int*>(dbase + o_idx);

    const bool track = m->profiling && !plan.slice_last_wave.empty();
    if (track) {
        while (m->wave_done.size() < plan.waves.size()) {
            cudaEvent_t e = nullptr;
            CUDA_TRY(cudaEventCreate(&e));
            m->wave_done.push_back(e);
        }
        if (!m->call_start) CUDA_TRY(cudaEventCreate(&m->call_start));
        CUDA_TRY(cudaEventRecord(m->call_start, m->stream));
        m->slice_last_wave = plan.slice_last_wave;
    }
    for (size_t wi = 0; wi < plan.waves.size(); ++wi) {
        const Wave& w = plan.waves[wi];
        if (w.oq_count > 0) {
            Timed t(m, 3);
            const int gx = std::min(64, std::max(1, (m->chi * m->chi + 1023) / 1024));
            apply_1q_kernel<<<dim3(gx, w.oq_count), 256, 0, m->stream>>>(d_oq + w.oq_off, d_mats, m->dev);
            count_launch(m, 3);
        }
        if (w.njobs == 0) {
            if (track) CUDA_TRY(cudaEventRecord(m->wave_done[wi], m->stream));
            continue;
        }
        const SplitJob* d_jobs = d_jobs_all + w.jobs_off;
        const int nj = w.njobs;
        // The plain and precision forms end on FP64 columns of an FP64 theta:
        // no singular value is FP32 noise.  The tensor-core form's theta
        // carries FP32-level error (~1e-7 of its norm), which shows as
        // singular values of ~1e-8 of the largest where theta has none; those
        // below 1e-6 of the largest count as zero.
        const double noise_rel = m->tc ? 1e-6 : 0.0;
        {
            Timed t(m, 1);
            // A state that was not told which merge to use takes the FMA tiles
            // where they are faster (one merge at bond 32 15 us against 27, at
            // 128 37 against 49, at 192 58 against 58, at 256 73 against 64).
            const bool oz = m->oz && (!m->oz_auto || std::min(w.max_dl, w.max_dr) > kOzAutoBond);
            if (oz || m->tc) {
                prepare_kernel<<<(nj + 127) / 128, 128, 0, m->stream>>>(d_jobs, m->d_state, nj, m->dev);
                count_launch(m, 1);
            }
            if (oz) {
                // rows of L by warps, N tiles of R (8 values of b) by blocks
                const int a_blocks = std::max(1, (w.max_rows + 7) / 8);
                const int ntiles = (w.max_dr + 7) / 8;
                const int b_blocks = ntiles * (m->oz_planes.kpad / kOzKBlock);
                oz_prep_merge_kernel<<<dim3(a_blocks + b_blocks, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->dev,
                                                                                           m->oz_planes, a_blocks);
                count_launch(m, 1);
                const dim3 g(ntiles, (w.max_rows + kOzTileM - 1) / kOzTileM, nj);
                CUDA_TRY(launch_oz_merge(m->oz_planes, g, m->stream, TcMergeArgs{d_jobs, m->d_state, m->d_slots},
                                         m->d_status));
                count_launch(m, 1);
            } else if (m->tc) {
                // one thread per complex value of L, one block per 32 K values of an N tile of R
                const int a_blocks = std::max(1, (w.max_rows * m->chi + 255) / 256);
                const dim3 gp(a_blocks + ((w.max_dr + 31) / 32) * (m->tc_kpad / kTcKBlock), nj);
                tc_prep_merge_kernel<<<gp, 256, 0, m->stream>>>(d_jobs, m->d_state, m->dev, m->tc_a, m->tc_b,
                                                                m->tc_rpad, m->tc_npad, m->tc_kpad, a_blocks);
                count_launch(m, 1);
                const dim3 g((w.max_dr + 31) / 32, (w.max_rows + kTcTileM - 1) / kTcTileM, nj);
                CUDA_TRY(launch_tc_merge(m->tc_map_a, m->tc_map_b, g, m->stream,
                                         TcMergeArgs{d_jobs, m->d_state, m->d_slots}, m->d_status));
                count_launch(m, 1);
            } else {
                dim3 g((w.max_dr + 15) / 16, (w.max_dl + 15) / 16, nj);
                merge_gate_kernel<<<g, 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, m->dev);
                count_launch(m, 1);
            }
        }
        auto launch_phase = [&](const Group& gr, const PhaseCfg& pc, int mode, int phase, bool fp32,
                                cudaStream_t on) -> wqc_status {
            Timed t(m, 0, on);
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(gr.count * pc.C);
            cfg.blockDim = dim3(pc.threads);
            cfg.dynamicSmemBytes = pc.smem;
            cfg.stream = on;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = pc.C;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (pc.staged)
                CUDA_TRY(launch_jacobi_staged(fp32, cfg, d_jobs, m->d_state, m->d_slots, d_idx + pc.idx_off, mode, phase,
                                              kMaxSweeps, pc.b, m->d_status, m->d_counters));
            else
                CUDA_TRY(launch_jacobi(fp32, pc.kr, cfg, d_jobs, m->d_state, m->d_slots, d_idx + pc.idx_off, mode,
                                       phase, kMaxSweeps, m->d_status, m->d_counters));
            count_launch(m, 0);
            return WQC_OK;
        };
        auto jacobi = [&](int mode, cudaStream_t on) -> wqc_status {
            bool any = false;
            for (const Group& gr : w.groups) {
                if (gr.mode != mode) continue;
                any = true;
                if (gr.qr_kr) {
                    Timed t(m, 0, on);
                    CUDA_TRY(launch_jacobi_qr(gr.qr_kr, gr.qr_C, gr.count, on, d_jobs, m->d_state, m->d_slots,
                                              d_idx + gr.ph[0].idx_off, mode, m->d_status));
                    count_launch(m, 0);
                }
                if (gr.nph == 1) {
                    if (wqc_status s = launch_phase(gr, gr.ph[0], mode, kPhasePlain, false, on)) return s;
                } else if (wqc_status s = launch_phase(gr, gr.ph[0], mode, kPhaseFp32V, true, on)) {
                    return s;
                }
            }
            if (!any) return WQC_OK;
            if (m->fp32) {
                // V orthonormalised (two Newton-Schulz steps), X V for every job of the mode, then the FP64 finish.
                Timed t(m, 0, on);
                const int side = std::max(w.max_rows, w.max_cols);
                // Small tiles while large ones would leave SMs idle.  A batch
                // takes large ones whatever it holds: the two round
                // differently, and a slice's results do not depend on the
                // other slices.
                const int large = (side + kPrecondTile - 1) / kPrecondTile;
                const bool small = !m->batch && long(large) * large * nj < 2L * m->ctx->sm_count;
                const unsigned side_t = unsigned(small ? (side + kTile - 1) / kTile : large);
                for (int stage = 0; stage < kPrecondStages; ++stage) {
                    if (small)
                        precond_gemm_kernel<true><<<dim3(side_t, side_t, nj), 256, 0, on>>>(d_jobs, m->d_state, m->d_slots,
                                                                                             mode, stage);
                    else
                        precond_gemm_kernel<false><<<dim3(side_t, side_t, nj), 256, 0, on>>>(d_jobs, m->d_state, m->d_slots,
                                                                                             mode, stage);
                    count_launch(m, 0);
                }
            }
            for (const Group& gr : w.groups)
                if (gr.mode == mode && gr.nph == 2)
                    if (wqc_status s = launch_phase(gr, gr.ph[1], mode, kPhaseFinish, false, on)) return s;
            // The check only reads the SVD: beside the cut where the side
            // stream is free; the next wave waits for it.
            const bool aside = !w.any_rsvd;
            if (aside) {
                CUDA_TRY(cudaEventRecord(m->fork_ev, on));
                CUDA_TRY(cudaStreamWaitEvent(m->side, m->fork_ev, 0));
            }
            cudaStream_t ps = aside ? m->side : on;
            {
                Timed t(m, 4, ps);
                svd_probe_kernel<<<dim3(nj, 2), kProbeThreads, 0, ps>>>(d_jobs, m->d_state, m->d_slots, mode, 0,
                                                                        m->d_status);
                count_launch(m, 4);
            }
            if (aside) CUDA_TRY(cudaEventRecord(m->join_ev, m->side));
            return WQC_OK;
        };
        // Exact-path SVDs on the side stream, concurrently with the range
        // finder below (different jobs, different slots and records).
        const bool fork = w.any_rsvd;
        cudaStream_t xs = fork ? m->side : m->stream;
        if (fork) {
            CUDA_TRY(cudaEventRecord(m->fork_ev, m->stream));
            CUDA_TRY(cudaStreamWaitEvent(m->side, m->fork_ev, 0));
        }
        if (wqc_status s = jacobi(kJacobiExact, xs)) return s;
        auto tiles = [](int x) { return (x + 15) / 16; };
        if (!w.any_rsvd) {
            Timed t(m, 4);
            const int kmax = std::min(m->chi, std::min(w.max_rows, w.max_cols));
            const int tn = tiles(std::max(w.max_cols, kmax)), tm = tiles(std::max(w.max_rows, kmax));
            const int copies = std::max(1, std::min(64, std::max(w.max_rows, w.max_cols) * kmax / 1024));
            cut_kernel<<<dim3(tm * tn + copies, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, m->dev, tm * tn,
                                                                        tn, m->chi, noise_rel, m->d_records, m->d_status);
            count_launch(m, 4);
            CUDA_TRY(cudaStreamWaitEvent(m->stream, m->join_ev, 0));
            if (track) CUDA_TRY(cudaEventRecord(m->wave_done[wi], m->stream));
            continue;
        }
        {
            Timed t(m, 4, xs);
            finalize_kernel<<<nj, 256, 0, xs>>>(d_jobs, m->d_state, m->d_slots, kJacobiExact, m->chi, noise_rel,
                                                m->d_records, m->d_status);
            count_launch(m, 4);
        }
        if (fork) CUDA_TRY(cudaEventRecord(m->join_ev, m->side));
        if (w.any_rsvd) {
            {
                Timed t(m, 2);
                omega_kernel<<<dim3(32, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots);
                const int tr = tiles(w.max_rows), tc = tiles(w.max_cols), te = tiles(w.max_ell);
                rsvd_gemm_kernel<<<dim3(te, tr, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kStageY0);
                rsvd_gemm_kernel<<<dim3(te, tc, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kStageZ);
                rsvd_gemm_kernel<<<dim3(te, tr, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kStageY);
                // Columns in shared memory on the smallest cluster that holds
                // them; else in global memory on the largest cluster; Y taller
                // than the cluster kernel's reflector registers hold: one CTA.
                int cq = 0;
                bool qglobal = false;
                const bool qfits = w.max_rows <= kQrRowsPerThread * kQrClusterThreads;
                for (int c = 8; qfits && c <= m->ctx->max_cluster; c *= 2)
                    if (qr_cluster_smem_bytes(w.max_rows, w.max_ell, c) <= kSmemLimit) {
                        cq = c;
                        break;
                    }
                if (qfits && !cq &&
                    qr_cluster_smem_bytes(w.max_rows, w.max_ell, m->ctx->max_cluster, true) <= kSmemLimit) {
                    cq = m->ctx->max_cluster;
                    qglobal = true;
                }
                if (cq) {
                    cudaLaunchConfig_t cfg = {};
                    cfg.gridDim = dim3(nj * cq);
                    cfg.blockDim = dim3(kQrClusterThreads);
                    cfg.dynamicSmemBytes = qr_cluster_smem_bytes(w.max_rows, w.max_ell, cq, qglobal);
                    cfg.stream = m->stream;
                    cudaLaunchAttribute attr[1];
                    attr[0].id = cudaLaunchAttributeClusterDimension;
                    attr[0].val.clusterDim.x = cq;
                    attr[0].val.clusterDim.y = 1;
                    attr[0].val.clusterDim.z = 1;
                    cfg.attrs = attr;
                    cfg.numAttrs = 1;
                    CUDA_TRY(launch_qr_cluster(qglobal, cfg, d_jobs, m->d_state, m->d_slots));
                } else {
                    householder_qr_kernel<<<nj, 512, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots);
                }
                rsvd_gemm_kernel<<<dim3(tc, te, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kStageB);
                for (int k = 0; k < 6; ++k) count_launch(m, 2);
            }
            if (wqc_status s = jacobi(kJacobiRsvd, m->stream)) return s;
            {
                Timed t(m, 4);
                finalize_kernel<<<nj, 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kJacobiRsvd, m->chi, noise_rel,
                                                            m->d_records, m->d_status);
                count_launch(m, 4);
            }
            if (wqc_status s = jacobi(kJacobiFallback, m->stream)) return s;
            {
                Timed t(m, 4);
                finalize_kernel<<<nj, 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, kJacobiFallback, m->chi, noise_rel,
                                                            m->d_records, m->d_status);
                count_launch(m, 4);
            }
        }
        if (fork) CUDA_TRY(cudaStreamWaitEvent(m->stream, m->join_ev, 0));
        {
            Timed t(m, 4);
            // The side the Jacobi does not accumulate, as tiled GEMMs over the
            // kept columns (chi <= min(chi_max, rows, cols)).
            const int kmax = std::min(m->chi, std::min(w.max_rows, w.max_cols));
            recover_gemm_kernel<<<dim3(tiles(std::max(w.max_cols, kmax)), tiles(std::max(w.max_ell, kmax)), nj), 256, 0,
                              m->stream>>>(
                d_jobs, m->d_state, m->d_slots, m->dev, kRecoverBW);
            recover_gemm_kernel<<<dim3(tiles(kmax), tiles(w.max_rows), nj), 256, 0, m->stream>>>(
                d_jobs, m->d_state, m->d_slots, m->dev, kRecoverQT);
            count_launch(m, 4);
            count_launch(m, 4);
            recover_gemm_kernel<<<dim3(tiles(std::max(w.max_cols, kmax)), tiles(std::max(w.max_rows, kmax)), nj), 256,
                                  0, m->stream>>>(d_jobs, m->d_state, m->d_slots, m->dev, kRecoverExact);
            count_launch(m, 4);
            const int per = std::max(w.max_rows, w.max_cols) * std::min(m->chi, std::max(w.max_rows, w.max_cols));
            const int gx = std::max(1, std::min(128, per / 256));
            absorb_kernel<<<dim3(gx, nj), 256, 0, m->stream>>>(d_jobs, m->d_state, m->d_slots, m->dev);
            count_launch(m, 4);
        }
        if (track) CUDA_TRY(cudaEventRecord(m->wave_done[wi], m->stream));
    }
    CUDA_TRY(cudaGetLastError());
    m->rec_count = plan.first_seq + plan.nsplits;
    return WQC_OK;
}

// After uploads: every site's left bond must equal its left neighbour's right
// bond, and each slice must start and end on a bond of 1.  An upload is one
// site at a time, so the chain can only be checked once the caller computes
// on it; a broken chain is refused instead of giving wrong results.
wqc_status check_uploaded_chain(wqc_mps* m) {
    if (!m->uploaded) return WQC_OK;
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    std::vector<int> dl(m->n), dr(m->n);
    CUDA_TRY(cudaMemcpy(dl.data(), m->d_dl, m->n * sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(dr.data(), m->d_dr, m->n * sizeof(int), cudaMemcpyDeviceToHost));
    for (size_t sl = 0; sl < m->seg_first.size(); ++sl) {
        const int first = m->seg_first[sl], last = first + m->seg_n[sl] - 1;
        for (int q = first; q <= last; ++q) {
            const int want = q == first ? 1 : dr[q - 1];
            if (dl[q] != want)
                return fail(WQC_ERR_INVALID, "uploaded sites do not chain: site " + std::to_string(q - first) +
                                                 " has left bond " + std::to_string(dl[q]) + ", expected " +
                                                 std::to_string(want));
        }
        if (dr[last] != 1)
            return fail(WQC_ERR_INVALID, "uploaded sites do not chain: the last site's right bond is " +
                                             std::to_string(dr[last]) + ", expected 1");
    }
    m->uploaded = false;
    return WQC_OK;
}

wqc_status run_ops(wqc_mps* m, const std::vector<Op>& ops) {
    if (*m->h_cancel) return fail(WQC_ERR_CANCELLED, "computation cancelled: the client has gone");
    if (wqc_status s = check_uploaded_chain(m)) return s;
    Plan plan;
    build_plan(m, ops, plan);
    return launch_plan(m, plan);
}

// |0> on every site, all bonds 1, status cleared (mps.rs:101-109).
wqc_status reset_sites(wqc_mps* m) {
    reset_sites_kernel<<<(m->n + 255) / 256, 256, 0, m->stream>>>(m->dev);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return WQC_OK;
}

wqc_status sync_status(wqc_mps* m) {
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    int stv[5] = {0, 0, 0, 0, 0};
    CUDA_TRY(cudaMemcpy(stv, m->d_status, sizeof(stv), cudaMemcpyDeviceToHost));
    const int st = stv[0];
    if (*m->h_cancel) return fail(WQC_ERR_CANCELLED, "computation cancelled: the client has gone");
    if (st & kStatusCancelled) return fail(WQC_ERR_CANCELLED, "computation cancelled: the client has gone");
    if (st & kStatusTruncationRejected) return fail(WQC_ERR_TRUNCATION_REJECTED, "mps bond exceeded chi");
    if (st & kStatusNonFinite) return fail(WQC_ERR_SVD_FAILED, "SVD of a two-site matrix produced non-finite values");
    if (st & kStatusSvdCheck) return fail(WQC_ERR_SVD_FAILED, "SVD of a two-site matrix failed its check");
    if (st & kStatusDeviceTimeout) return fail(WQC_ERR_DEVICE_TIMEOUT, "a tensor-core merge gave up waiting on its operands");
    if (st & kStatusJacobiNoConvergence) {
        const unsigned long long bits = (static_cast<unsigned long long>(static_cast<unsigned>(stv[3])) << 32) |
                                        static_cast<unsigned>(stv[4]);
        double rel2;
        std::memcpy(&rel2, &bits, sizeof(rel2));
        char buf[200];
        std::snprintf(buf, sizeof(buf),
                      "Jacobi SVD of a two-site matrix did not converge in 60 sweeps (split %d: last sweep %d "
                      "rotations, max |gamma|/sqrt(alpha beta) %.3e)",
                      stv[1] - 1, stv[2], std::sqrt(rel2));
        return fail(WQC_ERR_SVD_FAILED, buf);
    }
    if (st & kStatusBadShape) return fail(WQC_ERR_INVALID, "two-site matrix without a Jacobi workspace");
    return WQC_OK;
}

// The bonds left of every site, then right of every site, as they are on the
// device; waits for the stream.
wqc_status read_bonds(wqc_mps* m, std::vector<int>& dl_dr) {
    dl_dr.resize(2 * size_t(m->n));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    CUDA_TRY(cudaMemcpy(dl_dr.data(), m->d_dl, dl_dr.size() * sizeof(int), cudaMemcpyDeviceToHost));
    return WQC_OK;
}

// <psi|P_t|psi> of every term on every segment of `width` sites, vals[seg *
// nterms + t]; ends with the state's synchronisation.  Terms are cut to the
// sites between their first and last non-identity ones and share the identity
// environments on both sides, so a local observable costs one chain and a few
// products a term: 99 local terms on 50 sites took 141 ms as walks over all
// sites and 2.0 ms so at bond 128, 1.8 and 0.59 at 32, 1.28 and 0.59 at 24.  At
// small bonds, where a site's products are shorter than a launch, one launch
// walks every term over all sites: bond 16, 20 sites 0.12 ms against 0.27; and
// bond 24 where the terms span the register (20 such terms on 20 sites 0.22 ms
// against 0.48, at bond 32 0.98 against 0.50).  The rule looks at a segment's
// own bonds: a slice's values do not depend on the other slices of its batch.
// The chains hold 3 cap^2 entries a site, where cap is the state's chi_max; it
// is the largest bond instead, which takes a synchronisation, where that
// would be more than is kept between reads.  Where the device has no room for
// the chains the terms go one at a time, and then all segments walk, with
// four cap^2 entries for as many terms as fit.
constexpr int kPauliWalkBond = 16, kPauliWalkBondLong = 24;
wqc_status pauli_values(wqc_mps* m, const std::vector<int>& firsts, int width, const char* labels, uint32_t nterms,
                        std::vector<double2>& vals) {
    const int nseg = int(firsts.size());
    vals.resize(size_t(nseg) * nterms);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t lab_b = al(size_t(nterms) * width + 16), int_b = al(size_t(nterms) * sizeof(int));
    const size_t out_b = al(size_t(nseg) * nterms * sizeof(double2)), first_b = al(nseg * sizeof(int));
    std::vector<int> start(nterms), span(nterms);
    int longest_all = 1;
    for (uint32_t t = 0; t < nterms; ++t) {
        int lo = width, hi = -1;
        for (int q = 0; q < width; ++q)
            if (labels[size_t(t) * width + (width - 1 - q)] != 'I') {
                lo = std::min(lo, q);
                hi = q;
            }
        start[t] = hi < 0 ? 0 : lo;
        span[t] = hi < 0 ? 1 : hi - lo + 1;
        longest_all = std::max(longest_all, span[t]);
    }
    // The walked segments first, then those that take chains.
    std::vector<int> order, chained;
    int bond = 1;  // bound of the chained segments' bonds
    for (int sl = 0; sl < nseg; ++sl) {
        int own = 1;
        for (int q = firsts[sl]; q + 1 < firsts[sl] + width; ++q) own = std::max(own, m->ub[q]);
        if (own <= kPauliWalkBond || (own <= kPauliWalkBondLong && 2 * longest_all > width)) {
            order.push_back(sl);
        } else {
            chained.push_back(sl);
            bond = std::max(bond, own);
        }
    }
    int nwalk = int(order.size()), nchain = int(chained.size());
    std::vector<int> chain_firsts;
    for (int sl : chained) {
        order.push_back(sl);
        chain_firsts.push_back(firsts[sl]);
    }
    // Segments and terms at a time, within the memory that is kept between
    // reads, or within what there is.
    int segs = 1;
    uint32_t terms = 1, walk_terms = nterms;
    // Of an environment's side.  Not the host's bounds of the bonds: a split
    // that a cancellation skips leaves a larger bond than they say.
    int cap = m->chi;
    size_t E = 1;
    auto size_chains = [&](bool least) {
        E = size_t(cap) * cap;
        const size_t seg_b = (size_t(3) * width + 4) * E * sizeof(double2), term_b = 4 * E * sizeof(double2);
        segs = least ? 1
                     : int(std::max<size_t>(1, std::min<size_t>(size_t(std::min(nchain, 16384)),
                                                                (kScratchKeep / 2) / seg_b)));
        terms = least ? 1
                      : uint32_t(std::max<size_t>(1, std::min<size_t>(std::min<size_t>(nterms, 65535 / segs),
                                                                      (kScratchKeep / 4) / (term_b * segs))));
    };
    auto work_bytes = [&]() {
        const size_t walk_e = nwalk ? size_t(walk_terms) * 4 * E : 0;
        const size_t chain_e = nchain ? size_t(segs) * ((size_t(3) * width + 4) * E + size_t(terms) * 4 * E) : 0;
        return al(std::max(walk_e, chain_e) * sizeof(double2));
    };
    size_chains(false);
    bool tight = false;
    auto tighten = [&]() -> wqc_status {
        std::vector<int> now;
        if (wqc_status st = sync_status(m)) return st;
        if (wqc_status st = read_bonds(m, now)) return st;
        cap = *std::max_element(now.begin(), now.end());
        bond = std::min(bond, cap);
        tight = true;
        size_chains(false);
        return WQC_OK;
    };
    if (work_bytes() > kScratchKeep)
        if (wqc_status st = tighten()) return st;
    Scratch scratch(m);
    size_t work_b = 0;
    for (const ErrorState before;;) {
        work_b = work_bytes();
        const wqc_status st = scratch.get(work_b + lab_b + 2 * int_b + out_b + first_b);
        if (st == WQC_OK) {
            before.restore();
            break;
        }
        if (st != WQC_ERR_OOM) return st;
        if (!tight) {
            if (wqc_status ts = tighten()) return ts;
        } else if (nchain && (segs > 1 || terms > 1)) {
            size_chains(true);
        } else if (nchain) {
            nwalk = nseg;
            nchain = 0;
        } else if (walk_terms > 1) {
            walk_terms = (walk_terms + 1) / 2;
        } else {
            return st;
        }
    }
    char* p = static_cast<char*>(scratch.p);
    double2* work = reinterpret_cast<double2*>(p);
    char* d_lab = p + work_b;
    int* d_start = reinterpret_cast<int*>(d_lab + lab_b);
    int* d_span = reinterpret_cast<int*>(reinterpret_cast<char*>(d_start) + int_b);
    double2* d_out = reinterpret_cast<double2*>(reinterpret_cast<char*>(d_span) + int_b);
    int* d_first = reinterpret_cast<int*>(reinterpret_cast<char*>(d_out) + out_b);
    CUDA_TRY(cudaMemcpyAsync(d_lab, labels, size_t(nterms) * width, cudaMemcpyHostToDevice, m->stream));
    // One launch per walked segment on a view of its sites; launches share the scratch in stream order.
    for (int s = 0; s < nwalk; ++s) {
        const int first = firsts[order[s]];
        DeviceMps view = m->dev;
        view.site += first;
        view.dl += first;
        view.dr += first;
        view.n = width;
        for (uint32_t t0 = 0; t0 < nterms; t0 += walk_terms) {
            const uint32_t count = std::min(walk_terms, nterms - t0);
            pauli_expectation_kernel<<<count, 256, 0, m->stream>>>(view, d_lab + size_t(t0) * width, int(count), work,
                                                                   cap, d_out + size_t(s) * nterms + t0);
            count_launch(m, -1);
        }
    }
    if (nchain) {
        CUDA_TRY(cudaMemcpyAsync(d_start, start.data(), nterms * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(d_span, span.data(), nterms * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(d_first, chain_firsts.data(), nchain * sizeof(int), cudaMemcpyHostToDevice, m->stream));
        for (int s0 = 0; s0 < nchain; s0 += segs) {
            EnvChains ch{};
            ch.base = work;
            ch.seg_stride = (size_t(3) * width + 4) * E;
            ch.t_off = 0;
            ch.l_off = size_t(2) * width * E;
            ch.r_off = ch.l_off + 2 * E;
            ch.h_off = ch.r_off + size_t(width) * E;
            ch.firsts = d_first + s0;
            ch.nseg = std::min(segs, nchain - s0);
            ch.width = width;
            ch.cap = cap;
            ch.left = true;
            const EnvTerms tm{d_lab, d_start, d_span, work + size_t(segs) * ch.seg_stride};
            m->stats.total_launches += launch_env_chains(m->dev, ch, true, bond, m->stream);
            for (uint32_t t0 = 0; t0 < nterms; t0 += terms) {
                const int count = int(std::min<uint32_t>(terms, nterms - t0));
                const int longest = *std::max_element(span.begin() + t0, span.begin() + t0 + count);
                m->stats.total_launches += launch_env_terms(m->dev, ch, tm, int(t0), count, int(nterms), longest, bond,
                                                            d_out + size_t(nwalk + s0) * nterms, m->stream);
            }
        }
    }
    CUDA_TRY(cudaGetLastError());
    std::vector<double2> got(vals.size());
    CUDA_TRY(cudaMemcpyAsync(got.data(), d_out, got.size() * sizeof(double2), cudaMemcpyDeviceToHost, m->stream));
    const wqc_status rc = sync_status(m);
    scratch.drained = rc != WQC_ERR_CUDA;
    for (int s = 0; s < nseg; ++s)
        std::copy_n(got.begin() + size_t(s) * nterms, nterms, vals.begin() + size_t(order[s]) * nterms);
    return rc;
}

}  // namespace

// Lets entry points defined in other files of the library set the message
// that wqc_cuda_last_error returns.
namespace wqc {
wqc_status record_error(wqc_status code, const std::string& msg) { return fail(code, msg); }
wqc_status record_oom(uint64_t required, uint64_t available) { return fail_oom(required, available); }
wqc_status check_circuit_gate(int n, const wqc_gate& g) { return check_gate(n, g); }
void gate_matrix_2x2(int kind, double theta, double2 out[4]) {
    const Mat2 m = unary_matrix(kind, theta);
    for (int i = 0; i < 4; ++i) out[i] = m.u[i];
}
int context_device(const wqc_cuda_ctx* ctx) { return ctx->device; }
int context_sm_count(const wqc_cuda_ctx* ctx) { return ctx->sm_count; }
}  // namespace wqc

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

const char* wqc_cuda_last_error(void) { return g_err.c_str(); }

void wqc_cuda_last_oom(uint64_t* required, uint64_t* available) {
    if (required) *required = g_oom_required;
    if (available) *available = g_oom_available;
}

wqc_status wqc_cuda_open(int device, wqc_cuda_ctx** out) {
    if (!out) return fail(WQC_ERR_INVALID, "null output pointer");
    if (device < 0) {
        const char* env = std::getenv("WQC_CUDA_DEVICE");
        device = env ? std::atoi(env) : 0;
    }
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return fail(WQC_ERR_NO_DEVICE, "CUDA device not found");
    }
    if (device >= count) return fail(WQC_ERR_NO_DEVICE, "CUDA device index out of range");
    CUDA_TRY(cudaSetDevice(device));
    cudaDeviceProp prop{};
    CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (prop.major < 10) return fail(WQC_ERR_NO_DEVICE, "the cuda MPS backend is built for sm_100a (B200)");
    std::call_once(g_attr_once, set_kernel_attributes);
    if (g_attr_err != cudaSuccess) return fail(WQC_ERR_CUDA, std::string("kernel attributes: ") + cudaGetErrorString(g_attr_err));
    auto* ctx = new wqc_cuda_ctx();
    ctx->device = device;
    ctx->sm_count = prop.multiProcessorCount;
    // Largest cluster the device schedules with a full shared-memory CTA.
    ctx->max_cluster = 8;
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(512);
        cfg.dynamicSmemBytes = 200 * 1024;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 16;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, jacobi_staged(false), &cfg) == cudaSuccess && clusters > 0)
            ctx->max_cluster = 16;
        cudaGetLastError();
    }
    *out = ctx;
    return WQC_OK;
}

void wqc_cuda_close(wqc_cuda_ctx* ctx) {
    if (ctx) scratch_release(ctx->device);
    delete ctx;
}

wqc_status wqc_cuda_device_info(wqc_cuda_ctx* ctx, uint64_t* total_bytes, uint64_t* free_bytes, int32_t* sm_count) {
    if (!ctx) return fail(WQC_ERR_INVALID, "null context");
    CUDA_TRY(cudaSetDevice(ctx->device));
    scratch_release(ctx->device);
    size_t fr = 0, tot = 0;
    CUDA_TRY(cudaMemGetInfo(&fr, &tot));
    if (total_bytes) *total_bytes = tot;
    if (free_bytes) *free_bytes = fr;
    if (sm_count) *sm_count = ctx->sm_count;
    return WQC_OK;
}

uint64_t wqc_mps_workspace_bytes(uint32_t n, uint32_t chi) {
    const unsigned __int128 v = (unsigned __int128)n * chi * chi * 32;
    return v > ~uint64_t(0) ? ~uint64_t(0) : uint64_t(v);
}

// The host side of a state: its slices, the capacity of every site (offsets
// into the site pool) and the buckets of split slots.  No device work.
static void lay_out(wqc_mps* m, wqc_cuda_ctx* ctx, const std::vector<int>& ns, const std::vector<int>& chis,
                    int32_t precision, int nslots_req, std::vector<size_t>& site_off,
                    std::vector<size_t>& bucket_bytes, std::vector<size_t>& bucket_gs) {
    int n = 0;
    for (size_t sl = 0; sl < ns.size(); ++sl) {
        n += ns[sl];
        m->chi = std::max(m->chi, chis[sl]);
    }
    m->ctx = ctx;
    m->n = n;
    m->fp32 = precision != WQC_PRECISION_FP64;
    m->tc = precision == WQC_PRECISION_TF32X3;
    m->ub.assign(n > 0 ? n - 1 : 0, 1);
    m->site_chi.resize(n);
    m->site_slice.resize(n);
    site_off.assign(n + 1, 0);
    for (size_t sl = 0, g = 0; sl < ns.size(); ++sl) {
        m->seg_first.push_back(int(g));
        m->seg_n.push_back(ns[sl]);
        m->seg_chi.push_back(chis[sl]);
        for (int q = 0; q < ns[sl]; ++q, ++g) {
            m->site_chi[g] = chis[sl];
            m->site_slice[g] = int(sl);
            site_off[g + 1] = site_off[g] + size_t(chis[sl]) * 2 * chis[sl];
        }
    }
    // Split workspace: one bucket of slots per distinct chi_max, each slot
    // holding theta, w, z, the range finder's buffers and tau for two-site
    // matrices up to R x R, R = 2 chi_max (plus the staged Jacobi's workspace
    // when such a matrix can exceed a cluster's shared memory).  A bucket
    // gets a slot per two sites of its slices, at most kSlotBudget bytes of
    // them: waves take as many splits of a bucket as it has slots.
    // The staged Jacobi's workspace holds (R + 32) x R complex128 values: the
    // padded FP64 columns, or the precision form's complex64 columns with V
    // under them ((R + 32) x 2R complex64 values, the same bytes).
    const bool fp32 = precision != WQC_PRECISION_FP64;
    auto no_cluster = [&](int M, int N) {
        return choose_cluster(nullptr, M, N, ctx->max_cluster, 1, ctx->sm_count, sizeof(double2), false) < 1 ||
               (fp32 &&
                choose_cluster(nullptr, M, N, ctx->max_cluster, 1, ctx->sm_count, sizeof(float2), false, N) < 1);
    };
    {
        std::vector<int> cs(chis);
        std::sort(cs.begin(), cs.end());
        cs.erase(std::unique(cs.begin(), cs.end()), cs.end());
        m->nslots = 0;
        for (int c : cs) {
            const int R = 2 * c, E = std::min(c + kRsvdOversample, R);
            const bool staged = no_cluster(R, R) || no_cluster(R, E);
            const size_t gs_c = staged ? jacobi_staged_elems(R) : 0;
            const size_t slot_c = size_t(R) * R * 3 + size_t(R) * E * 6 + E + gs_c;
            const size_t bytes = ((slot_c * sizeof(double2) + size_t(R) * (sizeof(double) + sizeof(int)) + 4095) / 4096) * 4096;
            long count = 0;
            for (size_t sl = 0; sl < ns.size(); ++sl)
                if (chis[sl] == c) count += ns[sl] / 2;
            long cap = std::max<long>(1, std::min<long>(std::max<long>(count, 1), long(kSlotBudget / bytes)));
            if (nslots_req > 0) cap = std::min<long>(cap, nslots_req);
            m->bucket_chi.push_back(c);
            m->bucket_base.push_back(m->nslots);
            m->bucket_cap.push_back(int(cap));
            bucket_bytes.push_back(bytes);
            bucket_gs.push_back(gs_c);
            m->nslots += int(cap);
        }
    }
}

static wqc_status create_state(wqc_cuda_ctx* ctx, const std::vector<int>& ns, const std::vector<int>& chis,
                               int32_t precision, bool reject, int nslots_req, wqc_mps** out,
                               bool single_state = false) {
    if (!ctx || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (ns.empty()) return fail(WQC_ERR_INVALID, "no slices");
    long total_n = 0;
    int chi_cap = 0;
    for (size_t i = 0; i < ns.size(); ++i) {
        if (ns[i] <= 0)
            return fail(WQC_ERR_INVALID_QUBIT_COUNT, "Invalid qubit count: " + std::to_string(ns[i]) + ". Max limit is 40.");
        if (chis[i] <= 0) return fail(WQC_ERR_INVALID, "MPS max bond dimension must be > 0");
        if (chis[i] > 256) return fail(WQC_ERR_INVALID, "the cuda backend supports max_bond_dim <= 256");
        total_n += ns[i];
        chi_cap = std::max(chi_cap, chis[i]);
    }
    if (precision != WQC_PRECISION_FP64 && precision != WQC_PRECISION_FP32 && precision != WQC_PRECISION_TF32X3)
        return fail(WQC_ERR_INVALID, "unsupported precision form");
    if (total_n > (1L << 24)) return fail(WQC_ERR_INVALID, "too many sites");
    CUDA_TRY(cudaSetDevice(ctx->device));
    auto* m = new wqc_mps();
    const int n = int(total_n);
    m->reject = reject;
    std::vector<size_t> site_off, bucket_bytes, bucket_gs;
    lay_out(m, ctx, ns, chis, precision, nslots_req, site_off, bucket_bytes, bucket_gs);
    scratch_states(ctx->device, 1);
    m->device = ctx->device;
    auto bail = [&](wqc_status st) {
        wqc_mps_destroy(m);
        return st;
    };
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(fail(WQC_ERR_CUDA, "stream"));
    if (cudaStreamCreateWithFlags(&m->side, cudaStreamNonBlocking) != cudaSuccess) return bail(fail(WQC_ERR_CUDA, "stream"));
    if (cudaEventCreateWithFlags(&m->fork_ev, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&m->join_ev, cudaEventDisableTiming) != cudaSuccess)
        return bail(fail(WQC_ERR_CUDA, "event"));
    if (cudaEventCreateWithFlags(&m->stage_done, cudaEventDisableTiming) != cudaSuccess) return bail(fail(WQC_ERR_CUDA, "event"));
    cudaEventRecord(m->stage_done, m->stream);
    size_t slot_pool_bytes = 0;
    for (size_t b = 0; b < m->bucket_chi.size(); ++b) slot_pool_bytes += bucket_bytes[b] * size_t(m->bucket_cap[b]);
    const size_t site_bytes = site_off[n] * sizeof(double2);
    // Tensor-core form: TF32 hi/lo planes of both merge operands for every job
    // a wave can hold (one per slot), padded to whole tiles of the largest
    // two-site matrix.
    size_t tc_a_bytes = 0, tc_b_bytes = 0;
    if (m->tc) {
        m->tc_rpad = tc_rpad(2 * chi_cap);
        m->tc_kpad = tc_kpad(chi_cap);
        m->tc_npad = tc_npad(2 * chi_cap);
        tc_a_bytes = size_t(2) * m->nslots * m->tc_rpad * m->tc_kpad * sizeof(float);
        tc_b_bytes = size_t(2) * m->nslots * m->tc_npad * m->tc_kpad * sizeof(float);
    }
    // States from wqc_mps_create merge from int8 digit slices on the tensor
    // cores where that is faster (FP64-level, kOzAutoBond); batches (a batch of
    // one included) keep FMA merges, whose many slots would each need digit
    // planes.
    const bool oz_default = single_state && !m->tc;
    const uint64_t need = site_bytes + uint64_t(slot_pool_bytes) + tc_a_bytes + tc_b_bytes +
                          (oz_default ? oz_state_bytes(m) : 0);
    size_t fr = 0;
    if (device_room(need, &fr) != cudaSuccess) return bail(fail(WQC_ERR_CUDA, "cudaMemGetInfo"));
    if (need > fr) return bail(fail_oom(need, fr));
    void* p = nullptr;
    if (wqc_status st = dmalloc(m, &p, site_bytes)) return bail(st);
    m->site_pool = static_cast<double2*>(p);
    if (wqc_status st = dmalloc(m, &p, size_t(n) * sizeof(double2*))) return bail(st);
    m->d_site_ptr = static_cast<double2**>(p);
    if (wqc_status st = dmalloc(m, &p, 2 * size_t(n) * sizeof(int) + 64)) return bail(st);
    m->d_dl = static_cast<int*>(p);
    m->d_dr = m->d_dl + n;
    m->d_status = m->d_dr + n;
    if (wqc_status st = dmalloc(m, &p, 2 * ns.size() * sizeof(int))) return bail(st);
    m->d_seg = static_cast<int*>(p);
    if (wqc_status st = dmalloc(m, &p, slot_pool_bytes)) return bail(st);
    m->slot_pool = static_cast<char*>(p);
    if (m->tc) {
        if (wqc_status st = dmalloc(m, &p, tc_a_bytes)) return bail(st);
        m->tc_a = static_cast<float*>(p);
        if (wqc_status st = dmalloc(m, &p, tc_b_bytes)) return bail(st);
        m->tc_b = static_cast<float*>(p);
        if (!tc_encode_planes(&m->tc_map_a, m->tc_a, m->tc_kpad, m->tc_rpad, 2 * m->nslots) ||
            !tc_encode_planes(&m->tc_map_b, m->tc_b, m->tc_kpad, m->tc_npad, 2 * m->nslots))
            return bail(fail(WQC_ERR_CUDA, "cuTensorMapEncodeTiled refused the merge operand planes"));
    }
    if (wqc_status st = dmalloc(m, &p, m->nslots * sizeof(SlotBuffers))) return bail(st);
    m->d_slots = static_cast<SlotBuffers*>(p);
    if (wqc_status st = dmalloc(m, &p, m->nslots * sizeof(SplitState))) return bail(st);
    m->d_state = static_cast<SplitState*>(p);
    const size_t small = std::max<size_t>(64, 2 * ns.size() + 8);
    if (wqc_status st = dmalloc(m, &p, small * sizeof(double2))) return bail(st);
    m->d_small = static_cast<double2*>(p);
    m->d_counters = reinterpret_cast<unsigned long long*>(m->d_small + small - 4);
    if (cudaMemset(m->d_small, 0, small * sizeof(double2)) != cudaSuccess) return bail(fail(WQC_ERR_CUDA, "memset"));
    m->oz_auto = oz_default;
    if (oz_default)
        if (wqc_status st = oz_enable(m)) return bail(st);
    if (ns.size() == 1) {  // the trace feeders' environment cache (single states)
        const size_t env_bytes = 2 * size_t(n) * chi_cap * sizeof(double2) + size_t(n) * 2 * sizeof(double2) +
                                 size_t(n) * sizeof(int);
        if (wqc_status st = dmalloc(m, &p, env_bytes)) return bail(st);
        m->d_envL = static_cast<double2*>(p);
        m->d_envR = m->d_envL + size_t(n) * chi_cap;
        m->d_env_out = m->d_envR + size_t(n) * chi_cap;
        m->d_targets = reinterpret_cast<int*>(m->d_env_out + size_t(n) * 2);
    }
    m->lvalid = 0;
    m->rvalid = n - 1;
    int* hc = nullptr;
    if (cudaHostAlloc(reinterpret_cast<void**>(&hc), sizeof(int), cudaHostAllocMapped) != cudaSuccess)
        return bail(fail(WQC_ERR_CUDA, "cudaHostAlloc"));
    *hc = 0;
    m->h_cancel = hc;
    if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&m->d_cancel), hc, 0) != cudaSuccess)
        return bail(fail(WQC_ERR_CUDA, "cudaHostGetDevicePointer"));
    m->site_ptr.resize(n);
    for (int i = 0; i < n; ++i) m->site_ptr[i] = m->site_pool + site_off[i];
    std::vector<int> seg(2 * ns.size());
    for (size_t sl = 0; sl < ns.size(); ++sl) {
        seg[2 * sl] = m->seg_first[sl];
        seg[2 * sl + 1] = m->seg_n[sl];
    }
    if (cudaMemcpy(m->d_site_ptr, m->site_ptr.data(), size_t(n) * sizeof(double2*), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(m->d_seg, seg.data(), seg.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
        return bail(fail(WQC_ERR_CUDA, "initial upload"));
    std::vector<SlotBuffers> slots(m->nslots);
    m->slot_R.assign(m->nslots, 0);
    m->slot_E.assign(m->nslots, 0);
    char* base = m->slot_pool;
    for (int sl = 0; sl < m->nslots; ++sl) {
        size_t bk = 0;
        while (bk + 1 < m->bucket_chi.size() && sl >= m->bucket_base[bk + 1]) ++bk;
        const int R = 2 * m->bucket_chi[bk], E = std::min(m->bucket_chi[bk] + kRsvdOversample, R);
        const size_t gs_c = bucket_gs[bk];
        m->slot_R[sl] = R;
        m->slot_E[sl] = E;
        double2* c = reinterpret_cast<double2*>(base);
        base += bucket_bytes[bk];
        SlotBuffers& bf = slots[sl];
        bf.theta = c; c += size_t(R) * R;
        bf.w = c; c += size_t(R) * R;
        bf.z = c; c += size_t(R) * R;
        bf.omega = c; c += size_t(R) * E;
        bf.y0 = c; c += size_t(R) * E;
        bf.zr = c; c += size_t(R) * E;
        bf.y = c; c += size_t(R) * E;
        bf.q = c; c += size_t(R) * E;
        bf.b = c; c += size_t(R) * E;
        bf.tau = c; c += E;
        bf.gs = gs_c ? static_cast<void*>(c) : nullptr;
        c += gs_c;
        bf.sigma = reinterpret_cast<double*>(c);
        bf.perm = reinterpret_cast<int*>(bf.sigma + R);
    }
    if (cudaMemcpy(m->d_slots, slots.data(), slots.size() * sizeof(SlotBuffers), cudaMemcpyHostToDevice) != cudaSuccess)
        return bail(fail(WQC_ERR_CUDA, "slot table upload"));
    m->dev.site = m->d_site_ptr;
    m->dev.dl = m->d_dl;
    m->dev.dr = m->d_dr;
    m->dev.n = n;
    m->dev.chi_max = chi_cap;
    m->dev.status = m->d_status;
    m->dev.cancel = m->d_cancel;
    if (wqc_status st = ensure_records(m, 1024)) return bail(st);
    if (wqc_status st = reset_sites(m)) return bail(st);
    *out = m;
    return WQC_OK;
}

wqc_status wqc_mps_create(wqc_cuda_ctx* ctx, uint32_t n, uint32_t chi, int32_t precision, uint8_t reject,
                          wqc_mps** out) {
    return create_state(ctx, {int(n)}, {int(chi)}, precision, reject != 0, 0, out, true);
}

wqc_status wqc_batch_create(wqc_cuda_ctx* ctx, uint32_t count, const uint32_t* qubit_counts,
                            const uint32_t* max_bond_dims, int32_t precision, uint32_t max_concurrent_splits,
                            wqc_mps** out) {
    if (!qubit_counts || !max_bond_dims || count == 0) return fail(WQC_ERR_INVALID, "null argument");
    std::vector<int> ns(count), chis(count);
    for (uint32_t i = 0; i < count; ++i) {
        ns[i] = int(qubit_counts[i]);
        chis[i] = int(max_bond_dims[i]);
    }
    const wqc_status st = create_state(ctx, ns, chis, precision, false, int(max_concurrent_splits), out);
    if (st == WQC_OK) (*out)->batch = true;
    return st;
}

wqc_status wqc_mps_reset(wqc_mps* m) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    // A reset starts the next request whatever the last one ended with (an
    // error status, a cancellation): the queue drains, the cancel word and the
    // device status word are cleared and the sites return to |0...0>.
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    *m->h_cancel = 0;
    if (wqc_status st = reset_sites(m)) return st;
    std::fill(m->ub.begin(), m->ub.end(), 1);
    m->rec_count = 0;
    m->lvalid = 0;
    m->rvalid = m->n - 1;
    return WQC_OK;
}

void wqc_mps_destroy(wqc_mps* m) {
    if (!m) return;
    if (m->stream) cudaStreamSynchronize(m->stream);
    dfree(m, m->site_pool, 0);
    dfree(m, m->d_site_ptr, 0);
    dfree(m, m->d_dl, 0);
    dfree(m, m->slot_pool, 0);
    dfree(m, m->tc_a, 0);
    dfree(m, m->tc_b, 0);
    dfree(m, m->oz_pool, 0);
    dfree(m, m->d_slots, 0);
    dfree(m, m->d_state, 0);
    dfree(m, m->d_small, 0);
    dfree(m, m->d_records, 0);
    dfree(m, m->d_seg, 0);
    dfree(m, m->d_envL, 0);
    for (auto e : m->wave_done) cudaEventDestroy(e);
    if (m->call_start) cudaEventDestroy(m->call_start);
    dfree(m, m->d_stage.d, 0);
    if (m->h_stage) cudaFreeHost(m->h_stage);
    if (m->h_cancel) cudaFreeHost(const_cast<int*>(m->h_cancel));
    for (auto& e : m->events) {
        cudaEventDestroy(e.second.first);
        cudaEventDestroy(e.second.second);
    }
    for (auto e : m->event_pool) cudaEventDestroy(e);
    if (m->stage_done) cudaEventDestroy(m->stage_done);
    if (m->fork_ev) cudaEventDestroy(m->fork_ev);
    if (m->join_ev) cudaEventDestroy(m->join_ev);
    if (m->side) cudaStreamDestroy(m->side);
    if (m->stream) cudaStreamDestroy(m->stream);
    if (m->device >= 0) scratch_states(m->device, -1);
    delete m;
}

wqc_status wqc_schedule_gates(uint32_t n, const wqc_gate* gates, uint32_t count, int32_t* split_site,
                              int32_t* split_level, uint32_t max, uint32_t* nsplits, uint32_t* nlevels) {
    if (n == 0 || (!gates && count) || !nsplits || !nlevels) return fail(WQC_ERR_INVALID, "null argument");
    Expander ex;
    if (wqc_status s = expand(int(n), gates, count, false, ex)) return s;
    std::vector<int> level_of;
    assign_levels(int(n), ex.ops, level_of);
    uint32_t k = 0;
    int top = -1;
    for (size_t i = 0; i < ex.ops.size(); ++i) {
        top = std::max(top, level_of[i]);
        if (!ex.ops[i].two) continue;
        if (k < max) {
            if (split_site) split_site[k] = ex.ops[i].site;
            if (split_level) split_level[k] = level_of[i];
        }
        ++k;
    }
    *nsplits = k;
    *nlevels = uint32_t(top + 1);
    return WQC_OK;
}

wqc_status wqc_mps_debug_limit_bytes(wqc_mps* m, uint64_t bytes) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    m->bytes_limit = bytes ? m->bytes_now + bytes : ~uint64_t(0);
    return WQC_OK;
}

wqc_status wqc_debug_svd_launches(uint32_t n, uint32_t chi, uint32_t slices, int32_t precision, int32_t rule,
                                  int32_t sm_count, int32_t max_cluster, int32_t force_cluster, const wqc_gate* gates,
                                  uint32_t count, int32_t* out, uint32_t max, uint32_t* launches) {
    if (n == 0 || chi == 0 || chi > 256 || (!gates && count) || !launches || (!out && max))
        return fail(WQC_ERR_INVALID, "null argument");
    Expander ex;
    if (wqc_status s = expand(int(n), gates, count, false, ex)) return s;
    wqc_cuda_ctx ctx;
    ctx.sm_count = sm_count;
    ctx.max_cluster = max_cluster;
    ctx.force_C = force_cluster;
    wqc_mps m;
    std::vector<size_t> site_off, bucket_bytes, bucket_gs;
    const size_t nseg = std::max(1u, slices);
    lay_out(&m, &ctx, std::vector<int>(nseg, int(n)), std::vector<int>(nseg, int(chi)), precision, 0, site_off,
            bucket_bytes, bucket_gs);
    m.batch = slices > 0;
    m.exact_only = rule != WQC_SPLIT_RULE_REFERENCE;
    m.direct_svd = rule < 0;
    std::vector<Op> ops;
    for (size_t sl = 0; sl < nseg; ++sl)
        for (Op o : ex.ops) {
            o.site += int(sl * n);
            o.slice = int(sl);
            ops.push_back(o);
        }
    Plan plan;
    build_plan(&m, ops, plan);
    uint32_t k = 0;
    auto put = [&](int wave, int kind, int tasks, int C, int threads, int limit, size_t smem) {
        const int32_t row[8] = {wave, kind, tasks, C, threads, limit, int32_t(smem), int32_t(kSmemLimit)};
        if (k < max) std::copy(row, row + 8, out + size_t(k) * 8);
        ++k;
    };
    for (size_t wi = 0; wi < plan.waves.size(); ++wi)
        for (const Group& g : plan.waves[wi].groups)
            for (int ph = 0; ph < g.nph; ++ph) {
                const PhaseCfg& pc = g.ph[ph];
                put(int(wi), pc.staged ? 1 : 0, g.count, pc.C, pc.threads,
                    phase_thread_limit(pc, g.nph == 2 && ph == 0), pc.smem);
            }
    *launches = k;
    return WQC_OK;
}

wqc_status wqc_mps_apply_gates(wqc_mps* m, const wqc_gate* gates, uint32_t count) {
    if (!m || (!gates && count)) return fail(WQC_ERR_INVALID, "null argument");
    Expander ex;
    if (wqc_status s = expand(m->n, gates, count, false, ex)) return s;
    return run_ops(m, ex.ops);
}

wqc_status wqc_mps_apply_gates_adjoint(wqc_mps* m, const wqc_gate* gates, uint32_t count) {
    if (!m || (!gates && count)) return fail(WQC_ERR_INVALID, "null argument");
    Expander ex;
    if (wqc_status s = expand(m->n, gates, count, true, ex)) return s;
    return run_ops(m, ex.ops);
}

wqc_status wqc_batch_apply_gates(wqc_mps* m, const wqc_gate* gates, const uint32_t* offsets) {
    if (!m || !offsets) return fail(WQC_ERR_INVALID, "null argument");
    Expander all;
    for (size_t sl = 0; sl < m->seg_first.size(); ++sl) {
        const uint32_t g0 = offsets[sl], g1 = offsets[sl + 1];
        if (g1 < g0) return fail(WQC_ERR_INVALID, "gate offsets must not decrease");
        if (g1 == g0) continue;
        if (!gates) return fail(WQC_ERR_INVALID, "null gates");
        Expander ex;
        if (wqc_status s = expand(m->seg_n[sl], gates + g0, g1 - g0, false, ex)) return s;
        for (Op& o : ex.ops) {
            o.site += m->seg_first[sl];
            o.slice = int(sl);
            all.ops.push_back(o);
        }
    }
    return run_ops(m, all.ops);
}

wqc_status wqc_batch_amplitudes(wqc_mps* m, double* out) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (wqc_status st = check_uploaded_chain(m)) return st;
    const int nseg = int(m->seg_first.size());
    amplitude_zero_kernel<<<nseg, 512, 2 * m->chi * sizeof(double2), m->stream>>>(m->dev, m->d_seg, m->d_small);
    count_launch(m, -1);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(out, m->d_small, nseg * sizeof(double2), cudaMemcpyDeviceToHost, m->stream));
    m->stats.d2h_bytes += nseg * sizeof(double2);
    return sync_status(m);
}

wqc_status wqc_batch_expectation_pauli(wqc_mps* m, const char* labels, const double* coeffs, uint32_t nterms,
                                       double* out) {
    if (!m || !labels || !coeffs || !out) return fail(WQC_ERR_INVALID, "null argument");
    const int nseg = int(m->seg_first.size());
    const int width = nseg > 0 ? (m->n / nseg) : 0;
    for (int s = 0; s < nseg; ++s) {
        const int first = m->seg_first[s], last = s + 1 < nseg ? m->seg_first[s + 1] : m->n;
        if (last - first != width) return fail(WQC_ERR_INVALID, "batch expectation needs slices of one width");
    }
    for (size_t i = 0; i < size_t(nterms) * width; ++i) {
        const char ch = labels[i];
        if (ch != 'I' && ch != 'X' && ch != 'Y' && ch != 'Z')
            return fail(WQC_ERR_INVALID, std::string("invalid pauli character in label"));
    }
    if (nterms == 0 || nseg == 0) {
        for (int s = 0; s < 2 * nseg; ++s) out[s] = 0;
        return WQC_OK;
    }
    std::vector<int> firsts(m->seg_first.begin(), m->seg_first.end());
    std::vector<double2> vals;
    if (wqc_status st = pauli_values(m, firsts, width, labels, nterms, vals)) return st;
    for (int s = 0; s < nseg; ++s) {
        double re = 0, im = 0;
        for (uint32_t t = 0; t < nterms; ++t) {  // coeff * Re<P> (expectation.rs:177-185), term order
            const double v = vals[size_t(s) * nterms + t].x;
            re += coeffs[2 * t] * v;
            im += coeffs[2 * t + 1] * v;
        }
        out[2 * s] = re;
        out[2 * s + 1] = im;
    }
    return WQC_OK;
}

wqc_status wqc_batch_slice_times(wqc_mps* m, double* out_ms) {
    if (!m || !out_ms) return fail(WQC_ERR_INVALID, "null argument");
    if (wqc_status s = sync_status(m)) return s;
    const size_t nseg = m->seg_first.size();
    for (size_t sl = 0; sl < nseg; ++sl) {
        const int w = sl < m->slice_last_wave.size() ? m->slice_last_wave[sl] : -1;
        float ms = -1.0f;
        if (w >= 0 && m->call_start && size_t(w) < m->wave_done.size())
            CUDA_TRY(cudaEventElapsedTime(&ms, m->call_start, m->wave_done[w]));
        out_ms[sl] = double(ms);
    }
    return WQC_OK;
}

wqc_status wqc_mps_apply_1q(wqc_mps* m, uint32_t site, const double u[8]) {
    if (!m || !u) return fail(WQC_ERR_INVALID, "null argument");
    if (site >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "site out of range");
    Expander ex;
    Mat2 mm;
    for (int i = 0; i < 4; ++i) mm.u[i] = make_double2(u[2 * i], u[2 * i + 1]);
    ex.one(int(site), mm);
    return run_ops(m, ex.ops);
}

static Mat4 mat4_from(const double u[32]) {
    Mat4 mm;
    for (int i = 0; i < 16; ++i) mm.u[i] = make_double2(u[2 * i], u[2 * i + 1]);
    return mm;
}

wqc_status wqc_mps_apply_2q(wqc_mps* m, uint32_t left, const double u[32], uint8_t cf, wqc_split_info* info) {
    if (!m || !u) return fail(WQC_ERR_INVALID, "null argument");
    if (uint64_t(left) + 1 >= uint64_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "two-site apply needs adjacent positions");
    Expander ex;
    ex.two_at(int(left), mat4_from(u), cf != 0);
    const uint32_t seq = m->rec_count;
    if (wqc_status s = run_ops(m, ex.ops)) return s;
    if (info) {
        if (wqc_status s = sync_status(m)) return s;
        CUDA_TRY(cudaMemcpy(info, m->d_records + seq, sizeof(wqc_split_info), cudaMemcpyDeviceToHost));
    }
    return WQC_OK;
}

wqc_status wqc_mps_apply_2q_routed(wqc_mps* m, uint32_t ctrl, uint32_t tgt, const double u[32]) {
    if (!m || !u) return fail(WQC_ERR_INVALID, "null argument");
    if (ctrl >= uint32_t(m->n) || tgt >= uint32_t(m->n) || ctrl == tgt) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "bad qubit pair");
    Expander ex;
    ex.two_routed(int(ctrl), int(tgt), mat4_from(u));
    return run_ops(m, ex.ops);
}

wqc_status wqc_mps_apply_layer(wqc_mps* m, const wqc_gate* gates, uint32_t count) {
    if (!m || (!gates && count)) return fail(WQC_ERR_INVALID, "null argument");
    if (count >= 2) {
        std::vector<int> seen;
        for (uint32_t i = 0; i < count; ++i) {
            const wqc_gate& g = gates[i];
            if (g.kind != WQC_GATE_CNOT && g.kind != WQC_GATE_CZ)
                return fail(WQC_ERR_INVALID, "disjoint layer contains a gate that is not CNOT or CZ");
        }
    }
    return wqc_mps_apply_gates(m, gates, count);
}

wqc_status wqc_mps_set_split_rule(wqc_mps* m, int32_t rule) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    if (rule != WQC_SPLIT_RULE_REFERENCE && rule != WQC_SPLIT_RULE_EXACT) return fail(WQC_ERR_INVALID, "unknown split rule");
    m->exact_only = rule == WQC_SPLIT_RULE_EXACT;
    return WQC_OK;
}

wqc_status wqc_mps_set_merge(wqc_mps* m, int32_t merge) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    if (merge != WQC_MERGE_FFMA && merge != WQC_MERGE_TC_INT8) return fail(WQC_ERR_INVALID, "unknown merge");
    if (m->tc) return fail(WQC_ERR_INVALID, "the tensor-core form merges on its own TF32 path");
    CUDA_TRY(cudaSetDevice(m->ctx->device));
    CUDA_TRY(cudaStreamSynchronize(m->stream));  // no enqueued merge still reads the planes
    m->oz_auto = false;
    if (merge == WQC_MERGE_TC_INT8) return oz_enable(m);
    m->oz = false;
    return WQC_OK;
}

wqc_status wqc_mps_synchronize(wqc_mps* m) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    return sync_status(m);
}

void wqc_mps_cancel(wqc_mps* m) {
    if (m && m->h_cancel) *const_cast<volatile int*>(m->h_cancel) = 1;
}

wqc_status wqc_mps_amplitude_zero(wqc_mps* m, double out[2]) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (wqc_status st = check_uploaded_chain(m)) return st;
    amplitude_zero_kernel<<<1, 512, 2 * m->chi * sizeof(double2), m->stream>>>(m->dev, m->d_seg, m->d_small);
    count_launch(m, -1);
    CUDA_TRY(cudaGetLastError());
    double2 h;
    CUDA_TRY(cudaMemcpyAsync(&h, m->d_small, sizeof(double2), cudaMemcpyDeviceToHost, m->stream));
    m->stats.d2h_bytes += sizeof(double2);
    if (wqc_status s = sync_status(m)) return s;
    out[0] = h.x;
    out[1] = h.y;
    return WQC_OK;
}

wqc_status wqc_mps_site_amplitudes_many(wqc_mps* m, const uint32_t* targets, uint32_t count, double* out) {
    if (!m || (count && (!targets || !out))) return fail(WQC_ERR_INVALID, "null argument");
    if (!m->d_envL) return fail(WQC_ERR_INVALID, "site amplitudes take a single state, not a batch");
    if (count == 0) return WQC_OK;
    if (count > uint32_t(m->n)) return fail(WQC_ERR_INVALID, "more targets than sites");
    std::vector<int> t(count);
    int lo = m->n, hi = -1;
    for (uint32_t k = 0; k < count; ++k) {
        if (targets[k] >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "target out of range");
        t[k] = int(targets[k]);
        lo = std::min(lo, t[k]);
        hi = std::max(hi, t[k]);
    }
    if (wqc_status st = check_uploaded_chain(m)) return st;
    const int lfrom = m->lvalid, lto = std::max(m->lvalid, hi);
    const int rfrom = m->rvalid, rto = std::min(m->rvalid, lo);
    CUDA_TRY(cudaMemcpyAsync(m->d_targets, t.data(), count * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    m->stats.h2d_bytes += count * sizeof(int);
    site_envs_kernel<<<1, 512, 0, m->stream>>>(m->dev, m->d_envL, m->d_envR, lfrom, lto, rfrom, rto, m->d_targets,
                                               int(count), m->d_env_out);
    count_launch(m, -1);
    CUDA_TRY(cudaGetLastError());
    std::vector<double2> h(2 * size_t(count));
    CUDA_TRY(cudaMemcpyAsync(h.data(), m->d_env_out, h.size() * sizeof(double2), cudaMemcpyDeviceToHost, m->stream));
    m->stats.d2h_bytes += h.size() * sizeof(double2);
    if (wqc_status s = sync_status(m)) return s;
    m->lvalid = lto;
    m->rvalid = rto;
    for (size_t k = 0; k < h.size(); ++k) {
        out[2 * k] = h[k].x;
        out[2 * k + 1] = h[k].y;
    }
    return WQC_OK;
}

wqc_status wqc_mps_site_amplitudes(wqc_mps* m, uint32_t target, double out[4]) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (target >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "target out of range");
    return wqc_mps_site_amplitudes_many(m, &target, 1, out);
}

wqc_status wqc_mps_to_dense(wqc_mps* m, int32_t mode, double* out) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (m->seg_first.size() != 1) return fail(WQC_ERR_INVALID, "the dense state takes a single state, not a batch");
    if (mode != WQC_DENSE_TO_DENSE_STATE && mode != WQC_DENSE_STATEVECTOR)
        return fail(WQC_ERR_INVALID, "unknown dense mode");
    const int n = m->n;
    if (mode == WQC_DENSE_STATEVECTOR && n > 20)  // mps.rs:217-221
        return fail(WQC_ERR_INVALID, "full statevector projection requires qubit_count <= 20");
    if (n > kDenseMaxQubits)
        return fail(WQC_ERR_INVALID_QUBIT_COUNT, "the dense state is limited to " + std::to_string(kDenseMaxQubits) +
                                                     " qubits");
    if (wqc_status st = check_uploaded_chain(m)) return st;
    if (wqc_status s = sync_status(m)) return s;
    std::vector<int> dl(n), dr(n);
    CUDA_TRY(cudaMemcpy(dl.data(), m->d_dl, n * sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(dr.data(), m->d_dr, n * sizeof(int), cudaMemcpyDeviceToHost));
    size_t most = 1;
    for (int q = 0; q < n; ++q) {
        if (dl[q] != (q ? dr[q - 1] : 1))  // mps.rs:229-234
            return fail(WQC_ERR_INVALID, "MPS bond layout mismatch during statevector projection");
        most = std::max(most, (size_t(2) << q) * size_t(dr[q]));
    }
    if (dr[n - 1] != 1) return fail(WQC_ERR_INVALID, "MPS bond layout mismatch during statevector projection");
    void *d_a = nullptr, *d_b = nullptr;
    if (wqc_status st = dmalloc(m, &d_a, most * sizeof(double2))) return st;
    if (wqc_status st = dmalloc(m, &d_b, most * sizeof(double2))) {
        dfree(m, d_a, most * sizeof(double2));
        return st;
    }
    double2* cur = static_cast<double2*>(d_a);
    double2* nxt = static_cast<double2*>(d_b);
    const double2 one = cmake(1.0, 0.0);
    cudaError_t e = cudaMemcpyAsync(cur, &one, sizeof(double2), cudaMemcpyHostToDevice, m->stream);
    const int prune = mode == WQC_DENSE_TO_DENSE_STATE ? 1 : 0;
    for (int q = 0; q < n && e == cudaSuccess; ++q) {
        const long prefix = 1L << q;
        const long total = 2 * prefix * dr[q];
        const int grid = int(std::min<long>((total + 255) / 256, 8L * m->ctx->sm_count));
        dense_step_kernel<<<grid, 256, 0, m->stream>>>(cur, m->site_ptr[q], dl[q], dr[q], prefix, prune, nxt);
        count_launch(m, -1);
        e = cudaGetLastError();
        std::swap(cur, nxt);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out, cur, (size_t(1) << n) * sizeof(double2), cudaMemcpyDeviceToHost, m->stream);
    m->stats.d2h_bytes += (size_t(1) << n) * sizeof(double2);
    wqc_status rc = e == cudaSuccess ? sync_status(m) : fail(WQC_ERR_CUDA, cudaGetErrorString(e));
    dfree(m, d_a, most * sizeof(double2));
    dfree(m, d_b, most * sizeof(double2));
    return rc;
}

wqc_status wqc_mps_bond_dims(wqc_mps* m, uint32_t* out) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (wqc_status s = sync_status(m)) return s;
    std::vector<int> dr(m->n);
    CUDA_TRY(cudaMemcpy(dr.data(), m->d_dr, m->n * sizeof(int), cudaMemcpyDeviceToHost));
    for (int i = 0; i < m->n; ++i) out[i] = uint32_t(dr[i]);
    return WQC_OK;
}

wqc_status wqc_mps_download_site(wqc_mps* m, uint32_t site, uint32_t* l, uint32_t* r, double* buf) {
    if (!m || !l || !r) return fail(WQC_ERR_INVALID, "null argument");
    if (site >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "site out of range");
    if (wqc_status s = sync_status(m)) return s;
    int dl = 0, dr = 0;
    CUDA_TRY(cudaMemcpy(&dl, m->d_dl + site, sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(&dr, m->d_dr + site, sizeof(int), cudaMemcpyDeviceToHost));
    *l = uint32_t(dl);
    *r = uint32_t(dr);
    if (buf)
        CUDA_TRY(cudaMemcpy(buf, m->site_ptr[site], size_t(dl) * 2 * dr * sizeof(double2),
                            cudaMemcpyDeviceToHost));
    return WQC_OK;
}

wqc_status wqc_mps_upload_site(wqc_mps* m, uint32_t site, uint32_t l, uint32_t r, const double* buf) {
    if (!m || !buf) return fail(WQC_ERR_INVALID, "null argument");
    if (site >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "site out of range");
    // Against the site's own capacity (a batch slice may have a smaller chi_max than the state).
    const uint32_t cap = uint32_t(m->site_chi[site]);
    if (l == 0 || r == 0 || l > cap || r > cap) return fail(WQC_ERR_INVALID, "site shape exceeds max_bond_dim");
    if (wqc_status s = sync_status(m)) return s;
    CUDA_TRY(cudaMemcpy(m->site_ptr[site], buf, size_t(l) * 2 * r * sizeof(double2), cudaMemcpyHostToDevice));
    const int il = int(l), ir = int(r);
    CUDA_TRY(cudaMemcpy(m->d_dl + site, &il, sizeof(int), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(m->d_dr + site, &ir, sizeof(int), cudaMemcpyHostToDevice));
    if (site > 0) m->ub[site - 1] = std::max(m->ub[site - 1], il);
    if (int(site) + 1 < m->n) m->ub[site] = std::max(m->ub[site], ir);
    m->uploaded = true;
    m->touch(int(site), int(site));
    return WQC_OK;
}

wqc_status wqc_mps_overlap(wqc_mps* ket, wqc_mps* bra, uint32_t env_limit, double out[2]) {
    if (!ket || !bra || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (ket->seg_first.size() != 1 || bra->seg_first.size() != 1)
        return fail(WQC_ERR_INVALID, "the overlap takes single states, not batches");
    if (ket->n != bra->n) return fail(WQC_ERR_INVALID, "mismatched register");  // EngineError::MismatchedRegister
    if (ket->ctx != bra->ctx) return fail(WQC_ERR_INVALID, "the two states live on different contexts");
    if (wqc_status s = sync_status(bra)) return s;
    if (wqc_status s = sync_status(ket)) return s;
    const int n = ket->n;
    std::vector<int> kdl(n), kdr(n), bdl(n), bdr(n);
    CUDA_TRY(cudaMemcpy(kdl.data(), ket->d_dl, n * sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(kdr.data(), ket->d_dr, n * sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(bdl.data(), bra->d_dl, n * sizeof(int), cudaMemcpyDeviceToHost));
    CUDA_TRY(cudaMemcpy(bdr.data(), bra->d_dr, n * sizeof(int), cudaMemcpyDeviceToHost));
    for (int q = 0; q < n; ++q) {
        if (kdl[q] != (q ? kdr[q - 1] : 1) || bdl[q] != (q ? bdr[q - 1] : 1))
            return fail(WQC_ERR_INVALID, "mps site shape does not match the overlap");
        if (env_limit && (unsigned long long)kdr[q] * bdr[q] > env_limit)  // mps.rs:1443-1448
            return fail(WQC_ERR_INVALID, "mps overlap environment exceeds " + std::to_string(env_limit));
    }
    const size_t env_bytes = size_t(ket->chi) * bra->chi * sizeof(double2);
    const size_t tmp_bytes = 2 * env_bytes;
    void *d_a = nullptr, *d_b = nullptr, *d_t = nullptr;
    auto release = [&]() {
        if (d_a) dfree(ket, d_a, env_bytes);
        if (d_b) dfree(ket, d_b, env_bytes);
        if (d_t) dfree(ket, d_t, tmp_bytes);
    };
    for (auto& pr : {std::make_pair(&d_a, env_bytes), std::make_pair(&d_b, env_bytes), std::make_pair(&d_t, tmp_bytes)})
        if (wqc_status st = dmalloc(ket, pr.first, pr.second)) {
            release();
            return st;
        }
    double2* env = static_cast<double2*>(d_a);
    double2* nxt = static_cast<double2*>(d_b);
    double2* tmp = static_cast<double2*>(d_t);
    const double2 one = cmake(1.0, 0.0);
    cudaError_t e = cudaMemcpyAsync(env, &one, sizeof(double2), cudaMemcpyHostToDevice, ket->stream);
    int kl = 1, bl = 1;
    for (int q = 0; q < n && e == cudaSuccess; ++q) {
        if (kdl[q] != kl || bdl[q] != bl) {
            e = cudaErrorInvalidValue;
            break;
        }
        const int kr = kdr[q], br = bdr[q];
        const long cap = 4L * ket->ctx->sm_count;
        overlap_half_kernel<<<int(std::min<long>((2L * bl * kr + 255) / 256, cap)), 256, 0, ket->stream>>>(
            env, kl, bl, ket->site_ptr[q], kr, tmp);
        overlap_next_kernel<<<int(std::min<long>((long(kr) * br + 255) / 256, cap)), 256, 0, ket->stream>>>(
            tmp, bl, kr, bra->site_ptr[q], br, nxt);
        count_launch(ket, -1);
        count_launch(ket, -1);
        std::swap(env, nxt);
        kl = kr;
        bl = br;
        e = cudaGetLastError();
    }
    double2 res = cmake(0, 0);
    wqc_status rc = WQC_OK;
    if (e == cudaErrorInvalidValue)
        rc = fail(WQC_ERR_INVALID, "mps site shape does not match the overlap");
    else if (e == cudaSuccess && (kl != 1 || bl != 1))
        rc = fail(WQC_ERR_INVALID, "mps overlap left an open bond");
    else if (e == cudaSuccess)
        e = cudaMemcpyAsync(&res, env, sizeof(double2), cudaMemcpyDeviceToHost, ket->stream);
    if (rc == WQC_OK) rc = e == cudaSuccess ? sync_status(ket) : fail(WQC_ERR_CUDA, cudaGetErrorString(e));
    release();
    if (rc != WQC_OK) return rc;
    out[0] = res.x;
    out[1] = res.y;
    return WQC_OK;
}

wqc_status wqc_mps_sample(wqc_mps* m, const uint32_t* qubits, uint32_t count, uint32_t shots, uint64_t seed,
                          uint64_t* out) {
    if (!m || (!qubits && count) || (!out && shots)) return fail(WQC_ERR_INVALID, "null argument");
    if (m->seg_first.size() != 1) return fail(WQC_ERR_INVALID, "sampling takes a single state, not a batch");
    if (count > 64) return fail(WQC_ERR_INVALID, "at most 64 measured qubits per shot");
    std::vector<int> bitpos(m->n, -1);
    for (uint32_t j = 0; j < count; ++j) {
        if (qubits[j] >= uint32_t(m->n)) return fail(WQC_ERR_QUBIT_OUT_OF_RANGE, "measured qubit out of range");
        if (bitpos[qubits[j]] >= 0) return fail(WQC_ERR_INVALID, "a qubit is listed twice");
        bitpos[qubits[j]] = int(j);
    }
    if (shots == 0) return WQC_OK;
    if (wqc_status s = check_uploaded_chain(m)) return s;
    if (wqc_status s = sync_status(m)) return s;
    const int n = m->n;
    // The right environments of the sites, chi^2 entries each, then H.  Where
    // that is more than is kept between reads, or than there is, site q's (dr[q]
    // x dr[q]) lies at env_at[q], which takes a copy of the bonds and a load a
    // step (0.14 ms of 6.5 for the reads of a 50-qubit state).
    int bond = m->chi;
    std::vector<unsigned long long> env_at;
    size_t entries = size_t(n) * bond * bond;
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t at_bytes = al(n * sizeof(unsigned long long)), bit_bytes = al((n + 1) * sizeof(int));
    const size_t out_bytes = size_t(shots) * sizeof(uint64_t);
    size_t env_bytes = 0;
    Scratch scratch(m);
    for (const ErrorState before;;) {
        env_bytes = al((entries + 2 * size_t(bond) * bond) * sizeof(double2));
        wqc_status st = WQC_ERR_OOM;
        if (!env_at.empty() || env_bytes <= kScratchKeep)
            st = scratch.get(env_bytes + at_bytes + bit_bytes + out_bytes);
        if (st == WQC_OK) {
            before.restore();
            break;
        }
        if (st != WQC_ERR_OOM || !env_at.empty()) return st;
        std::vector<int> bonds;
        if (wqc_status rs = read_bonds(m, bonds)) return rs;
        bond = *std::max_element(bonds.begin(), bonds.end());
        env_at.resize(n);
        entries = 0;
        for (int q = 0; q < n; ++q) {
            env_at[q] = entries;
            entries += size_t(bonds[n + q]) * bonds[n + q];
        }
    }
    double2* env = static_cast<double2*>(scratch.p);
    auto* at = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch.p) + env_bytes);
    const unsigned long long* d_at = env_at.empty() ? nullptr : at;
    int* d_bitpos = reinterpret_cast<int*>(reinterpret_cast<char*>(at) + at_bytes);
    auto* d_out = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(d_bitpos) + bit_bytes);
    bitpos.push_back(0);  // the chain's first site, after the bit positions
    CUDA_TRY(cudaMemcpyAsync(d_bitpos, bitpos.data(), (n + 1) * sizeof(int), cudaMemcpyHostToDevice, m->stream));
    if (d_at)
        CUDA_TRY(cudaMemcpyAsync(at, env_at.data(), n * sizeof(unsigned long long), cudaMemcpyHostToDevice, m->stream));
    EnvChains ch{};
    ch.base = env;
    ch.r_at = d_at;
    ch.h_off = entries;
    ch.firsts = d_bitpos + n;
    ch.nseg = 1;
    ch.width = n;
    ch.cap = bond;
    ch.left = false;
    int widest = 1;
    for (int b : m->ub) widest = std::max(widest, b);
    m->stats.total_launches += launch_env_chains(m->dev, ch, true, std::min(widest, bond), m->stream);
    const int grid = int(std::min<long>(long(shots), 8L * m->ctx->sm_count));
    const size_t smem = 3 * m->chi * sizeof(double2);
    if (d_at)
        sample_shots_kernel<true><<<grid, 256, smem, m->stream>>>(m->dev, env, d_at, d_bitpos, seed, int(shots), d_out);
    else
        sample_shots_kernel<false><<<grid, 256, smem, m->stream>>>(m->dev, env, d_at, d_bitpos, seed, int(shots), d_out);
    count_launch(m, -1);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(out, d_out, out_bytes, cudaMemcpyDeviceToHost, m->stream));
    m->stats.d2h_bytes += out_bytes;
    const wqc_status rc = sync_status(m);
    scratch.drained = rc != WQC_ERR_CUDA;
    return rc;
}

wqc_status wqc_mps_expectation_pauli(wqc_mps* m, const char* labels, const double* coeffs, uint32_t nterms,
                                     double out[2]) {
    if (!m || !labels || !coeffs || !out) return fail(WQC_ERR_INVALID, "null argument");
    for (size_t i = 0; i < size_t(nterms) * m->n; ++i) {
        const char ch = labels[i];
        if (ch != 'I' && ch != 'X' && ch != 'Y' && ch != 'Z')
            return fail(WQC_ERR_INVALID, std::string("invalid pauli character in label"));
    }
    if (nterms == 0) {
        out[0] = out[1] = 0;
        return WQC_OK;
    }
    if (wqc_status st = check_uploaded_chain(m)) return st;
    std::vector<double2> vals;
    if (wqc_status st = pauli_values(m, {0}, m->n, labels, nterms, vals)) return st;
    double re = 0, im = 0;
    for (uint32_t t = 0; t < nterms; ++t) {  // coeff * Re<P> (expectation.rs:177-185)
        const double v = vals[t].x;
        re += coeffs[2 * t] * v;
        im += coeffs[2 * t + 1] * v;
    }
    out[0] = re;
    out[1] = im;
    return WQC_OK;
}

wqc_status wqc_mps_debug_workspace(wqc_mps* m, uint32_t slot, int32_t which, void* out, uint64_t bytes) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    if (slot >= uint32_t(m->nslots)) return fail(WQC_ERR_INVALID, "slot out of range");
    if (wqc_status s = sync_status(m)) return s;
    SlotBuffers b;
    CUDA_TRY(cudaMemcpy(&b, m->d_slots + slot, sizeof(b), cudaMemcpyDeviceToHost));
    const void* src = nullptr;
    const int R = m->slot_R[slot], E = m->slot_E[slot];
    size_t cap = 0;
    switch (which) {
        case 0: src = b.theta; cap = size_t(R) * R * sizeof(double2); break;
        case 1: src = b.omega; cap = size_t(R) * E * sizeof(double2); break;
        case 2: src = b.y0; cap = size_t(R) * E * sizeof(double2); break;
        case 3: src = b.zr; cap = size_t(R) * E * sizeof(double2); break;
        case 4: src = b.y; cap = size_t(R) * E * sizeof(double2); break;
        case 5: src = b.q; cap = size_t(R) * E * sizeof(double2); break;
        case 6: src = b.b; cap = size_t(R) * E * sizeof(double2); break;
        case 7: src = b.w; cap = size_t(R) * R * sizeof(double2); break;
        case 8: src = b.z; cap = size_t(R) * R * sizeof(double2); break;
        case 9: src = b.sigma; cap = size_t(R) * sizeof(double); break;
        case 10: src = b.perm; cap = size_t(R) * sizeof(int); break;
        case 11: src = b.tau; cap = size_t(E) * sizeof(double2); break;
        case 12: src = m->d_state + slot; cap = sizeof(SplitState); break;
        default: return fail(WQC_ERR_INVALID, "unknown workspace buffer");
    }
    CUDA_TRY(cudaMemcpy(out, src, std::min<size_t>(cap, bytes), cudaMemcpyDeviceToHost));
    return WQC_OK;
}

uint32_t wqc_mps_split_count(wqc_mps* m) { return m ? m->rec_count : 0; }

wqc_status wqc_mps_split_records(wqc_mps* m, wqc_split_info* out, uint32_t max, uint32_t* written) {
    if (!m || (!out && max)) return fail(WQC_ERR_INVALID, "null argument");
    if (wqc_status s = sync_status(m)) return s;
    const uint32_t k = std::min(max, m->rec_count);
    if (k) CUDA_TRY(cudaMemcpy(out, m->d_records, k * sizeof(wqc_split_info), cudaMemcpyDeviceToHost));
    if (written) *written = k;
    return WQC_OK;
}

uint64_t wqc_mps_peak_vram_bytes(wqc_mps* m) { return m ? m->bytes_peak : 0; }

const char* wqc_mps_backend_label(wqc_mps*) { return "cuda"; }

wqc_status wqc_mps_set_profiling(wqc_mps* m, int32_t on) {
    if (!m) return fail(WQC_ERR_INVALID, "null argument");
    m->profiling = on != 0;
    return WQC_OK;
}

wqc_status wqc_mps_kernel_stats(wqc_mps* m, wqc_kernel_stats* out) {
    if (!m || !out) return fail(WQC_ERR_INVALID, "null argument");
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    for (auto& e : m->events) {
        float ms = 0;
        if (cudaEventElapsedTime(&ms, e.second.first, e.second.second) == cudaSuccess) m->stats.milliseconds[e.first] += ms;
        m->event_pool.push_back(e.second.first);
        m->event_pool.push_back(e.second.second);
    }
    m->events.clear();
    unsigned long long c[3] = {0, 0, 0};
    CUDA_TRY(cudaMemcpy(c, m->d_counters, sizeof(c), cudaMemcpyDeviceToHost));
    m->stats.jacobi_tasks = c[0];
    m->stats.jacobi_sweeps = c[1];
    m->stats.jacobi_sweeps_first = c[2];
    *out = m->stats;
    return WQC_OK;
}

void wqc_mps_reset_stats(wqc_mps* m) {
    if (!m) return;
    cudaStreamSynchronize(m->stream);
    for (auto& e : m->events) {
        m->event_pool.push_back(e.second.first);
        m->event_pool.push_back(e.second.second);
    }
    m->events.clear();
    m->stats = wqc_kernel_stats{};
    cudaMemset(m->d_counters, 0, 3 * sizeof(unsigned long long));
}

void* wqc_mps_stream(wqc_mps* m) { return m ? static_cast<void*>(m->stream) : nullptr; }

}  // extern "C"

// ===========================================================================
// Differentiation form: the adjoint (reverse-mode) gradient of a Pauli-sum
// observable with respect to the rotation angles of the gate list.
//
// Forward: the gate list runs on the state from |0...0> in segments; the
// sites (and bonds) at the start of every segment but the first, and at the
// end, are copied to checkpoints.  Backward: the site cotangents of the end
// state come from the observable's environments; then, segment by segment
// from the last, the segment's state is restored from its checkpoint and its
// operations are recomputed by steps of disjoint ones, the inputs each needs
// in reverse (the site before a one-qubit gate; the sites, theta and the
// Jacobi's W, singular values and order of a split) copied to a tape, and the
// tape is swept in reverse (adjoint_kernels.cu).  The split rule is the exact one on
// every split (a range finder seeded by a rank-48 test matrix has no
// meaningful derivative), and the plain FP64 form is required.
// ===========================================================================
struct wqc_adjoint {
    wqc_mps* m = nullptr;
    std::vector<wqc_gate> gates;
    std::vector<uint32_t> starts;  // segment starts; segment s is [starts[s], starts[s + 1] or count)
    size_t pool_bytes = 0;         // the state's site pool
    // checkpoint c (1 .. nseg - 1: segment starts; nseg: the end state):
    // site pool, then dl and dr
    std::vector<char*> cp;
    std::vector<std::vector<int>> cp_ub;
    uint32_t end_records = 0;
    bool forward_done = false;
};

namespace {

// d u / d angle of the rotations of gates.rs:10-66.
bool rotation_derivative(const wqc_gate& g, double2* du) {
    const double s = 0.5 * std::sin(g.angle / 2.0), c = 0.5 * std::cos(g.angle / 2.0);
    switch (g.kind) {
        case WQC_GATE_RX:
            du[0] = C(-s); du[1] = C(0, -c); du[2] = C(0, -c); du[3] = C(-s);
            return true;
        case WQC_GATE_RY:
            du[0] = C(-s); du[1] = C(-c); du[2] = C(c); du[3] = C(-s);
            return true;
        case WQC_GATE_RZ:
            du[0] = C(-s, -c); du[1] = C(0); du[2] = C(0); du[3] = C(-s, c);
            return true;
        default:
            return false;
    }
}

size_t adj_pool_bytes(const wqc_mps* m) { return size_t(m->n) * m->chi * 2 * m->chi * sizeof(double2); }

wqc_status adj_save(wqc_adjoint* a, size_t c) {
    wqc_mps* m = a->m;
    const size_t bytes = a->pool_bytes + 2 * size_t(m->n) * sizeof(int);
    if (!a->cp[c]) {
        void* p = nullptr;
        if (wqc_status st = dmalloc(m, &p, bytes)) return st;
        a->cp[c] = static_cast<char*>(p);
    }
    CUDA_TRY(cudaMemcpyAsync(a->cp[c], m->site_pool, a->pool_bytes, cudaMemcpyDeviceToDevice, m->stream));
    CUDA_TRY(cudaMemcpyAsync(a->cp[c] + a->pool_bytes, m->d_dl, size_t(m->n) * sizeof(int), cudaMemcpyDeviceToDevice,
                             m->stream));
    CUDA_TRY(cudaMemcpyAsync(a->cp[c] + a->pool_bytes + size_t(m->n) * sizeof(int), m->d_dr,
                             size_t(m->n) * sizeof(int), cudaMemcpyDeviceToDevice, m->stream));
    a->cp_ub[c] = m->ub;
    return WQC_OK;
}

wqc_status adj_restore(wqc_adjoint* a, size_t c) {
    wqc_mps* m = a->m;
    if (c == 0) {
        reset_sites_kernel<<<(m->n + 255) / 256, 256, 0, m->stream>>>(m->dev);
        CUDA_TRY(cudaGetLastError());
        std::fill(m->ub.begin(), m->ub.end(), 1);
    } else {
        CUDA_TRY(cudaMemcpyAsync(m->site_pool, a->cp[c], a->pool_bytes, cudaMemcpyDeviceToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(m->d_dl, a->cp[c] + a->pool_bytes, size_t(m->n) * sizeof(int),
                                 cudaMemcpyDeviceToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(m->d_dr, a->cp[c] + a->pool_bytes + size_t(m->n) * sizeof(int),
                                 size_t(m->n) * sizeof(int), cudaMemcpyDeviceToDevice, m->stream));
        m->ub = a->cp_ub[c];
    }
    m->lvalid = 0;
    m->rvalid = m->n - 1;
    return WQC_OK;
}

// Device buffers of one backward pass, freed together.
struct AdjBuffers {
    wqc_mps* m;
    std::vector<std::pair<void*, size_t>> owned;
    explicit AdjBuffers(wqc_mps* mm) : m(mm) {}
    ~AdjBuffers() {
        if (m->stream) cudaStreamSynchronize(m->stream);
        for (auto& p : owned) dfree(m, p.first, p.second);
    }
    template <class T>
    wqc_status get(T** out, size_t count) {
        void* p = nullptr;
        const size_t bytes = std::max<size_t>(count * sizeof(T), 16);
        if (wqc_status st = dmalloc(m, &p, bytes)) return st;
        owned.push_back({p, bytes});
        *out = static_cast<T*>(p);
        return WQC_OK;
    }
    void release(void* p) {
        for (size_t i = 0; i < owned.size(); ++i)
            if (owned[i].first == p) {
                cudaStreamSynchronize(m->stream);
                dfree(m, p, owned[i].second);
                owned.erase(owned.begin() + long(i));
                return;
            }
    }
};

// Operations of a segment that touch disjoint sites and are of one kind: they
// are recomputed, taped and reversed together.  A segment is a chain of steps
// and each is bound by the latency of one split, so what counts is how many
// there are: the 32-qubit ansatz, 6 layers at chi 64 with a checkpoint every 2
// (ladders, so two splits a step at most), took 52 ms one operation at a time
// and takes 31.
struct AdjStep {
    bool two;
    std::vector<size_t> ops;  // indices into the segment's operations
};

// An operation goes into the first step of its kind after the last one on its
// sites; at most `most` splits a step (each has a slot of its own).
std::vector<AdjStep> adj_steps(int n, const std::vector<Op>& ops, size_t most) {
    std::vector<AdjStep> steps, out;
    std::vector<size_t> next(n, 0);  // first step that a site is free in; odd steps hold splits
    for (size_t i = 0; i < ops.size(); ++i) {
        const Op& o = ops[i];
        size_t t = o.two ? std::max(next[o.site], next[o.site + 1]) : next[o.site];
        if ((t & 1) != size_t(o.two)) ++t;
        while (steps.size() <= t) steps.push_back({(steps.size() & 1) != 0, {}});
        steps[t].ops.push_back(i);
        next[o.site] = t + 1;
        if (o.two) next[o.site + 1] = t + 1;
    }
    for (const AdjStep& s : steps)
        for (size_t i = 0; i < s.ops.size();) {
            const size_t cnt = std::min(s.ops.size() - i, s.two ? most : s.ops.size());
            out.push_back({s.two, std::vector<size_t>(s.ops.begin() + long(i), s.ops.begin() + long(i + cnt))});
            i += cnt;
        }
    return out;
}

}  // namespace

extern "C" {

wqc_status wqc_adjoint_forward(wqc_mps* m, const wqc_gate* gates, uint32_t count, const uint32_t* checkpoints,
                               uint32_t ncheckpoints, wqc_adjoint** out) {
    if (!m || !out || (!gates && count) || (ncheckpoints && !checkpoints)) return fail(WQC_ERR_INVALID, "null argument");
    if (m->seg_first.size() != 1) return fail(WQC_ERR_INVALID, "the adjoint takes a single state, not a batch");
    if (m->fp32) return fail(WQC_ERR_INVALID, "the adjoint differentiates the plain FP64 form");
    Expander check;
    if (wqc_status st = expand(m->n, gates, count, false, check)) return st;
    auto* a = new wqc_adjoint();
    a->m = m;
    a->gates.assign(gates, gates + count);
    a->starts.push_back(0);
    std::vector<uint32_t> cps(checkpoints, checkpoints + ncheckpoints);
    std::sort(cps.begin(), cps.end());
    for (uint32_t c : cps)
        if (c > a->starts.back() && c < count) a->starts.push_back(c);
    a->pool_bytes = adj_pool_bytes(m);
    a->cp.assign(a->starts.size() + 1, nullptr);
    a->cp_ub.resize(a->starts.size() + 1);
    const bool rule = m->exact_only;
    m->exact_only = true;
    m->direct_svd = true;
    wqc_status st = wqc_mps_reset(m);
    for (size_t sgi = 0; sgi < a->starts.size() && st == WQC_OK; ++sgi) {
        if (sgi > 0) st = adj_save(a, sgi);
        const uint32_t g0 = a->starts[sgi], g1 = sgi + 1 < a->starts.size() ? a->starts[sgi + 1] : count;
        if (st == WQC_OK && g1 > g0) {
            Expander ex;
            st = expand(m->n, a->gates.data() + g0, g1 - g0, false, ex);
            if (st == WQC_OK) st = run_ops(m, ex.ops);
        }
    }
    if (st == WQC_OK) st = adj_save(a, a->starts.size());
    if (st == WQC_OK) st = sync_status(m);
    m->exact_only = rule;
    m->direct_svd = false;
    a->end_records = m->rec_count;
    if (st != WQC_OK) {
        wqc_adjoint_destroy(a);
        return st;
    }
    a->forward_done = true;
    *out = a;
    return WQC_OK;
}

wqc_status wqc_adjoint_backward(wqc_adjoint* a, const char* labels, const double* coeffs, uint32_t nterms,
                                double value[2], double* grad) {
    if (!a || !a->forward_done || !labels || !coeffs || !value || (!grad && !a->gates.empty()))
        return fail(WQC_ERR_INVALID, "null argument");
    wqc_mps* m = a->m;
    const int n = m->n, chi = m->chi, R = 2 * chi;
    for (size_t i = 0; i < size_t(nterms) * n; ++i) {
        const char ch = labels[i];
        if (ch != 'I' && ch != 'X' && ch != 'Y' && ch != 'Z')
            return fail(WQC_ERR_INVALID, std::string("invalid pauli character in label"));
    }
    if (nterms == 0) return fail(WQC_ERR_INVALID, "the adjoint needs at least one Pauli term");
    CUDA_TRY(cudaSetDevice(m->ctx->device));
    const bool rule = m->exact_only;
    m->exact_only = true;
    m->direct_svd = true;
    struct RuleGuard {
        wqc_mps* m;
        bool rule;
        ~RuleGuard() {
            m->exact_only = rule;
            m->direct_svd = false;
        }
    } guard{m, rule};
    AdjBuffers buf(m);
    const size_t site_cap = size_t(chi) * 2 * chi;
    // Cotangent sites, one per site at the state's capacity, and their pointers.
    double2* bar_pool = nullptr;
    double2** d_bars = nullptr;
    if (wqc_status st = buf.get(&bar_pool, site_cap * n)) return st;
    if (wqc_status st = buf.get(&d_bars, n)) return st;
    std::vector<double2*> bars(n);
    for (int q = 0; q < n; ++q) bars[q] = bar_pool + site_cap * q;
    CUDA_TRY(cudaMemcpyAsync(d_bars, bars.data(), n * sizeof(double2*), cudaMemcpyHostToDevice, m->stream));
    // The end state and the observable's environments, values and cotangents.
    if (wqc_status st = adj_restore(a, a->starts.size())) return st;
    {
        const size_t E = size_t(chi) * chi;
        char* d_lab = nullptr;
        double* d_cre = nullptr;
        double2 *envs = nullptr, *tmp = nullptr, *vals = nullptr;
        if (wqc_status st = buf.get(&d_lab, size_t(nterms) * n + 16)) return st;
        if (wqc_status st = buf.get(&vals, nterms + (size_t(nterms) + 1) / 2)) return st;
        d_cre = reinterpret_cast<double*>(vals + nterms);
        if (wqc_status st = buf.get(&envs, size_t(nterms) * (2 * n + 1) * E)) return st;
        // Half-products of both directions, or of one after the other where
        // the device has no room for both.
        int dirs = 2;
        for (const ErrorState before;; dirs = 1) {
            const wqc_status st = buf.get(&tmp, size_t(nterms) * 2 * dirs * E);
            if (st == WQC_OK) {
                before.restore();
                break;
            }
            if (st != WQC_ERR_OOM || dirs == 1) return st;
        }
        std::vector<double> cre(nterms);
        for (uint32_t t = 0; t < nterms; ++t) cre[t] = coeffs[2 * t];
        CUDA_TRY(cudaMemcpyAsync(d_lab, labels, size_t(nterms) * n, cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(d_cre, cre.data(), nterms * sizeof(double), cudaMemcpyHostToDevice, m->stream));
        int bond = 1;
        for (int b : m->ub) bond = std::max(bond, b);
        const unsigned b1 = unsigned(bond + kTile - 1) / kTile, b2 = unsigned(2 * bond + kTile - 1) / kTile;
        for (int dir = 0; dir < 2; dir += dirs)
            for (int step = 0; step < n; ++step)
                for (int phase = 0; phase < 2; ++phase) {
                    const unsigned t = phase == 0 ? b2 : b1;
                    adj_pauli_envs_kernel<<<dim3(dirs * nterms, t, t), kTileThreads, 0, m->stream>>>(
                        m->dev, d_lab, chi, dirs, dir, step, phase, envs, tmp);
                    count_launch(m, -1);
                }
        // Holes in chunks of terms, accumulated in term order.  Allocated while
        // the environments are worked out (0.6 ms), and in their half-products'
        // place where the device has no room beside these.
        const size_t per_term = 2 * size_t(n) * site_cap * sizeof(double2);
        const int chunk = int(std::max<size_t>(1, std::min<size_t>(16, (size_t(1) << 30) / per_term)));
        double2 *holes = nullptr, *htmp = nullptr;
        for (double2** p : {&holes, &htmp}) {
            const ErrorState before;
            wqc_status st = buf.get(p, size_t(chunk) * n * site_cap);
            if (st == WQC_ERR_OOM && tmp) {
                buf.release(tmp);
                tmp = nullptr;
                st = buf.get(p, size_t(chunk) * n * site_cap);
                if (st == WQC_OK) before.restore();
            }
            if (st != WQC_OK) return st;
        }
        const int agrid = int(std::max<size_t>(1, std::min<size_t>((site_cap + 255) / 256, 64)));
        for (uint32_t t0 = 0; t0 < nterms; t0 += uint32_t(chunk)) {
            const int cnt = int(std::min<uint32_t>(uint32_t(chunk), nterms - t0));
            adj_pauli_holes_kernel<<<dim3(n * cnt, b1, b2), kTileThreads, 0, m->stream>>>(m->dev, d_lab, int(t0), chi, 0,
                                                                                          envs, htmp, holes);
            adj_pauli_holes_kernel<<<dim3(n * cnt, b2, b1), kTileThreads, 0, m->stream>>>(m->dev, d_lab, int(t0), chi, 1,
                                                                                          envs, htmp, holes);
            count_launch(m, -1);
            adj_pauli_accumulate_kernel<<<dim3(agrid, n), 256, 0, m->stream>>>(m->dev, d_bars, holes, d_cre, int(t0),
                                                                             cnt, chi, t0 == 0 ? 1 : 0);
            count_launch(m, -1);
            count_launch(m, -1);
        }
        const unsigned vgrid = std::min((nterms + 255) / 256, 1024u);
        adj_pauli_values_kernel<<<vgrid, 256, 0, m->stream>>>(envs, n, chi, int(nterms), vals);
        count_launch(m, -1);
        CUDA_TRY(cudaGetLastError());
        std::vector<double2> hv(nterms);
        CUDA_TRY(cudaMemcpyAsync(hv.data(), vals, nterms * sizeof(double2), cudaMemcpyDeviceToHost, m->stream));
        CUDA_TRY(cudaStreamSynchronize(m->stream));
        double re = 0, im = 0;
        for (uint32_t t = 0; t < nterms; ++t) {  // coeff * Re<P> (expectation.rs:177-185), term order
            re += coeffs[2 * t] * hv[t].x;
            im += coeffs[2 * t + 1] * hv[t].x;
        }
        value[0] = re;
        value[1] = im;
        buf.release(envs);
        if (tmp) buf.release(tmp);
        buf.release(holes);
        buf.release(htmp);
    }
    // Gradient slots: one per one-qubit operation of the whole list.
    Expander all;
    if (wqc_status st = expand(n, a->gates.data(), uint32_t(a->gates.size()), false, all)) return st;
    size_t n1q = 0;
    for (const Op& o : all.ops) n1q += o.two ? 0 : 1;
    double* d_grad = nullptr;
    if (wqc_status st = buf.get(&d_grad, n1q + 1)) return st;
    CUDA_TRY(cudaMemsetAsync(d_grad, 0, (n1q + 1) * sizeof(double), m->stream));
    std::vector<int> slot_gate;  // gate of each gradient slot
    // Split workspaces (ten column-major R x R matrices each), for as many
    // splits of a step at a time as fit 256 MiB, or else what the tape leaves of
    // the device: a circuit of ladders has about half a segment's layers in a step.
    const size_t RR = size_t(R) * R, ws_b = (10 * RR) * sizeof(double2) + 2 * size_t(R) * sizeof(double);
    const size_t most = size_t(std::min(m->bucket_cap[0], 32768));
    char* ws = nullptr;
    size_t width = std::max<size_t>(1, std::min(most, (size_t(256) << 20) / ws_b));
    auto get_ws = [&]() -> wqc_status {
        const ErrorState before;
        for (;; width /= 2) {
            const wqc_status st = buf.get(&ws, width * ws_b);
            if (st == WQC_OK) {
                before.restore();
                return st;
            }
            if (st != WQC_ERR_OOM || width == 1) return st;
        }
    };
    if (wqc_status st = get_ws()) return st;
    // Tape layout of one operation (bytes, 256-aligned parts).
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    AdjTapeLayout L{};
    L.site_b = al(site_cap * sizeof(double2));
    L.theta_off = 2 * L.site_b;
    L.w_off = L.theta_off + al(RR * sizeof(double2));
    L.sigma_off = L.w_off + al(RR * sizeof(double2));
    L.perm_off = L.sigma_off + al(R * sizeof(double));
    L.state_off = L.perm_off + al(R * sizeof(int));
    const size_t one_b = L.site_b + al(2 * sizeof(int));
    const size_t two_b = L.state_off + al(sizeof(SplitState));
    char* tape = nullptr;
    size_t tape_cap = 0;
    // First gradient slot of each segment (one-qubit operations in program order).
    std::vector<size_t> seg_slot0(a->starts.size());
    {
        size_t acc = 0;
        for (size_t sgi = 0; sgi < a->starts.size(); ++sgi) {
            seg_slot0[sgi] = acc;
            const uint32_t g1 = sgi + 1 < a->starts.size() ? a->starts[sgi + 1] : uint32_t(a->gates.size());
            for (const Op& o : all.ops)
                if (!o.two && o.gate >= int(a->starts[sgi]) && o.gate < int(g1)) ++acc;
        }
        for (const Op& o : all.ops)
            if (!o.two) slot_gate.push_back(o.gate);
    }
    const int eg = int(std::min<long>((long(R) * R + 255) / 256, 4L * m->ctx->sm_count));
    for (size_t sgi = a->starts.size(); sgi-- > 0;) {
        const uint32_t g0 = a->starts[sgi];
        const uint32_t g1 = sgi + 1 < a->starts.size() ? a->starts[sgi + 1] : uint32_t(a->gates.size());
        if (g1 <= g0) continue;
        Expander ex;
        if (wqc_status st = expand(n, a->gates.data() + g0, g1 - g0, false, ex)) return st;
        // The tape: every operation's data, then the steps' descriptors.
        const std::vector<AdjStep> steps = adj_steps(n, ex.ops, most);
        size_t nops[2] = {0, 0}, data_b = 0;
        for (const Op& o : ex.ops) {
            ++nops[o.two];
            data_b += o.two ? two_b : one_b;
        }
        const size_t tape_off = data_b, split_off = tape_off + al(ex.ops.size() * sizeof(AdjTape));
        const size_t one_off = split_off + al(nops[1] * sizeof(AdjSplit));
        const size_t need = one_off + al(nops[0] * sizeof(Adj1q));
        if (need > tape_cap) {
            if (tape) buf.release(tape);
            tape = nullptr;
            tape_cap = 0;
            // The tape comes before workspaces for more than one split.
            for (const ErrorState before;;) {
                const wqc_status st = buf.get(&tape, need);
                if (st == WQC_OK) {
                    before.restore();
                    break;
                }
                if (st != WQC_ERR_OOM || width == 1) return st;
                buf.release(ws);
                width /= 2;
                if (wqc_status ws_st = get_ws()) return ws_st;
            }
            tape_cap = need;
        }
        std::vector<size_t> slot_of(ex.ops.size());
        for (size_t i = 0, sl = seg_slot0[sgi]; i < ex.ops.size(); ++i) slot_of[i] = ex.ops[i].two ? 0 : sl++;
        std::vector<AdjTape> tapes;
        std::vector<AdjSplit> splits;
        std::vector<Adj1q> ones;
        char* base = tape;
        for (const AdjStep& s : steps)
            for (size_t i = 0; i < s.ops.size(); ++i) {
                const Op& o = ex.ops[s.ops[i]];
                tapes.push_back({base, o.site});
                if (!o.two) {
                    Adj1q g{};
                    std::memcpy(g.u, o.m2.u, sizeof(g.u));
                    g.has_du = rotation_derivative(a->gates[o.gate + int(g0)], g.du) ? 1 : 0;
                    g.slot = int(slot_of[s.ops[i]]);
                    g.bar = bars[o.site];
                    g.before = reinterpret_cast<const double2*>(base);
                    g.dims = reinterpret_cast<const int*>(base + L.site_b);
                    ones.push_back(g);
                    base += one_b;
                    continue;
                }
                AdjSplit A{};
                A.site_l = reinterpret_cast<const double2*>(base);
                A.site_r = reinterpret_cast<const double2*>(base + L.site_b);
                A.theta = reinterpret_cast<const double2*>(base + L.theta_off);
                A.w = reinterpret_cast<const double2*>(base + L.w_off);
                A.sigma = reinterpret_cast<const double*>(base + L.sigma_off);
                A.perm = reinterpret_cast<const int*>(base + L.perm_off);
                A.st = reinterpret_cast<const SplitState*>(base + L.state_off);
                A.bar_l = bars[o.site];
                A.bar_r = bars[o.site + 1];
                std::memcpy(A.u, o.ueff, sizeof(A.u));
                double2* w = reinterpret_cast<double2*>(ws + (i % width) * ws_b);
                A.U = w; A.V = w + RR; A.Ub = w + 2 * RR; A.Vb = w + 3 * RR; A.M = w + 4 * RR; A.Nm = w + 5 * RR;
                A.Z = w + 6 * RR; A.T1 = w + 7 * RR; A.tb = w + 8 * RR; A.tb0 = w + 9 * RR;
                A.inv = reinterpret_cast<double*>(w + 10 * RR);
                A.sq = A.inv + R;
                A.R = R;
                splits.push_back(A);
                base += two_b;
            }
        const AdjTape* d_tapes = reinterpret_cast<const AdjTape*>(tape + tape_off);
        const AdjSplit* d_splits = reinterpret_cast<const AdjSplit*>(tape + split_off);
        const Adj1q* d_ones = reinterpret_cast<const Adj1q*>(tape + one_off);
        CUDA_TRY(cudaMemcpyAsync(tape + tape_off, tapes.data(), tapes.size() * sizeof(AdjTape), cudaMemcpyHostToDevice,
                                 m->stream));
        CUDA_TRY(cudaMemcpyAsync(tape + split_off, splits.data(), splits.size() * sizeof(AdjSplit),
                                 cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(tape + one_off, ones.data(), ones.size() * sizeof(Adj1q), cudaMemcpyHostToDevice,
                                 m->stream));
        // Recompute the segment step by step, taping each one's inputs.
        if (wqc_status st = adj_restore(a, sgi)) return st;
        std::vector<Op> step_ops;
        size_t first = 0;
        for (const AdjStep& s : steps) {
            step_ops.clear();
            int bond = 1;
            for (size_t i : s.ops) {
                const Op& o = ex.ops[i];
                step_ops.push_back(o);
                bond = std::max(std::max(bond, m->left_bond(o.site)), m->right_bond(o.site));
                if (o.two) bond = std::max(bond, m->right_bond(o.site + 1));
            }
            const unsigned cnt = unsigned(s.ops.size());
            auto parts = [&](long entries) { return unsigned(std::max(1L, std::min(16L, entries / 1024))); };
            adj_tape_before_kernel<<<dim3(cnt, parts(2L * bond * bond)), 256, 0, m->stream>>>(m->dev, d_tapes + first, L,
                                                                                            s.two ? 1 : 0);
            count_launch(m, -1);
            if (wqc_status st = run_ops(m, step_ops)) return st;
            if (s.two) {
                adj_tape_after_kernel<<<dim3(cnt, parts(4L * bond * bond)), 256, 0, m->stream>>>(m->d_state, m->d_slots,
                                                                                               d_tapes + first, L);
                count_launch(m, -1);
            }
            first += s.ops.size();
        }
        // Reverse sweep over the segment.
        size_t at[2] = {nops[0], nops[1]};
        for (size_t k = steps.size(); k-- > 0;) {
            const unsigned all_of = unsigned(steps[k].ops.size());
            at[steps[k].two] -= all_of;
            if (!steps[k].two) {
                adj_one_qubit_kernel<<<all_of, 256, 0, m->stream>>>(d_ones + at[0], d_grad);
                count_launch(m, -1);
                continue;
            }
            for (unsigned i = 0; i < all_of; i += unsigned(width)) {
                const unsigned cnt = std::min(unsigned(width), all_of - i);
                const AdjSplit* A = d_splits + at[1] + i;
                const dim3 ge(eg, cnt), gg((R + kTile - 1) / kTile, (R + kTile - 1) / kTile, cnt);
                adj_split_prep_kernel<<<ge, 256, 0, m->stream>>>(A);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageOther);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageM);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageN);
                adj_split_assemble_kernel<<<ge, 256, 0, m->stream>>>(A);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageT1);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageTb);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageTb2);
                adj_split_gate_kernel<<<ge, 256, 0, m->stream>>>(A);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageBarL);
                adj_split_gemm_kernel<<<gg, kTileThreads, 0, m->stream>>>(A, kAdjStageBarR);
                for (int c = 0; c < 11; ++c) count_launch(m, -1);
            }
        }
        CUDA_TRY(cudaGetLastError());
    }
    std::vector<double> hg(n1q + 1);
    CUDA_TRY(cudaMemcpyAsync(hg.data(), d_grad, (n1q + 1) * sizeof(double), cudaMemcpyDeviceToHost, m->stream));
    if (wqc_status st = sync_status(m)) return st;
    for (size_t i = 0; i < a->gates.size(); ++i) grad[i] = 0.0;
    for (size_t sl = 0; sl < n1q; ++sl) grad[slot_gate[sl]] += hg[sl];
    // The state holds the end state again; its records are the forward's.
    if (wqc_status st = adj_restore(a, a->starts.size())) return st;
    m->rec_count = a->end_records;
    return sync_status(m);
}

void wqc_adjoint_destroy(wqc_adjoint* a) {
    if (!a) return;
    if (a->m) {
        if (a->m->stream) cudaStreamSynchronize(a->m->stream);
        const size_t bytes = a->pool_bytes + 2 * size_t(a->m->n) * sizeof(int);
        for (char* p : a->cp) dfree(a->m, p, bytes);
    }
    delete a;
}

}  // extern "C"

// ===========================================================================
// Autotuner of the Jacobi SVD's cluster size, with a fingerprinted cache (the
// pattern of the reference's GEMM side calibration, src/tn/gpu/gemm.rs:
// 495-543, 649-702: measure once per machine, keep the result in a file keyed
// by what the measurement depends on, reuse it on later starts).
//
// For every saturated shape of the configured chi_max values (2 chi x 2 chi,
// chi in 16, 32, 64, 128), in the plain form and in the precision form's
// first phase, and for both kinds of wave -- one latency-bound split, and a
// batch of 32 splits that fills the device -- each cluster size whose shared
// memory fits is timed on seeded random sites (Jacobi kernel time from the
// state's CUDA events, best of three) and the fastest is kept.  Shapes the
// table does not hold keep the cost model of choose_cluster.
// ===========================================================================
namespace {

constexpr int kTuneVersion = 1;

std::string tune_fingerprint(const wqc_cuda_ctx* ctx) {
    cudaDeviceProp prop{};
    cudaGetDeviceProperties(&prop, ctx->device);
    int drv = 0, rt = 0;
    cudaDriverGetVersion(&drv);
    cudaRuntimeGetVersion(&rt);
    std::string name(prop.name);
    for (char& c : name)
        if (c == '|' || c == '\n' || c == '\r') c = ' ';
    return "wqc-jacobi-clusters v" + std::to_string(kTuneVersion) + "|" + name + "|sm=" +
           std::to_string(prop.multiProcessorCount) + "|cc=" + std::to_string(prop.major) + "." +
           std::to_string(prop.minor) + "|driver=" + std::to_string(drv) + "|runtime=" + std::to_string(rt) +
           "|max_cluster=" + std::to_string(ctx->max_cluster) + "|jacobi=ring,qr";
}

std::string tune_cache_path(const char* path) {
    if (path && *path) return path;
    if (const char* p = std::getenv("WQC_TUNE_PATH")) return p;
    std::string base;
    if (const char* x = std::getenv("XDG_CACHE_HOME"))
        base = x;
    else if (const char* h = std::getenv("HOME"))
        base = std::string(h) + "/.cache";
    else
        base = ".";
    return base + "/wqc/jacobi-clusters";
}

bool tune_read(const std::string& path, const std::string& fp, std::vector<wqc_cuda_ctx::Tuned>& out) {
    FILE* f = std::fopen(path.c_str(), "r");
    if (!f) return false;
    char line[512];
    bool ok = std::fgets(line, sizeof(line), f) != nullptr;
    if (ok) {
        std::string first(line);
        while (!first.empty() && (first.back() == '\n' || first.back() == '\r')) first.pop_back();
        ok = first == fp;
    }
    std::vector<wqc_cuda_ctx::Tuned> t;
    while (ok && std::fgets(line, sizeof(line), f)) {
        wqc_cuda_ctx::Tuned e{};
        if (std::sscanf(line, "%d %d %d %d %d %d", &e.M, &e.N, &e.len, &e.elem, &e.throughput, &e.C) == 6 && e.C >= 1)
            t.push_back(e);
    }
    std::fclose(f);
    if (ok) out = t;
    return ok;
}

bool tune_write(const std::string& path, const std::string& fp, const std::vector<wqc_cuda_ctx::Tuned>& t) {
    const size_t slash = path.find_last_of('/');
    if (slash != std::string::npos) {  // create the parent directories
        std::string dir = path.substr(0, slash);
        for (size_t i = 1; i <= dir.size(); ++i)
            if (i == dir.size() || dir[i] == '/') {
                const std::string part = dir.substr(0, i);
                if (!part.empty()) mkdir(part.c_str(), 0755);
            }
    }
    const std::string tmp = path + ".tmp";
    FILE* f = std::fopen(tmp.c_str(), "w");
    if (!f) return false;
    std::fprintf(f, "%s\n", fp.c_str());
    for (const auto& e : t) std::fprintf(f, "%d %d %d %d %d %d\n", e.M, e.N, e.len, e.elem, e.throughput, e.C);
    const bool ok = std::fclose(f) == 0;
    return ok && std::rename(tmp.c_str(), path.c_str()) == 0;
}

// Seeded random complex entries in [-1, 1) (xorshift64*).
void fill_random(std::vector<double>& v, unsigned long long& state) {
    for (double& x : v) {
        state ^= state >> 12;
        state ^= state << 25;
        state ^= state >> 27;
        x = double((state * 2685821657736338717ull) >> 11) * (2.0 / 9007199254740992.0) - 1.0;
    }
}

// Jacobi milliseconds of one wave of `count` exact 2chi x 2chi splits at the
// cluster size the context forces (best of `reps`); < 0 on failure.
double tune_measure(wqc_cuda_ctx* ctx, int chi, int precision, int count, int reps) {
    std::vector<uint32_t> qs(count, 4), chis(count, uint32_t(chi));
    wqc_mps* m = nullptr;
    if (wqc_batch_create(ctx, uint32_t(count), qs.data(), chis.data(), precision, 0, &m) != WQC_OK) return -1.0;
    if (count == 1) m->batch = false;  // one split: the latency-bound kind of wave
    m->exact_only = true;
    unsigned long long rng = 0x9E3779B97F4A7C15ull ^ (unsigned long long)(chi * 131 + count);
    const int dims[4][2] = {{1, chi}, {chi, chi}, {chi, chi}, {chi, 1}};
    std::vector<double> buf;
    double best = -1.0;
    for (int rep = 0; rep <= reps; ++rep) {
        wqc_mps_reset(m);
        for (int sl = 0; sl < count; ++sl)
            for (int q = 0; q < 4; ++q) {
                buf.assign(size_t(dims[q][0]) * 2 * dims[q][1] * 2, 0.0);
                fill_random(buf, rng);
                if (wqc_mps_upload_site(m, uint32_t(sl * 4 + q), uint32_t(dims[q][0]), uint32_t(dims[q][1]),
                                        buf.data()) != WQC_OK) {
                    wqc_mps_destroy(m);
                    return -1.0;
                }
            }
        std::vector<wqc_gate> gates(count);
        std::vector<uint32_t> offs(count + 1);
        for (int sl = 0; sl < count; ++sl) {
            gates[sl] = wqc_gate{WQC_GATE_CZ, 1, 2, 0, 0.0};
            offs[sl] = uint32_t(sl);
        }
        offs[count] = uint32_t(count);
        wqc_mps_reset_stats(m);
        wqc_mps_set_profiling(m, rep > 0 ? 1 : 0);  // rep 0 warms up
        wqc_status st = wqc_batch_apply_gates(m, gates.data(), offs.data());
        wqc_kernel_stats ks{};
        if (st == WQC_OK) st = wqc_mps_synchronize(m);
        if (st == WQC_OK) st = wqc_mps_kernel_stats(m, &ks);
        if (st != WQC_OK) {
            wqc_mps_destroy(m);
            return -1.0;
        }
        if (rep > 0 && (best < 0 || ks.milliseconds[0] < best)) best = ks.milliseconds[0];
    }
    wqc_mps_destroy(m);
    return best;
}

}  // namespace

extern "C" {

wqc_status wqc_cuda_autotune(wqc_cuda_ctx* ctx, const char* cache_path, double budget_seconds, uint32_t* entries) {
    if (!ctx) return fail(WQC_ERR_INVALID, "null context");
    CUDA_TRY(cudaSetDevice(ctx->device));
    const std::string fp = tune_fingerprint(ctx);
    const std::string path = tune_cache_path(cache_path);
    std::vector<wqc_cuda_ctx::Tuned> table;
    if (tune_read(path, fp, table)) {
        ctx->tuned = table;
        if (entries) *entries = uint32_t(table.size());
        return WQC_OK;
    }
    const auto t0 = std::chrono::steady_clock::now();
    auto elapsed = [&]() {
        return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    };
    ctx->tuned.clear();
    for (int precision : {WQC_PRECISION_FP64, WQC_PRECISION_FP32}) {
        for (int chi : {16, 32, 64, 128}) {
            for (int throughput : {0, 1}) {
                if (budget_seconds > 0 && elapsed() > budget_seconds) break;
                const int M = 2 * chi, N = 2 * chi;
                const size_t elem = precision == WQC_PRECISION_FP32 ? sizeof(float2) : sizeof(double2);
                const int len = precision == WQC_PRECISION_FP32 ? M + N : M;
                int best_c = 0;
                double best_ms = 0.0;
                for (int c = 1; c <= std::min(ctx->max_cluster, kJacobiRingMaxCluster); c *= 2) {
                    RingShape shape;
                    if (!ring_shape(M, N, len - M, elem, c, &shape)) continue;
                    ctx->force_C = c;
                    const double ms = tune_measure(ctx, chi, precision, throughput ? 32 : 1, 3);
                    ctx->force_C = 0;
                    if (ms < 0) {
                        ctx->tuned.clear();
                        return fail(WQC_ERR_CUDA, std::string("autotune measurement failed: ") + g_err);
                    }
                    // A batch is throughput-bound: SM time (ms x C) decides.
                    const double cost = throughput ? ms * c : ms;
                    if (!best_c || cost < best_ms) {
                        best_c = c;
                        best_ms = cost;
                    }
                }
                if (best_c) ctx->tuned.push_back({M, N, len, int(elem), throughput, best_c});
            }
        }
    }
    tune_write(path, fp, ctx->tuned);  // a cache that cannot be written only costs the next start a measurement
    if (entries) *entries = uint32_t(ctx->tuned.size());
    return WQC_OK;
}

}  // extern "C"
