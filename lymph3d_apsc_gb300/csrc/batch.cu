// batch.cu -- many independent problems advanced by one persistent launch
// per time step (no counterpart in the reference, which runs one problem
// per MPI job).
//
// Every problem keeps its own context (operator blocks, mass inverse, RHS,
// state, degree, dt); the batch flattens all (problem, polyhedron) pairs
// into one work list.  A persistent grid of CTAs pulls items from an atomic
// queue and runs the same per-polyhedron body as the single-problem kernel
// (step_body.cuh) with the degree of the item's problem, so results are
// bit-identical to stepping each context alone.  A step's index (which selects
// each problem's buffer parity and time-function value) is the step counter
// plus its place in the graph; a 1-thread kernel beside each step clears the
// next one's queue and the graph's last one moves the counter on.  The loop is
// launched as CUDA graphs of 16 steps.  The grid size and the item order (largest
// cost first or problem-major) are picked by a timing autotuner whose choice
// is cached per batch signature.  The autotuner also picks the tile shape:
// the number of column slices S per degree (kBatchShapes).  Shape 0, the
// default before tuning, is the single-problem kernel's, so results are then
// bit-identical to stepping each context alone; the other shapes group the
// row's partial sums differently (deterministic, equal to rounding).  On the
// matrix-free path (mf.cu) the items are grouped by degree and each degree
// present gets its own persistent launch per step, side by side, so every
// degree runs with its own register and shared-memory budget.

#include <algorithm>
#include <cstdlib>
#include <filesystem>
#include <fstream>
#include <map>
#include <mutex>
#include <numeric>
#include <sstream>
#include <string>
#include <vector>

#include "step_body.cuh"

using namespace stepk;

size_t lymph_mf_batch_problem_bytes();
int lymph_mf_batch_ctas_per_sm(int p);
void lymph_mf_batch_problem(const lymph_ctx* c, int* status, void* out);
int lymph_mf_batch_u32(cudaStream_t st, const void* probs, const int2* items, int n_items, const int64_t* step_idx,
                       int step_off);
int lymph_mf_batch_step(const cudaStream_t* st, const int* grid, const void* probs, const int2* items, const int* off,
                        int* queue, const int64_t* step_idx, int step_off, const double* gvals, int64_t g_stride,
                        int* launched);

namespace {

constexpr int BATCH_THREADS = 320;   // the p = 4 shape; lower degrees leave lanes idle
constexpr int BATCH_MINB = 4;
// A row's head is prefetched before its coefficients are gathered where that pays: in
// batches of p = 1 and 2 alone, and from 3.4 GB of blocks per step on but for FP32 at p = 4
// (profitable side first, 48 steps; problems of 3^3..8^3 x 6: p = 2 in FP32 3.17 against 3.77 ms,
// p = 1 in FP64 2.42 against 2.63, degrees 1 to 4 in FP32 without 13.5 against 14.0; of
// 14^3..26^3, degrees 1 to 4 in FP32, 148.4 against 153.7).
constexpr int64_t BATCH_PREFETCH_MIN = 3400000000ll;
constexpr int BATCH_QUEUES = 4;      // item counters: one per degree on the matrix-free path

struct BatchProblem {
    StepArgs a;        // per-problem pointers; u0/un/out are filled per step
    double* buf[2];
    int cur0;          // buffer parity of the problem when the run started
    int p;
};

// Tile shapes the autotuner chooses from: column slices S for p = 1..4
// (index 0 unused); every ND * S fits the CTA's 320 threads.
constexpr int BATCH_SHAPES = 3;
constexpr int kBatchShapes[BATCH_SHAPES][5] = {{0, 8, 8, 4, 3}, {0, 16, 10, 5, 3}, {0, 24, 10, 5, 2}};

constexpr size_t zmax(size_t a, size_t b) { return a > b ? a : b; }
// FP64 problems of p = 2 have their integer columns in shape 0 alone (the others group a
// row's sums in another way than a lone problem anyway, and are faster without).
constexpr bool batch_int2(size_t elem, int shape) { return elem == 8 && shape == 0; }
template <typename KT, int V, bool HIGH> struct BatchSmem {
    static constexpr size_t low =
        zmax(SmemSize<1, KT, kBatchShapes[V][1]>::bytes, SmemSize<2, KT, kBatchShapes[V][2], batch_int2(sizeof(KT), V)>::bytes);
    static constexpr size_t bytes =
        HIGH ? zmax(low, zmax(SmemSize<3, KT, kBatchShapes[V][3]>::bytes, SmemSize<4, KT, kBatchShapes[V][4]>::bytes)) : low;
};
static_assert(Deg<1>::ND * kBatchShapes[2][1] <= BATCH_THREADS && Deg<2>::ND * kBatchShapes[1][2] <= BATCH_THREADS &&
                  Deg<3>::ND * kBatchShapes[1][3] <= BATCH_THREADS && Deg<4>::ND * kBatchShapes[0][4] <= BATCH_THREADS,
              "every tile shape fits the CTA");

// MINB: CTAs per SM that the registers are bounded for.  HIGH: with the code of p = 3 and
// 4.  ABS: with the code of absorbing faces.  48 registers (MINB = 4) hold the loads of an
// FP32 row in flight only if the item's arguments stay out of them, in shared memory, and
// so does the damping's code: with both in them 48 steps of 64 problems of 3^3..8^3 x 6 took
// 14.95 ms instead of 13.6, of 5 of 20^3..26^3 at p = 3 60.4 instead of 50.2.  The FP64
// kernels are faster with the arguments in registers (64 registers: 19.3 against 20.3 ms).
// FP64 with a grid of at most three CTAs per SM, which the tuner takes where the items are
// few, has 64 registers (24 problems of 2^3..4^3 x 6: 2.81 -> 2.33 ms), and in the shapes
// without integer columns at p = 2 a kernel of p = 1 and 2 alone (5 problems of 20^3..26^3
// at p = 1, tuned: 18.7 -> 18.0 ms, at p = 2 42.9 -> 40.0).  In those shapes the FP64 kernel
// of all degrees keeps the damping's code: what it spills lies in that code, and without it
// the compiler has fewer loads in flight (8 problems of 20^3..26^3, tuned: 124.9 against
// 122.5 ms, 64 of 3^3..8^3 27.3 against 27.0; in shape 0 46.0 without, 46.3 with at p = 2).
template <typename KT, int V, int MINB, bool HIGH, bool ABS>
__global__ void __launch_bounds__(BATCH_THREADS, MINB)
k_step_batch(const BatchProblem* __restrict__ probs, const int2* __restrict__ items, int n_items, int* queue,
             const int64_t* step_idx, int off, const double* gvals, int64_t g_stride) {
    constexpr bool SHARED = sizeof(KT) == 4;
    constexpr int CHAIN = SHARED || V == 0 ? 4 : 16;
    __shared__ __align__(16) char smem[BatchSmem<KT, V, HIGH>::bytes];
    __shared__ int s_item;
    __shared__ __align__(8) char s_args[SHARED ? sizeof(StepArgs) : 8];
    static_assert(sizeof(StepArgs) % 8 == 0, "copied as 8-byte words");
    const int64_t k = *step_idx + off;   // off: the step's place in the graph
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
        __syncthreads();
        const int it = s_item;
        __syncthreads();
        if (it >= n_items) break;
        const int2 w = items[it];
        const BatchProblem& pb = probs[w.x];
        const auto at_step = [&](StepArgs& A) {
            const int cur = pb.cur0 ^ (int)(k & 1);
            A.un = pb.buf[cur];
            A.u0 = pb.buf[cur ^ 1];
            A.out = pb.buf[cur ^ 1];
            A.gvals = gvals + (int64_t)w.x * g_stride;
            A.step_idx = step_idx;
            A.step_off = off;
        };
        const auto go = [&](const StepArgs& A) {
            if constexpr (HIGH) {
                if (pb.p == 3) return step_poly<3, KT, MODE_STEP, kBatchShapes[V][3], int_columns(3, sizeof(KT)), false, ABS, CHAIN>(A, w.y, smem);
                if (pb.p == 4) return step_poly<4, KT, MODE_STEP, kBatchShapes[V][4], int_columns(4, sizeof(KT)), false, ABS, CHAIN>(A, w.y, smem);
            }
            if (pb.p == 1) return step_poly<1, KT, MODE_STEP, kBatchShapes[V][1], false, false, ABS, CHAIN>(A, w.y, smem);
            if constexpr (batch_int2(sizeof(KT), V)) {
                if (A.Kex)   // integer columns, as the problem alone
                    return step_poly<2, KT, MODE_STEP, kBatchShapes[V][2], true, false, ABS, CHAIN>(A, w.y, smem);
            }
            step_poly<2, KT, MODE_STEP, kBatchShapes[V][2], false, false, ABS, CHAIN>(A, w.y, smem);
        };
        if constexpr (SHARED) {
            // the reads of the previous item's are over: a barrier parts them from here
            for (int i = threadIdx.x; i < (int)(sizeof(StepArgs) / 8); i += blockDim.x)
                ((int64_t*)s_args)[i] = ((const int64_t*)&pb.a)[i];
            __syncthreads();
            if (threadIdx.x == 0) at_step(*(StepArgs*)s_args);
            __syncthreads();
            go(*(const StepArgs*)s_args);
        } else {
            StepArgs A = pb.a;
            at_step(A);
            go(A);
        }
    }
}

// Clears the item counters of the next step and moves the step counter on by n
// (0 but at the end of a graph).
__global__ void k_batch_bump(int64_t* idx, int n, int* queue) {
    *idx += n;
    for (int i = 0; i < BATCH_QUEUES; ++i) queue[i] = 0;
}

constexpr int TUNE_VERSION = 3;
std::string tune_cache_path() {
    const char* e = std::getenv("LYMPH_TUNE_CACHE");
    if (e && *e) return e;
    const char* h = std::getenv("HOME");
    return std::string(h ? h : "/tmp") + "/.cache/lymph3d_gb300_tune3.txt";
}

std::mutex g_tune_mu;

bool tune_lookup(const std::string& key, int* grid, int* order, int* shape) {
    std::lock_guard<std::mutex> l(g_tune_mu);
    std::ifstream f(tune_cache_path());
    std::string k;
    int g, o, sh;
    while (f >> k >> g >> o >> sh)
        if (k == key && sh >= 0 && sh < BATCH_SHAPES) { *grid = g; *order = o; *shape = sh; return true; }
    return false;
}

void tune_store(const std::string& key, int grid, int order, int shape) {
    std::lock_guard<std::mutex> l(g_tune_mu);
    std::string path = tune_cache_path();
    size_t slash = path.rfind('/');
    if (slash != std::string::npos && slash > 0) {
        std::error_code ec;  // the cache is optional: a directory that cannot be made skips the store
        std::filesystem::create_directories(path.substr(0, slash), ec);
        if (ec) return;
    }
    std::ofstream f(path, std::ios::app);
    f << key << " " << grid << " " << order << " " << shape << "\n";
}

}  // namespace

struct lymph_batch {
    std::vector<lymph_ctx*> ctx;
    int precision = LYMPH_FP64;
    cudaStream_t stream = nullptr;
    void* d_probs = nullptr;         // BatchProblem[n], or the matrix-free path's records
    int2* d_items = nullptr;
    int n_items = 0;
    std::vector<int2> items_lpt, items_natural;
    int order = 0;       // 0 = largest cost first, 1 = problem-major
    int grid = 0;
    int shape = 0;       // tile shape (kBatchShapes row) of the FP64 / FP32-block kernel
    int* d_queue = nullptr;          // two sets of BATCH_QUEUES item counters (one per degree on the matrix-free
                                     // path), for the steps of even and odd place in a graph
    // the passes of a step that run beside the first (degrees on the
    // matrix-free path, the counters' reset) and what orders them
    cudaStream_t side[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t ev_fork = nullptr, ev_join[4] = {nullptr, nullptr, nullptr, nullptr};
    int mf_off[5] = {0, 0, 0, 0, 0};  // matrix-free path: degree p's items are [mf_off[p - 1], mf_off[p])
    int mf_occ[4] = {1, 1, 1, 1};     // matrix-free path: CTAs per SM of each degree's kernel
    int64_t* d_step_idx = nullptr;
    double* d_gvals = nullptr;
    int64_t gvals_cap = 0;
    int* d_status = nullptr;
    cudaGraphExec_t graph = nullptr;
    int64_t graph_stride = 0;   // of the time-function values it reads
    int graph_steps = 0;
    int64_t launches = 0;
    int step_nl = 2;     // kernels one batched step launches
    int sms = 0;
    bool high = false;        // a problem of p = 3 or 4
    bool absorbing = false;   // a problem with absorbing faces
    std::string key;
};

namespace {

int upload_items(lymph_batch* b) {
    const std::vector<int2>& v0 = b->order == 0 ? b->items_lpt : b->items_natural;
    std::vector<int2> grouped;
    const std::vector<int2>* v = &v0;
    if (b->precision == LYMPH_MIXED_MF) {
        // one group per degree, each in the chosen order
        for (int p = 1; p <= 4; ++p) {
            b->mf_off[p - 1] = (int)grouped.size();
            for (const int2& w : v0)
                if (b->ctx[w.x]->p == p) grouped.push_back(w);
        }
        b->mf_off[4] = (int)grouped.size();
        v = &grouped;
    }
    LYMPH_CUDA_TRY(cudaMemcpyAsync(b->d_items, v->data(), v->size() * sizeof(int2), cudaMemcpyHostToDevice, b->stream));
    LYMPH_CUDA_TRY(cudaStreamSynchronize(b->stream));  // the host vector goes out of scope
    if (b->graph) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }
    return LYMPH_OK;
}

int refresh_problems(lymph_batch* b) {
    if (b->precision == LYMPH_MIXED_MF) {
        const size_t rb = lymph_mf_batch_problem_bytes();
        std::vector<char> h(rb * b->ctx.size());
        for (size_t i = 0; i < b->ctx.size(); ++i) lymph_mf_batch_problem(b->ctx[i], b->d_status, h.data() + rb * i);
        LYMPH_CUDA_TRY(cudaMemcpyAsync(b->d_probs, h.data(), h.size(), cudaMemcpyHostToDevice, b->stream));
        return LYMPH_OK;
    }
    int64_t bytes = 0;   // of the blocks a step reads
    for (const lymph_ctx* c : b->ctx) bytes += c->n_blocks * c->nd * c->nd * (b->precision == LYMPH_FP64 ? 8 : 4);
    std::vector<BatchProblem> h(b->ctx.size());
    for (size_t i = 0; i < b->ctx.size(); ++i) {
        lymph_ctx* c = b->ctx[i];
        BatchProblem& P = h[i];
        P = BatchProblem();
        P.a.row_ptr = c->d_row_ptr;
        P.a.col = c->d_col;
        P.a.K = c->d_K;
        P.a.Kex = c->d_Kex;
        P.a.Minv = c->d_Minv;
        P.a.rhs_stat = c->d_rhs_stat;
        P.a.rhs_dyn = c->d_rhs_dyn;
        P.a.partial = nullptr;
        P.a.abs_idx = c->n_abs > 0 ? c->d_abs_idx : nullptr;
        P.a.Dabs = c->d_Dabs;
        P.a.Winv = c->d_Winv;
        P.a.dt = c->dt;
        P.a.dt2 = c->dt * c->dt;
        P.a.status = b->d_status;
        P.a.n_poly = c->n_poly;
        P.a.early = 0;
        P.a.prefetch = !b->high || (bytes >= BATCH_PREFETCH_MIN && (b->precision == LYMPH_FP64 || c->p <= 3));
        P.buf[0] = c->d_buf[0];
        P.buf[1] = c->d_buf[1];
        P.cur0 = c->cur;
        P.p = c->p;
    }
    LYMPH_CUDA_TRY(cudaMemcpyAsync(b->d_probs, h.data(), h.size() * sizeof(BatchProblem), cudaMemcpyHostToDevice, b->stream));
    return LYMPH_OK;
}

template <typename KT>
void launch_shape(lymph_batch* b, const BatchProblem* probs, int off, int* queue, int64_t g_stride) {
    auto go = [&](auto kernel) {
        kernel<<<b->grid, BATCH_THREADS, 0, b->stream>>>(probs, b->d_items, b->n_items, queue, b->d_step_idx, off,
                                                         b->d_gvals, g_stride);
    };
    auto shape = [&](auto v) {
        constexpr int V = decltype(v)::value;
        if constexpr (sizeof(KT) == 8) {
            if (!b->absorbing) {
                if (b->grid <= 3 * b->sms) return go(k_step_batch<KT, V, 3, true, false>);
                if constexpr (V == 0) {
                    return go(k_step_batch<KT, V, BATCH_MINB, true, false>);
                } else {
                    if (!b->high) return go(k_step_batch<KT, V, BATCH_MINB, false, false>);
                }
            }
            go(k_step_batch<KT, V, BATCH_MINB, true, true>);
        } else {
            if (b->absorbing) go(k_step_batch<KT, V, BATCH_MINB, true, true>);
            else go(k_step_batch<KT, V, BATCH_MINB, true, false>);
        }
    };
    switch (b->shape) {
        case 1: shape(std::integral_constant<int, 1>()); break;
        case 2: shape(std::integral_constant<int, 2>()); break;
        default: shape(std::integral_constant<int, 0>()); break;
    }
}

// The step at place `off` of a graph (or of the steps launched one by one after
// the last graph); bump: what the step counter moves on by after it.  The
// passes of the degrees present run side by side, each on a stream of its own
// (one after another, each left most SMs idle on small problems: 79 us a step
// of 32 problems of 3^3..8^3 x 6 tetrahedra), and the item counters of the next
// step are cleared beside them.
int launch_step(lymph_batch* b, int64_t g_stride, int off, int bump) {
    const BatchProblem* probs = (const BatchProblem*)b->d_probs;
    int* queue = b->d_queue + BATCH_QUEUES * (off & 1);
    int* next = b->d_queue + BATCH_QUEUES * ((off + 1) & 1);
    int nl = 1;
    const bool mf = b->precision == LYMPH_MIXED_MF;
    if (mf) LYMPH_TRY(lymph_mf_batch_u32(b->stream, b->d_probs, b->d_items, b->n_items, b->d_step_idx, off));
    LYMPH_CUDA_TRY(cudaEventRecord(b->ev_fork, b->stream));
    bool used[4] = {false, false, false, bump == 0};   // side[3] clears the counters unless the step counter moves
    if (used[3]) {
        LYMPH_CUDA_TRY(cudaStreamWaitEvent(b->side[3], b->ev_fork, 0));
        k_batch_bump<<<1, 1, 0, b->side[3]>>>(b->d_step_idx, 0, next);
    }
    if (mf) {
        // per degree: the tuned grid, at most what the SMs hold of that
        // degree's kernel and at most one CTA per item
        int grid[4], n_side = 0;
        cudaStream_t st[4];
        bool first = true;
        for (int p = 1; p <= 4; ++p) {
            const int n = b->mf_off[p] - b->mf_off[p - 1];
            grid[p - 1] = std::min(std::min(b->grid, b->mf_occ[p - 1] * b->sms), n);
            st[p - 1] = b->stream;
            if (n <= 0) continue;
            if (!first) {
                used[n_side] = true;
                st[p - 1] = b->side[n_side++];
                LYMPH_CUDA_TRY(cudaStreamWaitEvent(st[p - 1], b->ev_fork, 0));
            }
            first = false;
        }
        LYMPH_TRY(lymph_mf_batch_step(st, grid, b->d_probs, b->d_items, b->mf_off, queue, b->d_step_idx, off, b->d_gvals,
                                      g_stride, &nl));
        ++nl;   // the FP32 copies
    } else if (b->precision == LYMPH_MIXED) {
        launch_shape<float>(b, probs, off, queue, g_stride);
    } else {
        launch_shape<double>(b, probs, off, queue, g_stride);
    }
    for (int i = 0; i < 4; ++i)
        if (used[i]) {
            LYMPH_CUDA_TRY(cudaEventRecord(b->ev_join[i], b->side[i]));
            LYMPH_CUDA_TRY(cudaStreamWaitEvent(b->stream, b->ev_join[i], 0));
        }
    if (bump) k_batch_bump<<<1, 1, 0, b->stream>>>(b->d_step_idx, bump, next);
    b->step_nl = nl + 1;
    b->launches += b->step_nl;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

// Runs n steps with the current grid/order, as graphs of R (even) steps and the rest
// launched one by one; the time-function values are already on the device with
// stride g_stride per problem.  e0 (may be null) is recorded before the first step.
int run_loop(lymph_batch* b, int64_t n, int64_t g_stride, int R, cudaEvent_t e0) {
    LYMPH_TRY(refresh_problems(b));
    LYMPH_CUDA_TRY(cudaMemsetAsync(b->d_step_idx, 0, sizeof(int64_t), b->stream));
    LYMPH_CUDA_TRY(cudaMemsetAsync(b->d_queue, 0, 2 * BATCH_QUEUES * sizeof(int), b->stream));
    if (e0) LYMPH_CUDA_TRY(cudaEventRecord(e0, b->stream));
    int64_t i = 0;
    if (n >= R) {
        if (b->graph && (b->graph_stride != g_stride || b->graph_steps != R)) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }
        if (!b->graph) {
            cudaGraph_t g;
            LYMPH_CUDA_TRY(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
            int64_t l0 = b->launches;
            int rc = LYMPH_OK;
            for (int j = 0; j < R && rc == LYMPH_OK; ++j) rc = launch_step(b, g_stride, j, j == R - 1 ? R : 0);
            b->launches = l0;
            cudaError_t e = cudaStreamEndCapture(b->stream, &g);
            if (rc) {   // a graph without one of its launches would leave work out
                if (e == cudaSuccess) cudaGraphDestroy(g);
                return rc;
            }
            if (e != cudaSuccess) { lymph_set_error(std::string("batch graph capture: ") + cudaGetErrorString(e)); return LYMPH_ERR_CUDA; }
            e = cudaGraphInstantiate(&b->graph, g, 0);
            cudaGraphDestroy(g);
            if (e != cudaSuccess) { lymph_set_error(std::string("batch graph instantiate: ") + cudaGetErrorString(e)); return LYMPH_ERR_CUDA; }
            b->graph_stride = g_stride;
            b->graph_steps = R;
        }
        for (; i + R <= n; i += R) {
            LYMPH_CUDA_TRY(cudaGraphLaunch(b->graph, b->stream));
            b->launches += (int64_t)b->step_nl * R;
        }
    }
    for (int off = 0; i < n; ++i, ++off) LYMPH_TRY(launch_step(b, g_stride, off, 0));
    // each problem's buffers flipped n times
    if (n & 1)
        for (lymph_ctx* c : b->ctx) c->cur ^= 1;
    return LYMPH_OK;
}

int upload_g(lymph_batch* b, const double* g, int64_t n_steps) {
    int64_t need = (int64_t)b->ctx.size() * n_steps;
    if (need > b->gvals_cap) {
        if (b->d_gvals) cudaFree(b->d_gvals);
        b->d_gvals = nullptr;
        b->gvals_cap = need;
        if (cudaMalloc(&b->d_gvals, sizeof(double) * (size_t)need) != cudaSuccess) {
            lymph_set_error("lymph_batch: cannot allocate the time-function table");
            return LYMPH_ERR_OOM;
        }
        if (b->graph) { cudaGraphExecDestroy(b->graph); b->graph = nullptr; }
    }
    LYMPH_CUDA_TRY(cudaMemcpyAsync(b->d_gvals, g, sizeof(double) * (size_t)need, cudaMemcpyHostToDevice, b->stream));
    return LYMPH_OK;
}

int batch_status(lymph_batch* b, const char* where) {
    LYMPH_CUDA_TRY(cudaStreamSynchronize(b->stream));
    int st = 0;
    LYMPH_CUDA_TRY(cudaMemcpy(&st, b->d_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st) {
        LYMPH_CUDA_TRY(cudaMemset(b->d_status, 0, sizeof(int)));
        lymph_set_error(std::string(where) + ": non-finite value in a problem's state");
        return LYMPH_EXIT_INSTAB;
    }
    return LYMPH_OK;
}

}  // namespace

extern "C" {

int lymph_batch_create(lymph_ctx* const* ctxs, int32_t n, lymph_batch** out) {
    if (!out || !ctxs || n <= 0) { lymph_set_error("lymph_batch_create: bad argument"); return LYMPH_ERR_INVALID; }
    *out = nullptr;
    for (int i = 0; i < n; ++i) {
        if (!ctxs[i]) { lymph_set_error("lymph_batch_create: null context"); return LYMPH_ERR_INVALID; }
        if (!ctxs[i]->have_matrices) { lymph_set_error("lymph_batch_create: every context needs lymph_make_matrices first"); return LYMPH_ERR_ORDER; }
        if (ctxs[i]->precision != ctxs[0]->precision) { lymph_set_error("lymph_batch_create: mixed precisions in one batch"); return LYMPH_ERR_INVALID; }
    }
    lymph_batch* b = new lymph_batch();
    b->ctx.assign(ctxs, ctxs + n);
    b->precision = ctxs[0]->precision;
    auto fail = [&](int rc) { lymph_batch_destroy(b); return rc; };
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) { delete b; lymph_set_error("lymph_batch_create: stream"); return LYMPH_ERR_CUDA; }
    bool made = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; i < 4; ++i)
        made = made && cudaStreamCreateWithFlags(&b->side[i], cudaStreamNonBlocking) == cudaSuccess &&
               cudaEventCreateWithFlags(&b->ev_join[i], cudaEventDisableTiming) == cudaSuccess;
    if (!made) { lymph_set_error("lymph_batch_create: stream"); return fail(LYMPH_ERR_CUDA); }
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
    // work items and their cost (bytes of blocks streamed)
    std::vector<std::pair<int64_t, int2>> cost;
    std::ostringstream key;
    // TUNE_VERSION names the kernels the choice was measured with: to be raised with any
    // change that moves their costs
    key << "v" << TUNE_VERSION << "_sm" << b->sms << "_prec" << b->precision;
    std::map<int, std::pair<int64_t, int64_t>> per_p;   // blocks, those with integer columns
    for (int i = 0; i < n; ++i) {
        lymph_ctx* c = ctxs[i];
        for (int P = 0; P < c->n_poly; ++P) {
            int64_t nb = c->h_row_ptr[P + 1] - c->h_row_ptr[P];
            cost.push_back({nb * (int64_t)c->nd * c->nd, make_int2(i, P)});
            b->items_natural.push_back(make_int2(i, P));
        }
        per_p[c->p].first += c->n_blocks;
        if (c->d_Kex) per_p[c->p].second += c->n_blocks;
        b->high = b->high || c->p >= 3;
        b->absorbing = b->absorbing || c->n_abs > 0;
    }
    for (auto& kv : per_p) {
        key << "_p" << kv.first << "b" << kv.second.first;
        if (kv.second.second) key << "i" << kv.second.second;
    }
    if (b->absorbing) key << "_abs";
    b->key = key.str();
    std::stable_sort(cost.begin(), cost.end(), [](const std::pair<int64_t, int2>& x, const std::pair<int64_t, int2>& y) { return x.first > y.first; });
    for (auto& c : cost) b->items_lpt.push_back(c.second);
    b->n_items = (int)b->items_natural.size();
    const size_t prob_bytes = b->precision == LYMPH_MIXED_MF ? lymph_mf_batch_problem_bytes() : sizeof(BatchProblem);
    if (cudaMalloc(&b->d_probs, prob_bytes * n) != cudaSuccess ||
        cudaMalloc(&b->d_items, sizeof(int2) * b->n_items) != cudaSuccess ||
        cudaMalloc(&b->d_queue, 2 * BATCH_QUEUES * sizeof(int)) != cudaSuccess || cudaMalloc(&b->d_step_idx, sizeof(int64_t)) != cudaSuccess ||
        cudaMalloc(&b->d_status, sizeof(int)) != cudaSuccess) {
        lymph_set_error("lymph_batch_create: device allocation failed");
        return fail(LYMPH_ERR_OOM);
    }
    cudaMemsetAsync(b->d_status, 0, sizeof(int), b->stream);
    if (b->precision == LYMPH_MIXED_MF)
        for (int p = 1; p <= 4; ++p) b->mf_occ[p - 1] = lymph_mf_batch_ctas_per_sm(p);
    b->grid = 4 * b->sms;
    b->order = 0;
    b->shape = 0;
    int g, o, sh;
    if (tune_lookup(b->key, &g, &o, &sh)) { b->grid = g; b->order = o; b->shape = sh; }
    int rc = upload_items(b);
    if (rc) return fail(rc);
    *out = b;
    return LYMPH_OK;
}

int lymph_batch_destroy(lymph_batch* b) {
    if (!b) return LYMPH_OK;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->graph) cudaGraphExecDestroy(b->graph);
    for (void* p : {(void*)b->d_probs, (void*)b->d_items, (void*)b->d_queue, (void*)b->d_step_idx, (void*)b->d_gvals,
                    (void*)b->d_status})
        if (p) cudaFree(p);
    for (int i = 0; i < 4; ++i) {
        if (b->side[i]) cudaStreamDestroy(b->side[i]);
        if (b->ev_join[i]) cudaEventDestroy(b->ev_join[i]);
    }
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return LYMPH_OK;
}

int lymph_batch_run(lymph_batch* b, int64_t n_steps, const double* gvals, float* ms_total) {
    NvtxRange nvtx_("lymph_batch_run");
    if (!b || n_steps < 0 || (n_steps > 0 && !gvals)) return LYMPH_ERR_INVALID;
    if (ms_total) *ms_total = 0.0f;
    if (n_steps == 0) return LYMPH_OK;
    for (lymph_ctx* c : b->ctx) cudaStreamSynchronize(c->stream);  // contexts' own work first
    LYMPH_TRY(upload_g(b, gvals, n_steps));
    cudaEvent_t e0, e1;
    LYMPH_CUDA_TRY(cudaEventCreate(&e0));
    LYMPH_CUDA_TRY(cudaEventCreate(&e1));
    cudaEventRecord(e0, b->stream);
    int rc = run_loop(b, n_steps, n_steps, 16, nullptr);
    cudaEventRecord(e1, b->stream);
    cudaEventSynchronize(e1);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms_total) *ms_total = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    LYMPH_TRY(rc);
    return batch_status(b, "lymph_batch_run");
}

int lymph_batch_autotune(lymph_batch* b, int32_t trial_steps, int32_t use_cache, int32_t* grid, int32_t* order) {
    if (!b || trial_steps < 1) return LYMPH_ERR_INVALID;
    int g0, o0, s0;
    if (use_cache && tune_lookup(b->key, &g0, &o0, &s0)) {
        b->grid = g0;
        b->order = o0;
        b->shape = s0;
        LYMPH_TRY(upload_items(b));
    } else {
        // candidates: persistent grids of 1..k CTAs per SM (k: what one SM
        // holds of the step kernel), two item orders and, for the block
        // kernel, the tile shapes.  The trial steps advance the real state, so the state
        // is saved and restored around the trials.
        std::vector<std::vector<double>> save(b->ctx.size() * 2);
        for (size_t i = 0; i < b->ctx.size(); ++i) {
            lymph_ctx* c = b->ctx[i];
            size_t nv = (size_t)c->n_poly * c->nd;
            for (int k = 0; k < 2; ++k) {
                save[2 * i + k].resize(nv);
                LYMPH_CUDA_TRY(cudaMemcpy(save[2 * i + k].data(), c->d_buf[k], nv * sizeof(double), cudaMemcpyDeviceToHost));
            }
        }
        std::vector<int> curs;
        for (lymph_ctx* c : b->ctx) curs.push_back(c->cur);
        // a trial runs as the loop does, in a graph: launched one by one, the matrix-free
        // passes of small problems would be timed by the host's calls
        const int64_t T = (int64_t)trial_steps + (trial_steps & 1);
        const int R = (int)std::min<int64_t>(T, 16);
        std::vector<double> g(b->ctx.size() * (size_t)T, 0.0);
        LYMPH_TRY(upload_g(b, g.data(), T));
        float best = 1e30f;
        int bg = b->grid, bo = b->order, bs = b->shape;
        const int n_shapes = b->precision == LYMPH_MIXED_MF ? 1 : BATCH_SHAPES;
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        const int max_mult =
            b->precision == LYMPH_MIXED_MF ? *std::max_element(b->mf_occ, b->mf_occ + 4) : BATCH_MINB;
        for (int shp = 0; shp < n_shapes; ++shp)
        for (int ord = 0; ord < 2; ++ord)
            for (int mult = 1; mult <= max_mult; ++mult) {
                b->shape = shp;
                b->order = ord;
                b->grid = mult * b->sms;
                LYMPH_TRY(upload_items(b));
                LYMPH_TRY(run_loop(b, T, T, R, nullptr));  // makes the graph and warms up
                LYMPH_TRY(run_loop(b, T, T, R, e0));
                cudaEventRecord(e1, b->stream);
                cudaEventSynchronize(e1);
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, e0, e1);
                if (ms < best) { best = ms; bg = b->grid; bo = ord; bs = shp; }
            }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        for (size_t i = 0; i < b->ctx.size(); ++i) {
            lymph_ctx* c = b->ctx[i];
            size_t nv = (size_t)c->n_poly * c->nd;
            for (int k = 0; k < 2; ++k)
                LYMPH_CUDA_TRY(cudaMemcpy(c->d_buf[k], save[2 * i + k].data(), nv * sizeof(double), cudaMemcpyHostToDevice));
            c->cur = curs[i];
        }
        LYMPH_CUDA_TRY(cudaMemset(b->d_status, 0, sizeof(int)));
        b->grid = bg;
        b->order = bo;
        b->shape = bs;
        LYMPH_TRY(upload_items(b));
        tune_store(b->key, bg, bo, bs);
    }
    if (grid) *grid = b->grid;
    if (order) *order = b->order;
    LYMPH_CUDA_TRY(cudaStreamSynchronize(b->stream));
    return LYMPH_OK;
}

int lymph_batch_schedule(const lymph_batch* b, int32_t* grid, int32_t* order, int32_t* shape) {
    if (!b) return LYMPH_ERR_INVALID;
    if (grid) *grid = b->grid;
    if (order) *order = b->order;
    if (shape) *shape = b->shape;
    return LYMPH_OK;
}

int lymph_batch_launch_count(const lymph_batch* b, int64_t* count) {
    if (!b || !count) return LYMPH_ERR_INVALID;
    *count = b->launches;
    return LYMPH_OK;
}

}  // extern "C"
