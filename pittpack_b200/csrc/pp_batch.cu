// Batched solves: many independent grids of uneven sizes and boundary
// conditions, replayed as one CUDA graph.
//
// The reference solves one grid per PencilDcmp object and launches every
// step separately (src/pencilDcmp.cpp:5801-6430).  Here each grid keeps a
// handle (plans and twiddles resident on the device, zero-copy bound to the
// caller's RHS and solution buffers, the workspaces shared by the grids of a
// branch), the launch shape of each
// size class is chosen once by the autotuner, and the solves of all grids are
// captured into one graph whose branches run concurrently, so that small grids
// fill the GPU together and the whole batch costs one graph launch.
#include <map>
#include <new>
#include <string>
#include <tuple>
#include <vector>

#include <algorithm>

#include "../../include/pittpack_b200.h"
#include "pp_kernels.h"

struct pp_batch_s {
    int device = 0;
    std::vector<pp_handle> handles;
    // per branch, one workspace that its grids take in turn (two spectra, and
    // the FP32 residual of the refined solve): what a grid leaves in L2 is
    // overwritten there by the next one instead of going to memory
    struct Workspace {
        void* p[3] = {nullptr, nullptr, nullptr};
    };
    std::vector<Workspace> work;
    std::vector<cudaStream_t> branches;
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int nodes = 0;  // graph nodes (kernels and memsets) per replay
};

namespace {

void batch_free(pp_batch_s* b)
{
    if (!b) return;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    // the handles name the branch streams: release them first
    for (auto h : b->handles) pp_destroy(h);
    for (auto& w : b->work)
        for (void* q : w.p)
            if (q) cudaFree(q);
    for (auto s : b->branches) cudaStreamDestroy(s);
    if (b->cap) cudaStreamDestroy(b->cap);
    delete b;
}

// How many grids run at once, at most 'branches': of plain solves as many as keep their spectra
// in three quarters of L2 together (right-hand sides and solutions pass through
// the rest).  A grid's passes hand the two spectra from one to the next through
// L2; past its capacity every pass goes to memory and back (48 grids of 32 ..
// 192 points an edge, 126 MB of L2: 1.95 ms at 3 and 4 branches, 2.1 at 5, 2.40
// at 8, 2.44 at 16, 2.07 at 2, 2.53 at 1).  Larger grids still run two at a time,
// so that one fills the other's tails (two branches and one, ms: 12 of 192^3 1.57
// and 1.93, 8 of 256^3 2.20 and 2.49, 6 of 256 x 256 x 320 2.07 and 2.21, 16 mixed
// of 128 .. 320 3.42 and 3.72; with workspaces of their own 2, 3, 4 and 8 branches
// of these were within 6 %).
// Refined solves run as many as asked for: a sweep's residual, sums and zero-mode
// column are small launches that wait for one another, and more grids fill them
// (ms at 3, 6, 8 and 16 branches: 48 uneven grids 4.09, 3.19, 3.19 and 3.56, 96 of
// them 9.15, 7.48, 7.59 and 8.84, 24 of 128^3 2.25, 1.84, 1.84 and 1.84, 64 of 64^3
// 3.20, 1.83, 1.46 and 0.95, 8 of 256^3 4.64, 4.62, 4.59 and 4.59).
int branches_in_l2(const pp_batch_item* items, int n, bool refined, int branches)
{
    if (refined) return branches;
    int dev = 0, l2 = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess ||
        l2 <= 0)
        return branches;
    double bytes = 0.0;
    for (int i = 0; i < n; ++i) {
        // two real spectra (half spectra of a periodic x as much), the second one
        // complex for a periodic y alone
        if (items[i].nx <= 0 || items[i].ny <= 0 || items[i].nz <= 0) continue;  // rejected later
        const bool wide = items[i].bc[2] == 'P' && items[i].bc[0] != 'P';
        bytes += (wide ? 24.0 : 16.0) * items[i].nx * (double)items[i].ny * items[i].nz;
    }
    const double fit = bytes > 0 ? 0.75 * l2 * n / bytes : branches;
    return fit >= branches ? branches : std::min(branches, std::max(2, (int)fit));
}

// one handle per grid, tuned per size class, solved once outside the capture
int build_handles(pp_batch_s* b, const pp_batch_item* items, int n, const pp_options* opt, int branches, int autotune)
{
    const bool refined = opt && opt->precision == PP_PRECISION_MIXED;
    b->work.resize(branches);
    for (int k = 0; k < branches; ++k) {
        size_t bytes = 0;
        for (int i = k; i < n; i += branches) {
            const pp_batch_item& it = items[i];
            // (grids that pp_create refuses get their own error below)
            if (it.nx >= 2 && it.ny >= 2 && it.nz >= 3 && it.nz <= pp_zsolve_max_nz(false, false))
                bytes = std::max(bytes, pp_spectrum_bytes(it.nx, it.ny, it.nz, it.bc[2] == 'P'));
        }
        const size_t want[3] = {bytes, bytes, refined ? bytes / 4 : 0};
        for (int q = 0; q < 3; ++q)
            if (want[q] && cudaMalloc(&b->work[k].p[q], want[q]) != cudaSuccess) {
                cudaGetLastError();
                return PP_ALLOCATION_FAIL;
            }
    }
    // tuned launch shape per size class (nx, ny, nz, boundary letters)
    std::map<std::tuple<int, int, int, std::string>, pp_tuning> tuned;
    int rc = PP_SUCCESS;
    for (int i = 0; i < n && rc == PP_SUCCESS; ++i) {
        const pp_batch_item& it = items[i];
        pp_handle h = nullptr;
        void* const* w = b->work[i % branches].p;
        const size_t bytes = pp_spectrum_bytes(it.nx, it.ny, it.nz, it.bc[2] == 'P');
        if ((rc = pp_create_lent(it.nx, it.ny, it.nz, w[0], w[1], bytes, w[2], &h)) != PP_SUCCESS) break;
        b->handles.push_back(h);
        if ((rc = pp_set_box(h, it.box)) != PP_SUCCESS) break;
        if ((rc = pp_assign_boundary(h, it.bc)) != PP_SUCCESS) break;
        if (opt && (rc = pp_set_options(h, opt)) != PP_SUCCESS) break;
        if (!it.d_rhs || !it.d_P) {
            rc = PP_INPUT_ARGS;
            break;
        }
        if ((rc = pp_bind_device_buffers(h, it.d_rhs, 0, it.d_P)) != PP_SUCCESS) break;
        const auto key = std::make_tuple(it.nx, it.ny, it.nz, std::string(it.bc, 6));
        const auto f = tuned.find(key);
        if (f != tuned.end()) {
            rc = pp_set_tuning(h, &f->second);
        } else if (autotune) {
            pp_tuning t;
            double ms = 0.0;
            if ((rc = pp_autotune(h, 3, &t, &ms)) == PP_SUCCESS) tuned[key] = t;
        }
        // one solve outside the capture: kernel attributes and lazily sized
        // buffers are set up before any launch is recorded
        if (rc == PP_SUCCESS) rc = pp_solve(h);
    }
    if (rc == PP_SUCCESS && cudaDeviceSynchronize() != cudaSuccess) rc = PP_CUDA_ERROR;
    return rc;
}

}  // namespace

extern "C" int pp_batch_create(const pp_batch_item* items, int n, const pp_options* opt, int branches, int autotune,
                               pp_batch* out)
{
    if (!items || n < 1 || !out || branches < 1 || branches > 64) return PP_INPUT_ARGS;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return PP_GPU_INIT_FAILURE;
    pp_batch_s* b = new (std::nothrow) pp_batch_s;
    if (!b) return PP_ALLOCATION_FAIL;
    cudaGetDevice(&b->device);
    branches = branches_in_l2(items, n, opt && opt->precision == PP_PRECISION_MIXED, branches);
    int rc = build_handles(b, items, n, opt, branches, autotune);
    if (rc != PP_SUCCESS) {
        batch_free(b);
        return rc;
    }
    // capture: fork the grids over 'branches' streams, join, one graph
    cudaError_t e = cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking);
    std::vector<cudaEvent_t> ev(branches + 1, nullptr);
    for (auto& x : ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
    b->branches.assign(branches, nullptr);
    for (auto& s : b->branches)
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        cudaEventRecord(ev[0], b->cap);
        for (auto s : b->branches) cudaStreamWaitEvent(s, ev[0], 0);
        for (int i = 0; i < n && rc == PP_SUCCESS; ++i) {
            if ((rc = pp_set_stream(b->handles[i], b->branches[i % branches])) == PP_SUCCESS)
                rc = pp_solve(b->handles[i]);
        }
        for (int k = 0; k < branches; ++k) {
            cudaEventRecord(ev[k + 1], b->branches[k]);
            cudaStreamWaitEvent(b->cap, ev[k + 1], 0);
        }
        // the capture is always ended, also after a failed solve
        const cudaError_t e2 = cudaStreamEndCapture(b->cap, &b->graph);
        if (e2 != cudaSuccess && rc == PP_SUCCESS) rc = PP_CUDA_ERROR;
    } else {
        rc = PP_CUDA_ERROR;
    }
    if (rc == PP_SUCCESS && cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess) rc = PP_CUDA_ERROR;
    for (auto& x : ev)
        if (x) cudaEventDestroy(x);
    if (rc != PP_SUCCESS) {
        batch_free(b);
        return rc;
    }
    size_t nodes = 0;
    cudaGraphGetNodes(b->graph, nullptr, &nodes);
    b->nodes = (int)nodes;
    *out = b;
    return PP_SUCCESS;
}

extern "C" int pp_batch_run(pp_batch b, void* stream)
{
    if (!b) return PP_INVALID_HANDLE;
    cudaSetDevice(b->device);
    return cudaGraphLaunch(b->exec, (cudaStream_t)stream) == cudaSuccess ? PP_SUCCESS : PP_CUDA_ERROR;
}

extern "C" int pp_batch_info(pp_batch b, int* grids, int* graph_nodes)
{
    if (!b) return PP_INVALID_HANDLE;
    if (grids) *grids = (int)b->handles.size();
    if (graph_nodes) *graph_nodes = b->nodes;
    return PP_SUCCESS;
}

extern "C" int pp_batch_destroy(pp_batch b)
{
    if (!b) return PP_INVALID_HANDLE;
    cudaSetDevice(b->device);
    cudaDeviceSynchronize();
    batch_free(b);
    return PP_SUCCESS;
}
