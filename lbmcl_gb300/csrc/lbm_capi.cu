// lbm_capi.cu -- the extern "C" boundary (include/lbm.h): handle life cycle,
// device memory, the iteration loop, dumps, timing and reductions.
//
// Replaces the reference's OpenCL host plumbing of this path:
// buffer creation (lbmcl.hpp:403-417), the per-iteration kernel objects and
// the ping-pong argument swap (lbmcl.hpp:435-467), the enqueue loop
// (lbmcl.hpp:490-521), the blocking read-backs (lbmcl.hpp:159-277) and the
// event timing (lbmcl.hpp:548-593).  Failures return a status code and leave a
// message in lbm_last_error(); nothing here calls exit().
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "lbm.h"
#include "lbm_device.cuh"
#include "lbm_handle.h"
#include "lbm_launch.h"

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define LBM_CUDA(call)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess) {                                                                \
            cudaGetLastError();                                                                 \
            return fail(e_ == cudaErrorMemoryAllocation ? LBM_ENOMEM : LBM_ECUDA, "%s: %s", #call, \
                        cudaGetErrorString(e_));                                                \
        }                                                                                       \
    } while (0)

using lbm::macro_bytes;
using lbm::storage_bytes;
int vec_len(int prec) { return (int)(16 / storage_bytes(prec)); }
int dim_multiple(int prec) { return (prec == LBM_FP16 || prec == LBM_BF16) ? 8 : 4; }

constexpr size_t kStageElems = (size_t)1 << 25;  // dump / load staging, elements
constexpr size_t kPieceElems = (size_t)1 << 22;  // of it, per overlapped copy

__global__ void sum_partials_kernel(const double *__restrict__ partials, int nblocks, double *__restrict__ out)
{
    // one block of 256 threads, fixed summation order: deterministic
    double m = 0.0, e = 0.0;
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
        m += partials[2 * i];
        e += partials[2 * i + 1];
    }
    __shared__ double sm[2][256];
    sm[0][threadIdx.x] = m;
    sm[1][threadIdx.x] = e;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sm[0][threadIdx.x] += sm[0][threadIdx.x + w];
            sm[1][threadIdx.x] += sm[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = sm[0][0];
        out[1] = sm[1][0];
    }
}

}  // namespace

namespace lbm {
cudaError_t launch_sum_partials(const double *partials, int nblocks, double *out, cudaStream_t s)
{
    sum_partials_kernel<<<1, 256, 0, s>>>(partials, nblocks, out);
    return cudaGetLastError();
}

void set_last_error(const char *msg) { g_err = msg; }
}  // namespace lbm


namespace {

cudaError_t get_event(lbm_t *h, cudaEvent_t *ev)
{
    if (!h->spare.empty()) {
        *ev = h->spare.back();
        h->spare.pop_back();
        return cudaSuccess;
    }
    return cudaEventCreate(ev);
}

// Add the durations of finished event pairs to kernels_ms (in stream order).
int fold_events(lbm_t *h, bool wait)
{
    size_t k = 0;
    for (; k < h->pending.size(); ++k) {
        auto &p = h->pending[k];
        if (wait) {
            LBM_CUDA(cudaEventSynchronize(p.second));
        } else {
            cudaError_t q = cudaEventQuery(p.second);
            if (q == cudaErrorNotReady) break;
            LBM_CUDA(q);
        }
        float ms = 0;
        LBM_CUDA(cudaEventElapsedTime(&ms, p.first, p.second));
        h->kernels_ms += ms;
        h->spare.push_back(p.first);
        h->spare.push_back(p.second);
    }
    h->pending.erase(h->pending.begin(), h->pending.begin() + (ptrdiff_t)k);
    return LBM_OK;
}

void release(lbm_t *h)
{
    if (!h) return;
    const lbm::DeviceScope dev(h->cfg.device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    lbm::release_adjoint(h);
    for (void *p : {h->f[0], h->f[1], (void *)h->map, h->rho, h->u, h->lid, h->stage, (void *)h->partials,
                    (void *)h->red_out, (void *)h->status})
        lbm::device_free(h, p);
    for (auto &p : h->pending) {
        cudaEventDestroy(p.first);
        cudaEventDestroy(p.second);
    }
    for (auto e : h->spare) cudaEventDestroy(e);
    for (cudaGraphExec_t &g : h->graph_exec)
        if (g) cudaGraphExecDestroy(g), g = nullptr;
    // what the pool does not keep goes back now, not in some later call
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->ev_first) cudaEventDestroy(h->ev_first);
    if (h->ev_last) cudaEventDestroy(h->ev_last);
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
    if (h->ev_join) cudaEventDestroy(h->ev_join);
    if (h->side) cudaStreamDestroy(h->side);
    for (auto e : h->copy_events) cudaEventDestroy(e);
    if (h->copy) cudaStreamDestroy(h->copy);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

// Name and SM count of a device, asked for once per process (0.2 ms a query).
cudaError_t device_facts(int device, std::string &name, int &sms)
{
    static std::mutex mu;
    static std::map<int, std::pair<std::string, int>> known;
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(device);
    if (it == known.end()) {
        cudaDeviceProp prop;
        const cudaError_t e = cudaGetDeviceProperties(&prop, device);
        if (e != cudaSuccess) return e;
        it = known.emplace(device, std::make_pair(std::string(prop.name), prop.multiProcessorCount)).first;
    }
    name = it->second.first;
    sms = it->second.second;
    return cudaSuccess;
}

bool is_aa(const lbm_t *h) { return h->kernel == LBM_KERNEL_AA; }

// Iteration arguments from buffer `from` (two-lattice kernels) or of AA
// phase `phase` (the one lattice f[0]).
lbm::StepArgs step_args(const lbm_t *h, int from, int phase)
{
    lbm::StepArgs a;
    a.fin = is_aa(h) ? h->f[0] : h->f[from];
    a.fout = is_aa(h) ? h->f[0] : h->f[from ^ 1];
    a.aa_phase = phase;
    a.map = h->map;
    a.lid = h->lid;
    a.rho = h->rho;
    a.u = h->u;
    a.status = h->status;
    a.partials = h->partials;
    a.dim = h->dim;
    a.nvx = h->dim / h->V;
    a.n = h->n;
    a.inv_tau = h->inv_tau;
    a.omega_f = h->omega_f;
    a.rows = h->rows;
    a.gpp = h->gpp;
    a.ngroups = h->ngroups;
    a.stages = h->stages;
    a.sailfish = h->cfg.order == LBM_ORDER_SAILFISH ? 1 : 0;
    return a;
}
lbm::StepArgs step_args(const lbm_t *h, int from) { return step_args(h, from, h->aa_phase); }

// the buffer parity (two lattices) or phase (AA) of the current state, and
// its flip after one iteration
int parity(const lbm_t *h) { return is_aa(h) ? h->aa_phase : h->cur; }
void flip(lbm_t *h)
{
    if (is_aa(h)) h->aa_phase ^= 1;
    else h->cur ^= 1;
}
// layout of the current state for the dump / load kernels
int state_layout(const lbm_t *h)
{
    return is_aa(h) ? (h->aa_phase ? lbm::LAYOUT_AA_B : lbm::LAYOUT_AA_A) : lbm::LAYOUT_PULL;
}

const void *staged_ptr(int prec, int mode)
{
    switch (prec) {
    case LBM_FP32: return lbm::staged_kernel_ptr_f32(mode);
    case LBM_FP64: return lbm::staged_kernel_ptr_f64(mode);
    case LBM_FP16: return lbm::staged_kernel_ptr_f16(mode);
    default: return lbm::staged_kernel_ptr_bf16(mode);
    }
}

// Shape the staged variant: rows per group, ring depth, threads, persistent
// grid.  Returns false when the ring does not fit (the direct variant is used).
int setup_staged(lbm_t *h, int want_stages)
{
    const int dim = h->dim;
    const size_t sb = storage_bytes(h->prec);
    const int V = 4;
    const int nvx = dim / V;
    int rows = std::max(1, 512 / dim);
    rows = std::min(rows, dim - 2);
    const size_t stage_bytes = (size_t)lbm::Q * rows * dim * sb;
    int dev = 0, smem_optin = 0, nsm = 0;
    LBM_CUDA(cudaGetDevice(&dev));
    LBM_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    LBM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t cap = (size_t)smem_optin - 128;
    int stages = want_stages > 0 ? want_stages : (int)std::min<size_t>(8, std::max<size_t>(2, (110u << 10) / stage_bytes));
    while (stages > 2 && 128 + stages * stage_bytes > cap) --stages;
    if (stages < 2 || 128 + stages * stage_bytes > cap) return fail(LBM_EINVAL, "staged kernel: ring does not fit");
    const size_t smem = 128 + stages * stage_bytes;
    unsigned threads = (unsigned)std::min(256, ((rows * nvx + 31) / 32) * 32);
    int per_sm = 0;
    for (int mode : {lbm::MODE_STEP, lbm::MODE_STEP_MACRO}) {
        const void *k = staged_ptr(h->prec, mode);
        LBM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    LBM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, staged_ptr(h->prec, lbm::MODE_STEP),
                                                           (int)threads, smem));
    if (per_sm < 1) return fail(LBM_EINVAL, "staged kernel: no resident block");
    h->rows = rows;
    h->gpp = (dim - 2 + rows - 1) / rows;
    h->ngroups = (unsigned)h->gpp * (unsigned)(dim - 2);
    h->stages = stages;
    h->sblock = threads;
    h->ssmem = smem;
    h->sgrid = (unsigned)std::min<size_t>(h->ngroups, (size_t)per_sm * nsm);
    return LBM_OK;
}

// Vector width and launch count of an iteration of the direct and narrow
// variants: h->step_vb > 0, step_kernel with vectors of so many bytes, one
// launch; 0, pull_kernel's two launches with 16-byte vectors (large 16-bit
// lattices; FP32 DIRECT).
//
// Wide vectors cost registers and give few threads: a small lattice wants
// one or two sites per thread (its time is the latency of one thread's work
// after a launch), a large one the fewest instructions.  us per iteration in
// replayed graphs, 4- / 8- / 16-byte vectors, one launch; two launches:
//   FP16  32^3  2.4 / 2.4 / 4.1; 4.9   64^3 5.6 / 5.0 / 6.7; 6.0
//         96^3 14.0 / 10.9 / 11.8; 12.4   112^3 - / 19.6 / 18.8
//         128^3 34 / 29.4 / 29.3; 30.0   160^3 - / 55.0 / 55.5; 56.3
//         200^3 - / 105.0 / 104.7; 103.7   256^3 - / 200 / 208; 205
//         288^3 - / 299 / -; 292   320^3 - / 398 / -; 390   512^3 - / 1594 / 1610; 1527
//   BF16  32^3  2.4 / 2.4 / 3.6; 6.0   64^3 5.6 / 5.0 / 6.5; 7.0
//         96^3 13 / 11.4 / 11.6; 13.8   112^3 - / 19.8 / 18.5
//         128^3 31.6 / 29.7 / 29.1; 31.4   200^3 - / 106.1 / 105.5; 106.5
//         256^3 - / 202 / 208; 208   288^3 - / 302 / -; 297   320^3 - / 402 / -; 394
//         512^3 - / 1608 / 1597; 1558
//   FP32  32^3  2.9 / 3.2 / 4.9; 3.8   64^3 8.1 / 7.5 / 9.0; 7.9
//         128^3 57 / 48.0 / 55; 50.7   256^3 400 / 360 / 415; 375
//         512^3 3157 / 2910 / 3217; 2950
//   FP64 (8- / 16-byte) 16^3 10.8 / 21.1   32^3 12.0 / 24.1   64^3 63 / 134
//         128^3 467 / 1049   256^3 3480 / 8539
// The 16-bit line at 192^3: two launches are 2 to 4% ahead from 288^3 up; between
// it and 256^3 neither side is by more than 1.3%, but at 256^3 itself 8-byte
// vectors in one launch are by 2.3% (FP16) and 2.8% (BF16): a line for that one size
// would lose as much at 288^3.  FP32 DIRECT, the 16-byte vectors asked for: two
// launches 56^3 7.6, 256^3 380 against 8.4 and 397 in one.
int step_shape(int kernel, int prec, int dim)
{
    const bool s16 = prec == LBM_FP16 || prec == LBM_BF16;
    if (kernel == LBM_KERNEL_NARROW) return 8;
    if (prec == LBM_FP64) return kernel == LBM_KERNEL_DIRECT ? 16 : 8;
    if (kernel == LBM_KERNEL_DIRECT && !s16) return 0;
    if (prec == LBM_FP32) return dim <= 40 ? 4 : 8;
    if (dim > 192) return 0;
    if (kernel == LBM_KERNEL_DIRECT) return 16;
    return dim <= 40 ? 4 : dim <= 104 ? 8 : 16;
}

// The two launches of an iteration with 16-byte vectors, face rows on sf.
cudaError_t launch_rows(const lbm_t *h, int mode, const lbm::StepArgs &a, cudaStream_t sf)
{
    switch (h->prec) {
    case LBM_FP32: return lbm::launch_rows_f32(mode, a, h->step_block, h->stream, sf);
    case LBM_FP16: return lbm::launch_rows_f16(mode, a, h->step_block, h->stream, sf);
    default: return lbm::launch_rows_bf16(mode, a, h->step_block, h->stream, sf);
    }
}

cudaError_t launch_pull(const lbm_t *h, int mode, const lbm::StepArgs &a, unsigned *nparts = nullptr)
{
    if (h->kernel == LBM_KERNEL_AA) {
        switch (h->prec) {
        case LBM_FP32: return lbm::launch_aa_f32(mode, a, h->block, h->stream, nparts);
        case LBM_FP64: return lbm::launch_aa_f64(mode, a, h->block, h->stream, nparts);
        case LBM_FP16: return lbm::launch_aa_f16(mode, a, h->block, h->stream, nparts);
        default: return lbm::launch_aa_bf16(mode, a, h->block, h->stream, nparts);
        }
    }
    if (mode == lbm::MODE_REDUCE) {
        switch (h->prec) {
        case LBM_FP32: return lbm::launch_reduce_f32(a, h->block, h->stream, nparts);
        case LBM_FP64: return lbm::launch_reduce_f64(a, h->block, h->stream, nparts);
        case LBM_FP16: return lbm::launch_reduce_f16(a, h->block, h->stream, nparts);
        default: return lbm::launch_reduce_bf16(a, h->block, h->stream, nparts);
        }
    }
    if (h->kernel == LBM_KERNEL_STAGED && (mode == lbm::MODE_STEP || mode == lbm::MODE_STEP_MACRO)) {
        switch (h->prec) {
        case LBM_FP32: return lbm::launch_staged_f32(mode, a, h->sgrid, h->sblock, h->ssmem, h->stream);
        case LBM_FP64: return lbm::launch_staged_f64(mode, a, h->sgrid, h->sblock, h->ssmem, h->stream);
        case LBM_FP16: return lbm::launch_staged_f16(mode, a, h->sgrid, h->sblock, h->ssmem, h->stream);
        default: return lbm::launch_staged_bf16(mode, a, h->sgrid, h->sblock, h->ssmem, h->stream);
        }
    }
    // Iterations that also store the linearisation points: 8-byte vectors at
    // every 16-bit size beyond 40^3 (us per iteration of the adjoint forward,
    // 16-byte vectors -> 8: FP16 96^3 15.1 -> 14.5, 256^3 262 -> 250; BF16 128^3 38.6
    // -> 36.5, 256^3 278 -> 253).  Not for spills: the FP16 kernel had none with
    // 16-byte vectors and has 56 bytes at 128 registers with 8-byte ones, but
    // 16 warps per SM instead of 12.
    const int vb = mode == lbm::MODE_STEP_ADJ && h->prec != LBM_FP64 && h->step_vb != 4 ? 8 : h->step_vb;
    if (!vb) return launch_rows(h, mode, a, h->stream);
    switch (h->prec) {
    case LBM_FP32: return lbm::launch_step_f32(vb, mode, a, h->step_block, h->stream);
    case LBM_FP64: return lbm::launch_step_f64(vb, mode, a, h->step_block, h->stream);
    case LBM_FP16: return lbm::launch_step_f16(vb, mode, a, h->step_block, h->stream);
    default: return lbm::launch_step_bf16(vb, mode, a, h->step_block, h->stream);
    }
}

size_t dump_elem(int prec) { return prec == LBM_FP64 ? 8 : 4; }

// true when one of the iterations it0 + 1 .. it0 + G stores the moments
bool macro_within(int64_t it0, int G, int macro_every)
{
    if (macro_every == 0) return false;
    const int64_t next = (it0 / macro_every + 1) * macro_every;  // first macro iteration after it0
    return next <= it0 + G;
}

// the two-launch iterations
bool splits(const lbm_t *h) { return h->kernel != LBM_KERNEL_AA && h->kernel != LBM_KERNEL_STAGED && !h->step_vb; }

// One two-launch iteration with its face-row launch on the side stream, forked from and joined back into the handle's
// stream, so that (in a captured graph: as a second branch) it runs beside the
// interior-row launch; the two write disjoint rows of the output and read the
// same input.
cudaError_t split_iteration(const lbm_t *h, const lbm::StepArgs &a)
{
    cudaError_t e = cudaEventRecord(h->ev_fork, h->stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(h->side, h->ev_fork, 0);
    if (e != cudaSuccess) return e;
    e = launch_rows(h, lbm::MODE_STEP, a, h->side);
    // join even after a failed launch, so the capture can end
    const cudaError_t ej = cudaEventRecord(h->ev_join, h->side);
    const cudaError_t ew = ej == cudaSuccess ? cudaStreamWaitEvent(h->stream, h->ev_join, 0) : ej;
    return e != cudaSuccess ? e : ew;
}

// Replay (capturing on first use) the graph of h->graph_iters plain
// iterations that starts from buffer h->cur.  The kernels' arguments are
// fixed per parity (the two buffers ping-pong), so two graphs cover every
// call.  In two-launch iterations the face-row launch is a branch beside the
// interior-row launch.
cudaError_t replay_graph(lbm_t *h)
{
    cudaGraphExec_t &exec = h->graph_exec[parity(h)];
    if (!exec) {
        const bool split = splits(h);
        cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return e;
        int cur = h->cur, ph = h->aa_phase;
        for (int k = 0; k < h->graph_iters && e == cudaSuccess; ++k) {
            e = split ? split_iteration(h, step_args(h, cur, ph))
                      : launch_pull(h, lbm::MODE_STEP, step_args(h, cur, ph));
            if (is_aa(h)) ph ^= 1;
            else cur ^= 1;
        }
        cudaGraph_t g = nullptr;
        const cudaError_t ec = cudaStreamEndCapture(h->stream, &g);
        if (e == cudaSuccess) e = ec;
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            exec = nullptr;
            return e;
        }
    }
    return cudaGraphLaunch(exec, h->stream);
}

// One piece of the F dump (out) or load through slot `buf` of the staging buffer.
cudaError_t launch_piece(lbm_t *h, bool out, void *buf, size_t o0, size_t count)
{
    lbm::DumpArgs a;
    a.f = h->f[h->cur];
    a.map = h->map;
    a.lid = h->lid;
    a.buf = buf;
    a.o0 = o0;
    a.count = count;
    a.dim = h->dim;
    a.sd = h->sd;
    a.n = h->n;
    a.layout = state_layout(h);
    a.four = (h->sd < 0 || h->sd >= 2) && h->dim > 4 && h->n >> 29 == 0;
    a.div_dim = lbm::FastDiv((unsigned)h->dim);
    a.inv_n = ~0ull / h->n + 1;
    switch (h->prec) {
    case LBM_FP32: return out ? lbm::launch_dump_f32(a, h->stream) : lbm::launch_load_f32(a, h->stream);
    case LBM_FP64: return out ? lbm::launch_dump_f64(a, h->stream) : lbm::launch_load_f64(a, h->stream);
    case LBM_FP16: return out ? lbm::launch_dump_f16(a, h->stream) : lbm::launch_load_f16(a, h->stream);
    default: return out ? lbm::launch_dump_bf16(a, h->stream) : lbm::launch_load_bf16(a, h->stream);
    }
}

// F dump (out) or load through the staging buffer.  Page-locked host memory
// beyond two pieces' size: piece by piece with the copies on a stream of their
// own, so that only the first (last) piece's kernel is not behind a copy: 136^3
// FP32 dump 1.32 -> 1.07, load 1.25 -> 0.98 ms, the copy alone 0.99 and 0.91;
// 200^3 BF16 4.25 -> 3.29, 4.21 -> 3.04.  Pieces of 2^20, 2^21, 2^22, 2^23
// elements: 136^3 dump 1.12, 1.08, 1.07, 1.09, 256^3 7.25, 6.96, 6.81, 6.76 ms.
// Pageable memory, whose copies do not run beside kernels: a staging buffer's
// worth at a time.  In pieces a dump into memory not touched before took 49
// instead of 3 ms at 100^3 FP32 and 140 instead of 52 at 136^3, one into touched
// memory 1.41 instead of 1.18, and a load from a mapped file 12.4 instead of 11.3
// at 256^3.
int move_f(lbm_t *h, void *host, bool out)
{
    const size_t te = dump_elem(h->prec), total = (size_t)lbm::Q * h->n;
    if (total <= 2 * kPieceElems || !lbm::page_locked(host, total * te)) {
        for (size_t o0 = 0; o0 < total; o0 += kStageElems) {
            const size_t count = std::min(kStageElems, total - o0);
            char *at = static_cast<char *>(host) + o0 * te;
            if (!out) LBM_CUDA(cudaMemcpyAsync(h->stage, at, count * te, cudaMemcpyHostToDevice, h->stream));
            LBM_CUDA(launch_piece(h, out, h->stage, o0, count));
            if (out && total > kStageElems) lbm::make_pages(at, count * te);
            if (out) LBM_CUDA(cudaMemcpyAsync(at, h->stage, count * te, cudaMemcpyDeviceToHost, h->stream));
        }
        return LBM_OK;
    }
    const size_t slots = std::min(kStageElems, total) / kPieceElems;
    if (!h->copy) LBM_CUDA(cudaStreamCreateWithFlags(&h->copy, cudaStreamNonBlocking));
    while (h->copy_events.size() < 2 * slots) {
        cudaEvent_t e = nullptr;
        LBM_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        h->copy_events.push_back(e);
    }
    // filled[s]: slot s holds a piece; drained[s]: its piece has been taken out
    cudaEvent_t *filled = h->copy_events.data(), *drained = filled + slots;
    cudaStream_t fill = out ? h->stream : h->copy, drain = out ? h->copy : h->stream;
    auto pieces = [&]() -> int {
        if (!out) {  // behind what the handle's stream holds already
            LBM_CUDA(cudaEventRecord(drained[0], h->stream));
            LBM_CUDA(cudaStreamWaitEvent(h->copy, drained[0], 0));
        }
        size_t k = 0;
        for (size_t o0 = 0; o0 < total; o0 += kPieceElems, ++k) {
            const size_t s = k % slots, count = std::min(kPieceElems, total - o0);
            char *buf = static_cast<char *>(h->stage) + s * kPieceElems * te, *at = static_cast<char *>(host) + o0 * te;
            if (k >= slots) LBM_CUDA(cudaStreamWaitEvent(fill, drained[s], 0));
            if (out) LBM_CUDA(launch_piece(h, out, buf, o0, count));
            else LBM_CUDA(cudaMemcpyAsync(buf, at, count * te, cudaMemcpyHostToDevice, fill));
            LBM_CUDA(cudaEventRecord(filled[s], fill));
            LBM_CUDA(cudaStreamWaitEvent(drain, filled[s], 0));
            if (out) LBM_CUDA(cudaMemcpyAsync(at, buf, count * te, cudaMemcpyDeviceToHost, drain));
            else LBM_CUDA(launch_piece(h, out, buf, o0, count));
            LBM_CUDA(cudaEventRecord(drained[s], drain));
        }
        if (out) LBM_CUDA(cudaStreamWaitEvent(h->stream, drained[(k - 1) % slots], 0));
        return LBM_OK;
    };
    const int r = pieces();
    if (r != LBM_OK) cudaStreamSynchronize(h->copy);  // no copy outlives the call
    return r;
}

}  // namespace

namespace lbm {
cudaError_t replay_iterations(lbm_t *h) { return replay_graph(h); }

cudaError_t launch_iteration(const lbm_t *h, const void *fin, void *fout)
{
    StepArgs a = step_args(h, h->cur);
    a.fin = fin;
    a.fout = fout;
    return splits(h) ? split_iteration(h, a) : launch_pull(h, MODE_STEP, a);
}

cudaError_t launch_iteration_adj(const lbm_t *h, const void *fin, void *fout, void *point)
{
    StepArgs a = step_args(h, h->cur);
    a.fin = fin;
    a.fout = fout;
    a.rho = nullptr;
    a.u = point;
    return launch_pull(h, MODE_STEP_ADJ, a);
}
}  // namespace lbm

extern "C" {

void lbm_config_default(lbm_config *c)
{
    if (!c) return;
    memset(c, 0, sizeof *c);
    c->dim = 8;
    c->viscosity = 0.0089;
    c->velocity = 0.05;
    c->precision = LBM_FP32;
    c->stride = 32;
}

const char *lbm_last_error(void) { return g_err.c_str(); }

size_t lbm_size(const lbm_t *h, int what)
{
    if (!h) return 0;
    switch (what) {
    case LBM_DUMP_F: return (size_t)lbm::Q * h->n * dump_elem(h->prec);
    case LBM_DUMP_RHO: return h->n * macro_bytes(h->prec);
    case LBM_DUMP_U: return 3 * h->n * macro_bytes(h->prec);
    case LBM_DUMP_MAP: return h->n * sizeof(int32_t);
    case LBM_DUMP_MAP_U8: return h->n;
    case LBM_DUMP_F_RAW: return (size_t)lbm::Q * h->n * storage_bytes(h->prec);
    default: return 0;
    }
}

int lbm_init(lbm_t **out, const lbm_config *c)
{
    if (!out || !c) return fail(LBM_EINVAL, "lbm_init: NULL argument");
    *out = nullptr;
    if (c->precision < LBM_FP32 || c->precision > LBM_BF16)
        return fail(LBM_EINVAL, "lbm_init: unknown precision %d", c->precision);
    const int prec = c->precision;
    const int dim = c->dim;
    if (dim < 4 || dim % dim_multiple(prec) != 0 || dim > 2048)
        return fail(LBM_EINVAL, "lbm_init: dim %d must be in [4, 2048] and a multiple of %d for this precision", dim,
                    dim_multiple(prec));
    const size_t n = (size_t)dim * dim * dim;
    // CSoA stride of F dumps (kernels.cl:64): a power of two dividing dim^3;
    // 0 selects pure SoA, also for dims whose dim^3 is not a power of two
    // (sd = -1 then).
    const size_t stride = c->stride == 0 ? n : (size_t)c->stride;
    int sd = -1;
    if (c->stride < 0 || (c->stride > 0 && ((stride & (stride - 1)) != 0 || stride > n || n % stride != 0)))
        return fail(LBM_EINVAL, "lbm_init: stride %d must be a power of two dividing dim^3 (or 0 for SoA)",
                    c->stride);
    if ((stride & (stride - 1)) == 0) {
        sd = 0;
        while (((size_t)1 << sd) < stride) ++sd;
    }
    if (!(c->viscosity >= 0.0) && !(c->tau > 0.0))
        return fail(LBM_EINVAL, "lbm_init: viscosity must be >= 0");
    if (!std::isfinite(c->velocity)) return fail(LBM_EINVAL, "lbm_init: velocity must be finite");
    if (c->noise_sigma < 0.0 || !std::isfinite(c->noise_sigma))
        return fail(LBM_EINVAL, "lbm_init: noise_sigma must be finite and >= 0");
    if (c->kernel < LBM_KERNEL_AUTO || c->kernel > LBM_KERNEL_AA)
        return fail(LBM_EINVAL, "lbm_init: unknown kernel variant %d", c->kernel);
    if (c->stages < 0 || c->stages > 16) return fail(LBM_EINVAL, "lbm_init: stages %d out of range", c->stages);
    if (c->adjoint_steps < 0 || c->adjoint_steps > 2)
        return fail(LBM_EINVAL, "lbm_init: adjoint_steps %d out of range (0, 1, 2)", c->adjoint_steps);
    if (c->adjoint_max_states < 0)
        return fail(LBM_EINVAL, "lbm_init: adjoint_max_states %d must be >= 0", c->adjoint_max_states);
    if (c->adjoint_fp64 < 0 || c->adjoint_fp64 > 1)
        return fail(LBM_EINVAL, "lbm_init: adjoint_fp64 %d must be 0 or 1", c->adjoint_fp64);
    if (c->adjoint_full_states < 0 || c->adjoint_full_states > 1)
        return fail(LBM_EINVAL, "lbm_init: adjoint_full_states %d must be 0 or 1", c->adjoint_full_states);
    if (c->adjoint_kernel != LBM_KERNEL_AUTO && c->adjoint_kernel != LBM_KERNEL_DIRECT &&
        c->adjoint_kernel != LBM_KERNEL_STAGED)
        return fail(LBM_EINVAL, "lbm_init: adjoint_kernel %d must be 0, LBM_KERNEL_DIRECT or LBM_KERNEL_STAGED",
                    c->adjoint_kernel);
    if (c->adjoint_tail_segments < -1)
        return fail(LBM_EINVAL, "lbm_init: adjoint_tail_segments %d must be >= -1", c->adjoint_tail_segments);
    if (c->order < LBM_ORDER_REFERENCE || c->order > LBM_ORDER_SAILFISH)
        return fail(LBM_EINVAL, "lbm_init: unknown summation order %d", c->order);
    if (c->order == LBM_ORDER_SAILFISH && c->precision != LBM_FP32 && c->precision != LBM_FP64)
        return fail(LBM_EINVAL, "lbm_init: the Sailfish summation order needs FP32 or FP64 storage");
    if (c->graph_iterations < 0 || c->graph_iterations > 256 || (c->graph_iterations > 1 && c->graph_iterations % 2))
        return fail(LBM_EINVAL, "lbm_init: graph_iterations %d must be 0, 1 or an even number <= 256",
                    c->graph_iterations);
    if (c->block_threads < 0 || c->block_threads > 1024)
        return fail(LBM_EINVAL, "lbm_init: block_threads %d out of range", c->block_threads);
    if (c->lid_profile) {
        for (size_t k = 0; k < (size_t)dim * dim; ++k)
            if (!std::isfinite(c->lid_profile[k])) return fail(LBM_EINVAL, "lbm_init: lid_profile[%zu] not finite", k);
    }

    const int V = vec_len(prec);
    const size_t nvec = (size_t)(dim / V) * (size_t)(dim - 2) * (size_t)(dim - 2);
    unsigned block = c->block_threads > 0 ? (unsigned)(c->block_threads / 32 * 32) : 128u;
    if (block < 32) block = 32;
    // the iteration kernels' launch bounds: 128 threads for 16-bit storage
    const unsigned max_block = (prec == LBM_FP16 || prec == LBM_BF16) ? 128u : 256u;
    if (block > max_block) block = max_block;
    // reduction partials: one pair per block of the widest launch (the AA
    // variant's FP32 kernels use 8-byte vectors, twice the threads)
    const int Vr = (c->kernel == LBM_KERNEL_AA && prec == LBM_FP32) ? V / 2 : V;
    const size_t grid = ((size_t)(dim / Vr) * (size_t)(dim - 2) * (size_t)(dim - 2) + block - 1) / block;
    if (2 * nvec >= ((size_t)1 << 32)) return fail(LBM_EINVAL, "lbm_init: lattice too large");

    const size_t sb = storage_bytes(prec), mb = macro_bytes(prec);
    const size_t fbytes = (size_t)lbm::Q * n * sb;
    const size_t stage_elems = std::min(kStageElems, (size_t)lbm::Q * n);
    const bool aa = c->kernel == LBM_KERNEL_AA;  // one lattice
    const size_t need = (aa ? 1 : 2) * fbytes + n + 4 * n * mb + (size_t)dim * dim * mb + stage_elems * dump_elem(prec) +
                        (grid + 2) * 2 * sizeof(double) + 4 * sizeof(double) + sizeof(int);
    if (c->max_device_bytes > 0 && need > c->max_device_bytes)
        return fail(LBM_ENOMEM, "lbm_init: needs %zu device bytes, budget is %zu", need, c->max_device_bytes);

    lbm_t *h = new lbm_t();
    h->cfg = *c;
    h->cfg.lid_profile = nullptr;
    h->dim = dim;
    h->n = n;
    h->prec = prec;
    h->V = V;
    h->sd = sd;
    h->block = block;
    h->base_bytes = need;

    // tau = 3 nu + 0.5 and 1/tau in the compute precision (kernels.cl:61-62)
    if (prec == LBM_FP64) {
        const double tau = c->tau > 0 ? c->tau : (3.0 * c->viscosity) + 0.5;
        h->inv_tau = 1.0 / tau;
    } else {
        const float tau = c->tau > 0 ? (float)c->tau : (3.0f * (float)c->viscosity) + 0.5f;
        const float it = 1.0f / tau;
        h->inv_tau = (double)it;
    }
    h->omega_f = (float)h->inv_tau;
    if (!std::isfinite(h->inv_tau) || h->inv_tau <= 0)
        { release(h); return fail(LBM_EINVAL, "lbm_init: tau must be > 0"); }

    int rc = LBM_OK;
    auto setup = [&]() -> int {
        LBM_CUDA(cudaSetDevice(c->device));
        LBM_CUDA(device_facts(c->device, h->device_name, h->num_sms));
        h->graph_iters = c->graph_iterations == 0 ? 16 : c->graph_iterations;
        LBM_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        LBM_CUDA(cudaEventCreate(&h->ev_first));
        LBM_CUDA(cudaEventCreate(&h->ev_last));
        LBM_CUDA(lbm::device_alloc(h, &h->f[0], fbytes));
        if (!aa) LBM_CUDA(lbm::device_alloc(h, &h->f[1], fbytes));
        LBM_CUDA(lbm::device_alloc(h, (void **)&h->map, n));
        LBM_CUDA(lbm::device_alloc(h, &h->rho, n * mb));
        LBM_CUDA(lbm::device_alloc(h, &h->u, 3 * n * mb));
        LBM_CUDA(lbm::device_alloc(h, &h->lid, (size_t)dim * dim * mb));
        LBM_CUDA(lbm::device_alloc(h, &h->stage, stage_elems * dump_elem(prec)));
        LBM_CUDA(lbm::device_alloc(h, (void **)&h->partials, (grid + 2) * 2 * sizeof(double)));
        LBM_CUDA(lbm::device_alloc(h, (void **)&h->red_out, 4 * sizeof(double)));
        LBM_CUDA(lbm::device_alloc(h, (void **)&h->status, sizeof(int)));
        LBM_CUDA(cudaMemsetAsync(h->status, 0, sizeof(int), h->stream));

        // the wall rows of the second lattice: nothing writes them and no site
        // uses them, but LBM_DUMP_F_RAW shows what reaches the walls' slots, and
        // recycled memory would differ from run to run
        if (!aa) {
            const size_t row = (size_t)dim * sb, plane = row * dim, lattice = n * sb;
            char *f1 = static_cast<char *>(h->f[1]);
            for (size_t at : {(size_t)0, lattice - plane})
                LBM_CUDA(cudaMemset2DAsync(f1 + at, lattice, 0, plane, lbm::Q, h->stream));
            for (size_t at : {(size_t)0, plane - row})
                LBM_CUDA(cudaMemset2DAsync(f1 + at, plane, 0, row, (size_t)lbm::Q * dim, h->stream));
        }

        // lid profile in the macro precision (the reference's VELOCITY is a
        // literal of the kernel's real type, lbmcl.hpp:141)
        std::vector<unsigned char> lidh((size_t)dim * dim * mb);
        for (size_t k = 0; k < (size_t)dim * dim; ++k) {
            const double v = c->lid_profile ? c->lid_profile[k] : c->velocity;
            if (mb == 8) memcpy(&lidh[k * 8], &v, 8);
            else { const float fv = (float)v; memcpy(&lidh[k * 4], &fv, 4); }
        }
        LBM_CUDA(cudaMemcpyAsync(h->lid, lidh.data(), lidh.size(), cudaMemcpyHostToDevice, h->stream));

        lbm::InitArgs ia;
        ia.f = h->f[0];
        ia.map = h->map;
        ia.lid = h->lid;
        ia.rho = h->rho;
        ia.u = h->u;
        ia.dim = dim;
        ia.n = n;
        ia.seed = c->seed;
        ia.noise_sigma = c->noise_sigma;
        ia.noise_sigma_f = (float)c->noise_sigma;
        ia.in_place = aa ? 1 : 0;
        LBM_CUDA(cudaEventRecord(h->ev_first, h->stream));
        switch (prec) {
        case LBM_FP32: LBM_CUDA(lbm::launch_init_f32(ia, h->stream)); break;
        case LBM_FP64: LBM_CUDA(lbm::launch_init_f64(ia, h->stream)); break;
        case LBM_FP16: LBM_CUDA(lbm::launch_init_f16(ia, h->stream)); break;
        default: LBM_CUDA(lbm::launch_init_bf16(ia, h->stream)); break;
        }
        LBM_CUDA(cudaEventRecord(h->ev_last, h->stream));
        // the copy source (lidh) must outlive the copy
        LBM_CUDA(cudaStreamSynchronize(h->stream));

        const int want = c->kernel;
        h->kernel = aa ? LBM_KERNEL_AA : LBM_KERNEL_DIRECT;
        if (want == LBM_KERNEL_NARROW && prec != LBM_FP64) h->kernel = LBM_KERNEL_NARROW;
        h->step_vb = step_shape(want == LBM_KERNEL_NARROW && prec == LBM_FP64 ? LBM_KERNEL_AUTO : want, prec, dim);
        // 64-thread blocks: a finer last wave (FP16 512^3, us per iteration:
        // 32 threads 1539, 64 1527, 96 1556, 128 1558; FP32 200^3: 64 174.6,
        // 128 175.9, 256 183)
        h->step_block = c->block_threads > 0 ? block : 64u;
        if (!h->step_vb && !aa && want != LBM_KERNEL_STAGED) {  // splits(h)
            LBM_CUDA(cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking));
            LBM_CUDA(cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming));
            LBM_CUDA(cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming));
        }
        if (want == LBM_KERNEL_STAGED) {
            const int r = setup_staged(h, c->stages);
            if (r == LBM_OK) h->kernel = LBM_KERNEL_STAGED;
            else if (c->kernel == LBM_KERNEL_STAGED) return r;  // asked for explicitly
        }
        return LBM_OK;
    };
    rc = setup();
    if (rc != LBM_OK) {
        std::string msg = g_err;
        release(h);
        g_err = msg;
        return rc;
    }
    *out = h;
    return LBM_OK;
}

int lbm_step(lbm_t *h, int nsteps, int macro_every)
{
    if (!h) return fail(LBM_EINVAL, "lbm_step: NULL handle");
    const lbm::DeviceScope dev(h->cfg.device);
    if (nsteps < 0 || macro_every < 0) return fail(LBM_EINVAL, "lbm_step: nsteps and macro_every must be >= 0");
    if (nsteps == 0) return LBM_OK;
    h->state_is_init = false;
    h->adj.ready = false;
    int rc = fold_events(h, h->pending.size() > 4096);
    if (rc != LBM_OK) return rc;
    const bool per_step = h->cfg.profile_steps != 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (!per_step) {
        LBM_CUDA(get_event(h, &e0));
        LBM_CUDA(get_event(h, &e1));
        LBM_CUDA(cudaEventRecord(e0, h->stream));
    }
    for (int k = 0; k < nsteps;) {
        // a run of graph_iters plain iterations (no macro output, no
        // per-iteration events) replays the captured graph of this parity
        const int G = h->graph_iters;
        if (!per_step && G > 1 && nsteps - k >= G && !macro_within(h->it, G, macro_every)) {
            LBM_CUDA(replay_graph(h));
            k += G;
            h->it += G;  // G is even: h->cur / h->aa_phase is unchanged
            continue;
        }
        ++k;
        const int64_t it = h->it + 1;
        const bool macro = macro_every != 0 && (it % macro_every) == 0;
        const lbm::StepArgs a = step_args(h, h->cur);
        cudaEvent_t s0 = nullptr, s1 = nullptr;
        if (per_step) {
            LBM_CUDA(get_event(h, &s0));
            LBM_CUDA(get_event(h, &s1));
            LBM_CUDA(cudaEventRecord(s0, h->stream));
        }
        LBM_CUDA(launch_pull(h, macro ? lbm::MODE_STEP_MACRO : lbm::MODE_STEP, a));
        if (per_step) {
            LBM_CUDA(cudaEventRecord(s1, h->stream));
            h->pending.emplace_back(s0, s1);
        }
        flip(h);
        h->it = it;
    }
    if (!per_step) {
        LBM_CUDA(cudaEventRecord(e1, h->stream));
        h->pending.emplace_back(e0, e1);
    }
    LBM_CUDA(cudaEventRecord(h->ev_last, h->stream));
    return LBM_OK;
}

int lbm_sync(lbm_t *h)
{
    if (!h) return fail(LBM_EINVAL, "lbm_sync: NULL handle");
    const lbm::DeviceScope dev(h->cfg.device);
    LBM_CUDA(cudaStreamSynchronize(h->stream));
    int st = 0;
    LBM_CUDA(cudaMemcpy(&st, h->status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st & 1) return fail(LBM_EDIVERGED, "lbm_sync: a density <= 0 or NaN was seen (simulation diverged)");
    if (st & 2) return fail(LBM_ETIMEOUT, "lbm_sync: a kernel's bounded wait expired; its results are not valid");
    return LBM_OK;
}

int lbm_dump(lbm_t *h, int what, void *dst, size_t bytes)
{
    if (!h || !dst) return fail(LBM_EINVAL, "lbm_dump: NULL argument");
    const lbm::DeviceScope dev(h->cfg.device);
    const size_t want = lbm_size(h, what);
    if (want == 0) return fail(LBM_EINVAL, "lbm_dump: unknown quantity %d", what);
    if (bytes != want) return fail(LBM_EINVAL, "lbm_dump: buffer is %zu bytes, quantity %d needs %zu", bytes, what, want);
    switch (what) {
    case LBM_DUMP_F: {
        const int r = move_f(h, dst, true);
        if (r != LBM_OK) return r;
        break;
    }
    case LBM_DUMP_RHO:
        LBM_CUDA(cudaMemcpyAsync(dst, h->rho, bytes, cudaMemcpyDeviceToHost, h->stream));
        break;
    case LBM_DUMP_U:
        LBM_CUDA(cudaMemcpyAsync(dst, h->u, bytes, cudaMemcpyDeviceToHost, h->stream));
        break;
    case LBM_DUMP_MAP_U8:
        LBM_CUDA(cudaMemcpyAsync(dst, h->map, bytes, cudaMemcpyDeviceToHost, h->stream));
        break;
    case LBM_DUMP_MAP: {
        std::vector<uint8_t> m(h->n);
        LBM_CUDA(cudaMemcpyAsync(m.data(), h->map, h->n, cudaMemcpyDeviceToHost, h->stream));
        LBM_CUDA(cudaStreamSynchronize(h->stream));
        int32_t *o = static_cast<int32_t *>(dst);
        for (size_t k = 0; k < h->n; ++k) o[k] = lbm::unpack_cell(m[k]);
        break;
    }
    case LBM_DUMP_F_RAW:
        LBM_CUDA(cudaMemcpyAsync(dst, h->f[h->cur], bytes, cudaMemcpyDeviceToHost, h->stream));
        break;
    }
    LBM_CUDA(cudaEventRecord(h->ev_last, h->stream));
    LBM_CUDA(cudaStreamSynchronize(h->stream));
    return LBM_OK;
}

int lbm_load(lbm_t *h, int what, const void *src, size_t bytes)
{
    if (!h || !src) return fail(LBM_EINVAL, "lbm_load: NULL argument");
    const lbm::DeviceScope dev(h->cfg.device);
    if (what != LBM_DUMP_F && what != LBM_DUMP_F_RAW)
        return fail(LBM_EINVAL, "lbm_load: only LBM_DUMP_F and LBM_DUMP_F_RAW can be loaded");
    const size_t want = lbm_size(h, what);
    if (bytes != want) return fail(LBM_EINVAL, "lbm_load: buffer is %zu bytes, needs %zu", bytes, want);
    h->state_is_init = false;
    h->adj.ready = false;
    if (what == LBM_DUMP_F_RAW) {
        LBM_CUDA(cudaMemcpyAsync(h->f[h->cur], src, bytes, cudaMemcpyHostToDevice, h->stream));
    } else {
        // (the host buffer is only read)
        const int r = move_f(h, const_cast<void *>(src), false);
        if (r != LBM_OK) return r;
    }
    LBM_CUDA(cudaEventRecord(h->ev_last, h->stream));
    LBM_CUDA(cudaStreamSynchronize(h->stream));
    return LBM_OK;
}

int lbm_timing(lbm_t *h, double *total_ms, double *kernels_ms)
{
    if (!h) return fail(LBM_EINVAL, "lbm_timing: NULL handle");
    const lbm::DeviceScope dev(h->cfg.device);
    LBM_CUDA(cudaStreamSynchronize(h->stream));
    int rc = fold_events(h, true);
    if (rc != LBM_OK) return rc;
    float tot = 0;
    LBM_CUDA(cudaEventElapsedTime(&tot, h->ev_first, h->ev_last));
    if (total_ms) *total_ms = tot;
    if (kernels_ms) *kernels_ms = h->kernels_ms;
    return LBM_OK;
}

int lbm_iteration(const lbm_t *h, int64_t *it)
{
    if (!h || !it) return fail(LBM_EINVAL, "lbm_iteration: NULL argument");
    *it = h->it;
    return LBM_OK;
}

void *lbm_stream(lbm_t *h) { return h ? (void *)h->stream : nullptr; }

const char *lbm_device_name(const lbm_t *h) { return h ? h->device_name.c_str() : ""; }

int lbm_reduce(lbm_t *h, double out[3])
{
    if (!h || !out) return fail(LBM_EINVAL, "lbm_reduce: NULL argument");
    const lbm::DeviceScope dev(h->cfg.device);
    const lbm::StepArgs a = step_args(h, h->cur);
    unsigned nparts = 0;
    LBM_CUDA(launch_pull(h, lbm::MODE_REDUCE, a, &nparts));
    LBM_CUDA(lbm::launch_sum_partials(h->partials, (int)nparts, h->red_out, h->stream));
    double r[2];
    LBM_CUDA(cudaMemcpyAsync(r, h->red_out, sizeof r, cudaMemcpyDeviceToHost, h->stream));
    LBM_CUDA(cudaEventRecord(h->ev_last, h->stream));
    LBM_CUDA(cudaStreamSynchronize(h->stream));
    const double d4 = (double)(h->dim - 4);
    out[0] = r[0];
    out[1] = r[1];
    out[2] = d4 * d4 * d4 + d4 * d4;  // FLUID (dim-4)^3 + MOVING (dim-4)^2
    return LBM_OK;
}

void lbm_destroy(lbm_t *h) { release(h); }

int lbm_keep_memory(int device, size_t bytes)
{
    int count = 0;
    LBM_CUDA(cudaGetDeviceCount(&count));
    if (device < 0 || device >= count)
        return fail(LBM_EINVAL, "lbm_keep_memory: device %d of %d", device, count);
    LBM_CUDA(lbm::keep_memory(device, bytes));
    return LBM_OK;
}

}  // extern "C"
