// Host <-> device copies of row blocks between pageable host arrays and the
// padded device fields, through pinned staging buffers filled and drained by
// several host threads at once. A pageable cudaMemcpy runs at the speed of
// one driver staging thread; here each worker thread owns two pinned slots
// and its own stream, so host memcpy, PCIe transfer and the other workers
// overlap.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "wca_sim_internal.h"

using fcab::RowCopy;

namespace {

constexpr int MAX_DEV = 16;
constexpr int MAX_WORKERS = 16;
constexpr size_t SLOT = 4u << 20;    // bytes per pinned slot

struct Worker {
    cudaStream_t st = nullptr;
    char *slot[2] = {nullptr, nullptr};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaEvent_t done = nullptr;
};

struct Pool {
    bool ready = false;
    int n = 0;
    Worker w[MAX_WORKERS];
    cudaEvent_t start = nullptr;
};

std::mutex g_mu;
Pool g_pool[MAX_DEV];

int workers_wanted()
{
    if (const char *e = getenv("FCAB_COPY_THREADS")) {
        const int v = atoi(e);
        if (v >= 1)
            return std::min(v, MAX_WORKERS);
    }
    const unsigned hc = std::thread::hardware_concurrency();
    return (int)std::max(1u, std::min(8u, hc / 2));
}

cudaError_t ensure(Pool &p)
{
    if (p.ready)
        return cudaSuccess;
    // resources made by an earlier, failed attempt are kept and not remade
    cudaError_t e;
    p.n = workers_wanted();
    if (!p.start && (e = cudaEventCreateWithFlags(&p.start, cudaEventDisableTiming)) != cudaSuccess)
        return e;
    for (int i = 0; i < p.n; i++) {
        Worker &w = p.w[i];
        if (!w.st && (e = cudaStreamCreateWithFlags(&w.st, cudaStreamNonBlocking)) != cudaSuccess)
            return e;
        if (!w.done && (e = cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming)) != cudaSuccess)
            return e;
        for (int k = 0; k < 2; k++) {
            if (!w.slot[k] && (e = cudaMallocHost(&w.slot[k], SLOT)) != cudaSuccess)
                return e;
            if (!w.ev[k] && (e = cudaEventCreateWithFlags(&w.ev[k], cudaEventDisableTiming)) != cudaSuccess)
                return e;
        }
    }
    p.ready = true;
    return cudaSuccess;
}

// Rows [r0, r0 + nr) of field f.
struct Chunk {
    const RowCopy *f;
    size_t r0, nr;
    char *dev() const { return (char *)f->dev + r0 * f->dpitch; }
    char *host() const { return (char *)f->host + r0 * f->row_bytes; }
    size_t bytes() const { return nr * f->row_bytes; }
};

// A worker takes chunks from the shared counter: host -> device.
cudaError_t h2d_worker(Worker &w, const std::vector<Chunk> &ch, std::atomic<size_t> &next)
{
    cudaError_t e = cudaSuccess;
    int k = 0;
    for (size_t c; e == cudaSuccess && (c = next.fetch_add(1)) < ch.size(); k ^= 1) {
        const Chunk &x = ch[c];
        if ((e = cudaEventSynchronize(w.ev[k])) != cudaSuccess)   // the slot's last copy
            break;
        memcpy(w.slot[k], x.host(), x.bytes());
        e = cudaMemcpy2DAsync(x.dev(), x.f->dpitch, w.slot[k], x.f->row_bytes, x.f->row_bytes,
                              x.nr, cudaMemcpyHostToDevice, w.st);
        if (e == cudaSuccess)
            e = cudaEventRecord(w.ev[k], w.st);
    }
    return e;
}

// Device -> host, one copy in flight while the previous slot drains.
cudaError_t d2h_worker(Worker &w, const std::vector<Chunk> &ch, std::atomic<size_t> &next)
{
    cudaError_t e = cudaSuccess;
    const Chunk *pend = nullptr;    // chunk in flight in slot k ^ 1
    int k = 0;
    auto drain = [&](const Chunk &x, int slot) -> cudaError_t {
        const cudaError_t ee = cudaEventSynchronize(w.ev[slot]);
        if (ee == cudaSuccess)
            memcpy(x.host(), w.slot[slot], x.bytes());
        return ee;
    };
    for (size_t c; e == cudaSuccess && (c = next.fetch_add(1)) < ch.size(); k ^= 1) {
        const Chunk &x = ch[c];
        e = cudaMemcpy2DAsync(w.slot[k], x.f->row_bytes, x.dev(), x.f->dpitch, x.f->row_bytes,
                              x.nr, cudaMemcpyDeviceToHost, w.st);
        if (e == cudaSuccess)
            e = cudaEventRecord(w.ev[k], w.st);
        if (e == cudaSuccess && pend)
            e = drain(*pend, k ^ 1);
        pend = &x;
    }
    if (e == cudaSuccess && pend)
        e = drain(*pend, k ^ 1);
    return e;
}

// All fields' rows in chunks over the workers. A chunk is a slot at most, and
// small enough that every worker gets a few: one 4 MB field in one chunk went
// through one worker, its memcpy and its transfer one after the other. Measured
// for whole uploads (field after field in 4 MB chunks over four threads before,
// all fields over up to eight now): 1024^2 2.8 -> 1.9 ms, 4096^2 18.3 -> 9.3.
cudaError_t run_copies(const RowCopy *f, int nf, cudaStream_t stream, bool to_device)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    size_t total = 0;
    bool wide = dev < 0 || dev >= MAX_DEV;
    for (int i = 0; i < nf; i++) {
        total += f[i].rows * f[i].row_bytes;
        wide = wide || f[i].row_bytes > SLOT;
    }
    if (total == 0)
        return cudaSuccess;
    if (wide) {
        // rows wider than a slot: pageable copies
        for (int i = 0; i < nf && e == cudaSuccess; i++)
            e = to_device ? cudaMemcpy2DAsync(f[i].dev, f[i].dpitch, f[i].host, f[i].row_bytes,
                                              f[i].row_bytes, f[i].rows, cudaMemcpyHostToDevice,
                                              stream)
                          : cudaMemcpy2DAsync(f[i].host, f[i].row_bytes, f[i].dev, f[i].dpitch,
                                              f[i].row_bytes, f[i].rows, cudaMemcpyDeviceToHost,
                                              stream);
        return e == cudaSuccess && !to_device ? cudaStreamSynchronize(stream) : e;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    Pool &p = g_pool[dev];
    if ((e = ensure(p)) != cudaSuccess)
        return e;
    const size_t want = std::min(SLOT, std::max<size_t>(256u << 10, total / (4 * (size_t)p.n)));
    std::vector<Chunk> ch;
    for (int i = 0; i < nf; i++) {
        const size_t step = std::max<size_t>(1, want / std::max<size_t>(1, f[i].row_bytes));
        for (size_t r = 0; r < f[i].rows; r += step)
            ch.push_back(Chunk{&f[i], r, std::min(step, f[i].rows - r)});
    }
    // a thread costs about as much to start as 256 KB take to copy
    const size_t most = std::max<size_t>(1, total / (512u << 10));
    const int n = (int)std::min<size_t>({(size_t)p.n, ch.size(), most});
    // the copies follow the work already queued on `stream`
    if ((e = cudaEventRecord(p.start, stream)) != cudaSuccess)
        return e;
    for (int t = 0; t < n; t++)
        if ((e = cudaStreamWaitEvent(p.w[t].st, p.start, 0)) != cudaSuccess)
            return e;
    std::vector<cudaError_t> errs((size_t)n, cudaSuccess);
    std::vector<std::thread> th;
    std::atomic<size_t> next{0};
    auto body = [&](int t) {
        cudaSetDevice(dev);
        errs[(size_t)t] = to_device ? h2d_worker(p.w[t], ch, next) : d2h_worker(p.w[t], ch, next);
    };
    for (int t = 1; t < n; t++)
        th.emplace_back(body, t);
    body(0);
    for (auto &x : th)
        x.join();
    for (int t = 0; t < n; t++)
        if (errs[(size_t)t] != cudaSuccess)
            return errs[(size_t)t];
    // later work on `stream` follows the copies
    for (int t = 0; t < n; t++) {
        if ((e = cudaEventRecord(p.w[t].done, p.w[t].st)) != cudaSuccess ||
            (e = cudaStreamWaitEvent(stream, p.w[t].done, 0)) != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

}  // namespace

namespace fcab {

cudaError_t h2d_rows(const RowCopy *f, int n, cudaStream_t stream)
{
    return run_copies(f, n, stream, true);
}

cudaError_t d2h_rows(const RowCopy *f, int n, cudaStream_t stream)
{
    return run_copies(f, n, stream, false);
}

}  // namespace fcab
