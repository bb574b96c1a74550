// The single-product host-buffer call (pm_multiply_host, the fherma_run of the
// drop-in), pipelined.
//
// The caller's a, b, c are usually pageable (the harness's std::vector
// tensors), which the GPU cannot read: every byte goes through pinned staging.
// Done serially that is two host copies of 3.7 MB, an H2D of 7.3 MB, the
// kernels, a D2H of 3.7 MB and a host copy of 3.7 MB, one after the other.
// Here:
//   - the inputs are cut into pieces; a small pool of host threads copies
//     piece k into pinned staging (non-temporal stores) and queues its H2D at
//     once, so staging, the PCIe transfer and the other threads' copies
//     overlap (the reference gets the same overlap from its copy pool and
//     4-chunk input pipeline, host_copy_pool.h, input_pipeline.h:12-54,
//     rns/solve.cu:731-761);
//   - a's conversion starts on a side stream as soon as a's copies are queued,
//     so it runs while b is still on the link; b's conversion, the row and the
//     CRT kernels follow on the plan's stream; the product comes back in
//     pieces, each with an event, and the pool copies piece k out as soon as
//     its event fires, while later pieces are still on the link;
//   - the call is split (begin / end) so that a caller can do its own work --
//     the drop-in allocates the output tensor -- while the GPU runs.
// Pinned caller buffers skip the staging: their pieces are copied directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <immintrin.h>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/polymul.h"
#include "pm_internal.h"

namespace pm {

namespace {

// dst 32-byte aligned, bytes a multiple of 32: 256-bit loads, streaming stores
__attribute__((target("avx2"))) void stream_copy_avx2(void* dst, const void* src, size_t bytes) {
    auto* d = static_cast<__m256i*>(dst);
    auto* s = static_cast<const __m256i*>(src);
    const size_t n = bytes / 32;
    size_t k = 0;
    for (; k + 4 <= n; k += 4) {
        const __m256i x0 = _mm256_loadu_si256(s + k), x1 = _mm256_loadu_si256(s + k + 1);
        const __m256i x2 = _mm256_loadu_si256(s + k + 2), x3 = _mm256_loadu_si256(s + k + 3);
        _mm256_stream_si256(d + k, x0);
        _mm256_stream_si256(d + k + 1, x1);
        _mm256_stream_si256(d + k + 2, x2);
        _mm256_stream_si256(d + k + 3, x3);
    }
    for (; k < n; ++k) _mm256_stream_si256(d + k, _mm256_loadu_si256(s + k));
    _mm_sfence();
}

bool have_avx2() {
    static const bool yes = __builtin_cpu_supports("avx2");
    return yes;
}

// Copy that does not pull the destination into the cache when it can.
void host_copy(void* dst, const void* src, size_t bytes) {
    const uintptr_t d = reinterpret_cast<uintptr_t>(dst);
    if (have_avx2() && bytes >= 4096) {
        const size_t head = (32 - (d & 31)) & 31;
        if (head) std::memcpy(dst, src, head);
        const size_t body = (bytes - head) & ~size_t(31);
        stream_copy_avx2(static_cast<uint8_t*>(dst) + head, static_cast<const uint8_t*>(src) + head, body);
        const size_t tail = bytes - head - body;
        if (tail) std::memcpy(static_cast<uint8_t*>(dst) + head + body, static_cast<const uint8_t*>(src) + head + body, tail);
        return;
    }
    std::memcpy(dst, src, bytes);
}

bool is_pinned(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost;
}

}  // namespace

// How long an idle copy thread spins before it sleeps: PM_HOST_SPIN_US (microseconds,
// read once), 20000 by default.  A caller that leaves longer gaps between products finds
// the threads asleep and waits for them to wake: a harness that writes one case's 3.7 MB
// result and reads the next case's 7.3 MB between calls spends a few milliseconds there,
// and with a 2 ms spin its calls took 15 us longer at N = 32768.  The spin costs the
// pool's threads that long of CPU time after each call; 0 makes them sleep at once.
static long spin_us() {
    static const long us = [] {
        const char* e = std::getenv("PM_HOST_SPIN_US");
        if (!e || !*e) return 20000L;
        char* end = nullptr;
        const long v = std::strtol(e, &end, 10);
        return (end && *end == 0 && v >= 0 && v <= 10000000L) ? v : 20000L;
    }();
    return us;
}

// One host copy in pieces: f(k) for k in [0, pieces), handed out in order, of which the first
// `available` may run yet.
struct CopyJob {
    CopyJob(int n, const std::function<void(int)>& fn) : pieces(n), f(fn) {}
    const int pieces;
    const std::function<void(int)>& f;
    std::atomic<int> available{0}, next{0}, done{0}, inside{0};
    std::mutex error_m;
    std::exception_ptr error;

    // runs one available piece; false when none is left to take now
    bool step() {
        int k = next.load(std::memory_order_relaxed);
        do {
            if (k >= available.load(std::memory_order_acquire)) return false;
        } while (!next.compare_exchange_weak(k, k + 1, std::memory_order_relaxed));
        try {
            f(k);
        } catch (...) {
            std::lock_guard<std::mutex> lock(error_m);
            if (!error) error = std::current_exception();
        }
        done.fetch_add(1, std::memory_order_release);
        return true;
    }
    bool left() const {
        return next.load(std::memory_order_relaxed) < available.load(std::memory_order_acquire);
    }
};

// Host threads that run the pieces of open copy jobs; each job's calling thread takes pieces
// too.  Idle workers spin for a while (back-to-back calls find them awake), then sleep on
// a condition variable.  Every plan of the process shares one pool, made with the first
// plan that needs it and ended with the last: a pool per plan left each plan's threads
// spinning through the other plans' calls, and threads that call at once had eight each to share the
// cores.  N = 32768 on a 16-vCPU host, us a product, a pool per plan / one pool: calls from one thread
// 361 / 353 (three plans in turn 345 / 331), from two with a plan each 317 / 218, from four 482 / 195, from
// eight 739 / 196.  Jobs of calls on several threads are open side by side; workers never wait
// inside a piece, so one call's pending pieces do not hold up another's.
class CopyPool {
public:
    explicit CopyPool(int threads) {
        for (int t = 0; t < threads; ++t) workers_.emplace_back([this] { loop(); });
    }
    ~CopyPool() {
        {
            std::lock_guard<std::mutex> lock(m_);
            stop_ = true;
            generation_.fetch_add(1, std::memory_order_release);
        }
        cv_.notify_all();
        for (auto& w : workers_) w.join();
    }

    // the process's pool, alive while any plan holds it
    static std::shared_ptr<CopyPool> shared(int threads) {
        static std::mutex m;
        static std::weak_ptr<CopyPool> current;
        std::lock_guard<std::mutex> lock(m);
        std::shared_ptr<CopyPool> pool = current.lock();
        if (!pool) {
            pool = std::make_shared<CopyPool>(threads);
            current = pool;
        }
        return pool;
    }

    void open(CopyJob& job, int available) {
        {
            std::lock_guard<std::mutex> lock(m_);
            job.available.store(available, std::memory_order_release);
            jobs_.push_back(&job);
            generation_.fetch_add(1, std::memory_order_release);
        }
        cv_.notify_all();
    }
    // the job's first `available` pieces may run now
    void publish(CopyJob& job, int available) {
        {
            std::lock_guard<std::mutex> lock(m_);
            job.available.store(available, std::memory_order_release);
            generation_.fetch_add(1, std::memory_order_release);
        }
        cv_.notify_all();
    }
    // Ends the job: pieces already taken finish, the rest never start.  With `all`, waits for
    // (and helps with) every piece first and rethrows the first exception a piece threw.
    void close(CopyJob& job, bool all) {
        if (all)
            while (job.done.load(std::memory_order_acquire) < job.pieces)
                if (!job.step()) _mm_pause();
        {
            std::lock_guard<std::mutex> lock(m_);
            jobs_.erase(std::find(jobs_.begin(), jobs_.end(), &job));
        }
        job.next.store(job.pieces, std::memory_order_relaxed);
        while (job.inside.load(std::memory_order_acquire) > 0) _mm_pause();
        if (all && job.error) std::rethrow_exception(job.error);
    }

private:
    // an open job with a piece to take, entered by the calling worker; null when there is none
    CopyJob* enter() {
        for (CopyJob* j : jobs_)
            if (j->left()) {
                j->inside.fetch_add(1, std::memory_order_acq_rel);
                return j;
            }
        return nullptr;
    }
    void loop() {
        uint64_t seen = 0;
        while (true) {
            // spinning a while keeps the threads awake from one half of a product to the next
            // (the GPU's part lasts a few hundred microseconds) and between back-to-back calls
            const auto spin_until = std::chrono::steady_clock::now() + std::chrono::microseconds(spin_us());
            while (generation_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < spin_until)
                _mm_pause();
            std::unique_lock<std::mutex> lock(m_);
            cv_.wait(lock, [&] { return generation_.load() != seen; });
            seen = generation_.load();
            if (stop_) return;
            while (CopyJob* j = enter()) {
                lock.unlock();
                while (j->step()) {
                }
                j->inside.fetch_sub(1, std::memory_order_acq_rel);
                lock.lock();
            }
        }
    }

    std::vector<std::thread> workers_;
    std::mutex m_;
    std::condition_variable cv_;
    std::atomic<uint64_t> generation_{0};
    std::vector<CopyJob*> jobs_;
    bool stop_ = false;
};

namespace {
// Every copy the link makes costs about 3.7 us of its time on top of the bytes (B200,
// PCIe 5: 7.3 MB in 16 copies took 196 us against 139 us in one), so the host threads
// work in small units while the link gets few copies.  A staged input goes in copy
// groups of kGroupUnits units (one round of the threads); the first polynomial's groups
// grow geometrically (1/16, 1/8, 1/4, then the remaining 9/16) so that the link starts
// after a small first round instead of a quarter of the bytes -- the threads stage about
// twice as fast as the link moves -- and the second polynomial, staged while the first is
// on the link, goes in two halves.
constexpr int kGroupUnits = 9;  // staging units per H2D copy
constexpr int kMaxGroups = 6;   // H2D copies of the staged inputs (4 + 2)
constexpr int kOutPieces = 4;   // D2H copies of the product: 1/2, 1/4, 1/8, 1/8 of it, the last
                                // one's copy-out (after everything else) short
static_assert(kMaxGroups * kGroupUnits <= 64 && kOutPieces <= 64, "one ready flag per unit");

// D2H piece k of the product: offset and length
void out_piece(size_t io, int k, size_t* off, size_t* len) {
    const auto cut = [](size_t x) { return x & ~size_t(63); };
    const size_t b1 = cut(io / 2), b2 = b1 + cut(io / 4), b3 = b2 + cut(io / 8);
    const size_t bound[kOutPieces + 1] = {0, b1, b2, b3, io};
    *off = bound[k];
    *len = bound[k + 1] - bound[k];
}

// the H2D copies of the staged inputs: polynomial, byte offset and length of each
struct InGroups {
    int count = 0;
    int poly[kMaxGroups];
    size_t off[kMaxGroups], len[kMaxGroups];
    void add(int p, size_t o, size_t l) {
        poly[count] = p;
        off[count] = o;
        len[count] = l;
        ++count;
    }
};

InGroups input_groups(size_t io, bool pinned_a, bool pinned_b) {
    InGroups g;
    const auto cut = [](size_t x) { return x & ~size_t(63); };
    bool first = true;
    for (int poly = 0; poly < 2; ++poly) {
        if (poly == 0 ? pinned_a : pinned_b) continue;
        if (first) {
            size_t o = 0;
            for (int d = 16; d >= 4; d /= 2) {
                const size_t l = std::min(io - o, cut(io / size_t(d)));
                if (l) g.add(poly, o, l);
                o += l;
            }
            if (io > o) g.add(poly, o, io - o);
            first = false;
        } else {
            const size_t h = std::min(io, cut(io / 2 + 63));
            g.add(poly, 0, h);
            if (io > h) g.add(poly, h, io - h);
        }
    }
    return g;
}

int pool_threads() {
    const unsigned hw = std::thread::hardware_concurrency();
    int t = hw ? int(hw / 2) : 4;
    if (t > 8) t = 8;
    if (t < 1) t = 1;
    return t;
}

// piece k of `bytes` cut into `pieces` runs of 64-byte multiples
void piece(size_t bytes, int pieces, int k, size_t* off, size_t* len) {
    const size_t unit = ((bytes + pieces - 1) / pieces + 63) & ~size_t(63);
    *off = std::min(bytes, unit * size_t(k));
    *len = std::min(bytes, *off + unit) - *off;
}
}  // namespace

HostCall::~HostCall() {
    if (stream) cudaStreamSynchronize(stream);
    if (side) {
        cudaStreamSynchronize(side);
        cudaStreamDestroy(side);
    }
    if (a_in) cudaEventDestroy(a_in);
    if (a_converted) cudaEventDestroy(a_converted);
    for (auto& e : out_ready)
        if (e) cudaEventDestroy(e);
    cudaFree(d_io);
    cudaFreeHost(h_stage);
}

void multiply_host_begin(PlanCore& s, const uint64_t* a, const uint64_t* b, uint64_t* direct_out) {
    if (!s.host) s.host = std::make_unique<HostCall>();
    HostCall& h = *s.host;
    if (h.pending) throw Failure(PM_ERR_BUSY, "a host-buffer product of this plan is still open: end it first");
    if (!h.d_io) {
        h.stream = s.stream;
        cuda_check(cudaMalloc(&h.d_io, 3 * s.io_bytes), "allocate plan I/O buffers");
        // staging for a, b, c, then one word the device error flag is copied into
        cuda_check(cudaMallocHost(&h.h_stage, 3 * s.io_bytes + 64), "allocate pinned staging");
        h.out_ready.assign(kOutPieces, nullptr);
        for (auto& e : h.out_ready) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "output events");
        cuda_check(cudaStreamCreateWithFlags(&h.side, cudaStreamNonBlocking), "conversion stream");
        cuda_check(cudaEventCreateWithFlags(&h.a_in, cudaEventDisableTiming), "input event");
        cuda_check(cudaEventCreateWithFlags(&h.a_converted, cudaEventDisableTiming), "conversion event");
    }
    if (!h.pool) h.pool = CopyPool::shared(pool_threads());
    const size_t io = s.io_bytes;
    uint8_t* dev = static_cast<uint8_t*>(h.d_io);
    uint8_t* stage = static_cast<uint8_t*>(h.h_stage);
    const uint8_t* src[2] = {reinterpret_cast<const uint8_t*>(a), reinterpret_cast<const uint8_t*>(b)};
    const bool pinned[2] = {is_pinned(a), is_pinned(b)};
    // Where the plan converts one polynomial at a time, a's conversion runs on the side
    // stream as soon as a's copies are queued, while b is still on the link.
    const bool split = conversion_splits(s);
    uint32_t* work = s.d_work;
    bool a_aside = false;
    auto convert_a_aside = [&]() {
        cuda_check(cudaEventRecord(h.a_in, h.stream), "input event");
        cuda_check(cudaStreamWaitEvent(h.side, h.a_in, 0), "conversion stream wait");
        launch_tensor_convert_poly(s, reinterpret_cast<const uint32_t*>(dev), 0, work, h.side);
        cuda_check(cudaEventRecord(h.a_converted, h.side), "conversion event");
        a_aside = true;
    };
    // pinned inputs go straight to the link in one copy each
    for (int poly = 0; poly < 2; ++poly)
        if (pinned[poly]) {
            cuda_check(cudaMemcpyAsync(dev + poly * io, src[poly], io, cudaMemcpyHostToDevice, h.stream), "copy in");
            if (split && poly == 0) convert_a_aside();
        }
    // pageable inputs: the pool's threads stage the units (in index order, as they take
    // them) while this thread queues each copy group as soon as its units are staged -- one
    // thread talks to the runtime, so the copies enter the stream without contending
    const InGroups g = input_groups(io, pinned[0], pinned[1]);
    if (g.count) {
        const int nu = g.count * kGroupUnits;
        for (int k = 0; k < nu; ++k) h.ready[k].store(0, std::memory_order_relaxed);
        const std::function<void(int)> stage_unit = [&](int k) {
            const int grp = k / kGroupUnits, poly = g.poly[grp];
            size_t off, len;
            piece(g.len[grp], kGroupUnits, k % kGroupUnits, &off, &len);
            off += g.off[grp];
            if (len) host_copy(stage + poly * io + off, src[poly] + off, len);
            h.ready[k].store(1, std::memory_order_release);
        };
        CopyJob job(nu, stage_unit);
        h.pool->open(job, nu);
        try {
            for (int grp = 0; grp < g.count; ++grp) {
                // stage units too while this copy's are not all ready (the workers may be waking)
                for (int k = grp * kGroupUnits; k < (grp + 1) * kGroupUnits; ++k)
                    while (!h.ready[k].load(std::memory_order_acquire))
                        if (!job.step()) _mm_pause();
                const size_t off = g.off[grp];
                uint8_t* dst = dev + g.poly[grp] * io + off;
                cuda_check(cudaMemcpyAsync(dst, stage + g.poly[grp] * io + off, g.len[grp], cudaMemcpyHostToDevice,
                                           h.stream),
                           "copy in");
                if (split && !a_aside && g.poly[grp] == 0 && (grp + 1 == g.count || g.poly[grp + 1] != 0))
                    convert_a_aside();
            }
        } catch (...) {
            h.pool->close(job, false);
            throw;
        }
        h.pool->close(job, true);
    }
    if (a_aside) {
        launch_tensor_convert_poly(s, reinterpret_cast<const uint32_t*>(dev + io), 1, work, h.stream);
        cuda_check(cudaStreamWaitEvent(h.stream, h.a_converted, 0), "conversion wait");
        launch_tensor_after_conversion(s, reinterpret_cast<uint32_t*>(dev + 2 * io), work, 1, h.stream);
    } else {
        launch_product(s, reinterpret_cast<const uint64_t*>(dev), reinterpret_cast<const uint64_t*>(dev + io),
                       reinterpret_cast<uint64_t*>(dev + 2 * io), nullptr, h.stream);
    }
    // a pinned output takes the product directly; otherwise it lands in the staging
    h.direct_out = direct_out && is_pinned(direct_out) ? reinterpret_cast<uint8_t*>(direct_out) : nullptr;
    uint8_t* land = h.direct_out ? h.direct_out : stage + 2 * io;
    if (h.direct_out) {  // nothing to copy out afterwards: one transfer
        cuda_check(cudaMemcpyAsync(land, dev + 2 * io, io, cudaMemcpyDeviceToHost, h.stream), "copy out");
    } else {
        for (int k = 0; k < kOutPieces; ++k) {
            size_t off, len;
            out_piece(io, k, &off, &len);
            if (len)
                cuda_check(cudaMemcpyAsync(land + off, dev + 2 * io + off, len, cudaMemcpyDeviceToHost, h.stream),
                           "copy out");
            cuda_check(cudaEventRecord(h.out_ready[k], h.stream), "output event");
        }
    }
    // the error word rides on the same stream: no second round trip after the product
    cuda_check(cudaMemcpyAsync(stage + 3 * io, s.d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, h.stream),
               "read error word");
    h.pending = true;
}

void multiply_host_end(PlanCore& s, uint64_t* c) {
    if (!s.host || !s.host->pending) throw Failure(PM_ERR_INVALID, "no host-buffer product of this plan is open");
    HostCall& h = *s.host;
    h.pending = false;
    const size_t io = s.io_bytes;
    uint8_t* stage = static_cast<uint8_t*>(h.h_stage);
    uint8_t* dst = reinterpret_cast<uint8_t*>(c);
    if (h.direct_out && h.direct_out != dst)
        throw Failure(PM_ERR_INVALID, "the product was directed to another output buffer at the start of the call");
    // each product piece leaves the staging as soon as it has landed: this thread polls the
    // pieces' events in order (a blocking wait can sleep for longer than a piece takes) and
    // hands their units to the pool's threads
    if (!h.direct_out) {
        const std::function<void(int)> copy_unit = [&](int k) {  // unit k % 9 of piece k / 9
            size_t poff, plen, off, len;
            out_piece(io, k / kGroupUnits, &poff, &plen);
            piece(plen, kGroupUnits, k % kGroupUnits, &off, &len);
            if (len) host_copy(dst + poff + off, stage + 2 * io + poff + off, len);
        };
        CopyJob job(kOutPieces * kGroupUnits, copy_unit);
        h.pool->open(job, 0);
        try {
            const auto give_up = std::chrono::steady_clock::now() + std::chrono::seconds(60);
            for (int k = 0; k < kOutPieces; ++k) {
                cudaError_t e;
                while ((e = cudaEventQuery(h.out_ready[k])) == cudaErrorNotReady) {
                    if (std::chrono::steady_clock::now() > give_up)
                        throw Failure(PM_ERR_TIMEOUT, "the product did not come back within 60 s");
                    _mm_pause();
                }
                cuda_check(e, "product");
                h.pool->publish(job, (k + 1) * kGroupUnits);
            }
        } catch (...) {
            h.pool->close(job, false);
            throw;
        }
        h.pool->close(job, true);
    }
    cuda_check(cudaStreamSynchronize(h.stream), "product");
    uint32_t herr = 0;
    std::memcpy(&herr, stage + 3 * io, sizeof herr);
    if (herr) check_device_errors(s);
}

void multiply_host(PlanCore& s, const uint64_t* a, const uint64_t* b, uint64_t* c) {
    multiply_host_begin(s, a, b, c);
    multiply_host_end(s, c);
}

}  // namespace pm
