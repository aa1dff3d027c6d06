// Pageable host memory -> device through a small page-locked ring.
//
// One host thread copies at about 15 GB/s and the driver's own path for pageable memory reaches 11;
// the host link takes 53.  So the bytes are copied into the ring piece by piece by a few threads of
// a process-wide pool while the calling thread hands finished pieces to the copy engine in order.
// The ring belongs to the caller and has to stay until the stream has passed the last copy.

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"
#include "stream_copy.h"

namespace pb {

namespace {

constexpr int kPieces = 16;                     // pieces of the ring in flight
constexpr int64_t kPieceBytes = 1 << 20;
constexpr int64_t kDirectBytes = 384 << 10;     // below this one thread is done before the others are awake

struct UploadJob {
    const char* src;
    char* ring;
    int64_t bytes, piece;
    int n;                                      // pieces of the job
    std::atomic<int> next{0};                   // first piece nobody has taken
    std::atomic<int> freed{0};                  // pieces whose ring place has been read by the copy engine
    std::atomic<int> inside{0};                 // workers that hold a pointer to this job
    std::atomic<int> stop{0};                   // a CUDA call failed: nobody waits any more
    std::vector<std::atomic<int>> done;
    explicit UploadJob(int pieces) : n(pieces), done(pieces) {}

    // copies pieces until none is left; `once`: at most one, and only when its place is free
    void work(bool once) {
        for (;;) {
            int p = next.load();
            if (p >= n || stop.load()) return;
            if (p - freed.load() >= kPieces) {
                if (once) return;
                std::this_thread::yield();
                continue;
            }
            if (!next.compare_exchange_weak(p, p + 1)) continue;
            const int64_t off = (int64_t)p * piece;
            stream_copy(ring + (int64_t)(p % kPieces) * piece, src + off, bytes - off < piece ? bytes - off : piece);
            done[p].store(1, std::memory_order_release);
            if (once) return;
        }
    }
};

// Up to seven workers that sleep between jobs, fewer (or none) when the host gives no more threads.
// One job at a time: a second caller copies alone.
class Pool {
   public:
    Pool() {
        int n = (int)std::thread::hardware_concurrency() / 2 - 1;
        n = n < 0 ? 0 : (n > 7 ? 7 : n);
        for (int i = 0; i < n; ++i) {
            try {
                std::thread([this] { loop(); }).detach();
            } catch (const std::system_error&) {
                break;
            }
        }
    }
    bool offer(UploadJob* job) {
        std::lock_guard<std::mutex> lk(mu_);
        if (job_) return false;
        job_ = job;
        ++generation_;
        cv_.notify_all();
        return true;
    }
    void retract(UploadJob* job) {
        {
            std::lock_guard<std::mutex> lk(mu_);
            job_ = nullptr;
        }
        while (job->inside.load()) std::this_thread::yield();
    }

   private:
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            UploadJob* job;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return job_ && generation_ != seen; });
                seen = generation_;
                job = job_;
                job->inside.fetch_add(1);
            }
            job->work(false);
            job->inside.fetch_sub(1);
        }
    }
    std::mutex mu_;
    std::condition_variable cv_;
    UploadJob* job_ = nullptr;
    uint64_t generation_ = 0;
};

Pool& pool() {
    static Pool* p = new Pool();  // (never destroyed: its threads sleep until the process ends)
    return *p;
}

}  // namespace

}  // namespace pb

using namespace pb;

extern "C" int64_t pb_upload_ring_bytes(int64_t bytes) {
    if (bytes <= kDirectBytes) return bytes;
    const int64_t all = (bytes + kPieceBytes - 1) / kPieceBytes;
    return (all < kPieces ? all : kPieces) * kPieceBytes;
}

static int upload(void* dst, const void* src, int64_t bytes, void* ring, int64_t ring_bytes, void* stream_) {
    PB_REQUIRE(bytes >= 0 && (bytes == 0 || (dst && src && ring)), "null buffer");
    PB_REQUIRE(((uintptr_t)ring % 16) == 0, "ring must be 16-byte aligned");
    PB_REQUIRE(ring_bytes >= pb_upload_ring_bytes(bytes), "ring of %lld bytes is too small", (long long)ring_bytes);
    if (bytes == 0) return PB_OK;
    cudaStream_t stream = (cudaStream_t)stream_;
    if (bytes <= kDirectBytes) {
        stream_copy(static_cast<char*>(ring), static_cast<const char*>(src), bytes);
        PB_CUDA_TRY(cudaMemcpyAsync(dst, ring, (size_t)bytes, cudaMemcpyHostToDevice, stream));
        return PB_OK;
    }
    const int n = (int)((bytes + kPieceBytes - 1) / kPieceBytes);
    UploadJob job(n);
    Pool& helpers = pool();
    job.src = static_cast<const char*>(src);
    job.ring = static_cast<char*>(ring);
    job.bytes = bytes;
    job.piece = kPieceBytes;
    cudaEvent_t ev[kPieces] = {};
    cudaError_t err = cudaSuccess;
    const bool reuse = n > kPieces;             // only then a place of the ring is written twice
    for (int i = 0; reuse && i < kPieces && err == cudaSuccess; ++i)
        err = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
    const bool shared = err == cudaSuccess && helpers.offer(&job);
    int freed = 0;
    for (int p = 0; p < n && err == cudaSuccess; ++p) {
        while (!job.done[p].load(std::memory_order_acquire)) {
            if (reuse && freed < p) {           // pieces before p are with the copy engine
                const cudaError_t q = cudaEventQuery(ev[freed % kPieces]);
                if (q == cudaSuccess) {
                    job.freed.store(++freed);
                    continue;
                }
                if (q != cudaErrorNotReady) {
                    err = q;
                    break;
                }
            }
            job.work(true);
        }
        if (err != cudaSuccess) break;
        const int64_t off = (int64_t)p * kPieceBytes;
        const int64_t len = bytes - off < kPieceBytes ? bytes - off : kPieceBytes;
        err = cudaMemcpyAsync(static_cast<char*>(dst) + off, job.ring + (int64_t)(p % kPieces) * kPieceBytes, (size_t)len,
                              cudaMemcpyHostToDevice, stream);
        if (err == cudaSuccess && reuse) err = cudaEventRecord(ev[p % kPieces], stream);
    }
    if (err != cudaSuccess) job.stop.store(1);
    if (shared) helpers.retract(&job);
    for (int i = 0; i < kPieces; ++i)
        if (ev[i]) cudaEventDestroy(ev[i]);
    if (err != cudaSuccess) return fail_cuda(err, "pb_upload");
    return PB_OK;
}

extern "C" int pb_upload(void* dst, const void* src, int64_t bytes, void* ring, int64_t ring_bytes, void* stream) {
    return no_throw("pb_upload", [&] { return upload(dst, src, bytes, ring, ring_bytes, stream); });
}
