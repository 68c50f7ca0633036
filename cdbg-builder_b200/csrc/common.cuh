// Shared device/host helpers for the sm_100a kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cstring>
#include <map>
#include <stdexcept>
#include <string>
#include <vector>

namespace cdbg {

typedef unsigned __int128 u128;

extern std::atomic<uint64_t> g_launches;

// Message returned by cdbg_last_error() (thread-local).
void set_last_error(std::string const& msg);

// Per-kernel device time with CUDA events on the launching stream.  Enabled
// per engine call; a scope records an event before and after the launch it
// encloses, and resolve() folds the finished pairs into per-name totals.
struct kernel_profiler {
    struct pending {
        char const* name;
        cudaEvent_t a, b;
    };
    bool on = false;
    std::vector<pending> open;
    std::vector<cudaEvent_t> pool;
    std::map<std::string, std::pair<double, uint64_t>> totals;  // ms, launches
    std::map<std::string, double> bytes;  // algorithmic bytes declared at the launch sites
    cudaEvent_t get() {
        if (!pool.empty()) {
            cudaEvent_t e = pool.back();
            pool.pop_back();
            return e;
        }
        cudaEvent_t e;
        cudaEventCreate(&e);
        return e;
    }
    void resolve() {
        for (auto& p : open) {
            float ms = 0;
            cudaEventSynchronize(p.b);
            cudaEventElapsedTime(&ms, p.a, p.b);
            auto& t = totals[p.name];
            t.first += ms;
            t.second += 1;
            pool.push_back(p.a);
            pool.push_back(p.b);
        }
        open.clear();
    }
    ~kernel_profiler() {
        resolve();
        for (auto e : pool) cudaEventDestroy(e);
    }
};
extern thread_local kernel_profiler* g_prof;

struct prof_scope {
    kernel_profiler* p;
    cudaStream_t st;
    char const* name;
    cudaEvent_t a{};
    prof_scope(char const* n, cudaStream_t s, double alg_bytes = 0)
        : p(g_prof && g_prof->on ? g_prof : nullptr), st(s), name(n) {
        if (p) {
            a = p->get();
            cudaEventRecord(a, st);
            if (alg_bytes > 0) p->bytes[name] += alg_bytes;
        }
    }
    ~prof_scope() {
        if (p) {
            cudaEvent_t b = p->get();
            cudaEventRecord(b, st);
            p->open.push_back({name, a, b});
        }
    }
};
#define CDBG_PROF(name, st) ::cdbg::prof_scope cdbg_prof_scope_(name, st)
// Same, declaring the algorithmic bytes the launch reads and writes (the
// roofline numerator: data it must move, not probes or re-reads).
#define CDBG_PROF_BYTES(name, st, bytes) ::cdbg::prof_scope cdbg_prof_scope_(name, st, (double)(bytes))

#define CDBG_CUDA(call)                                                                        \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            throw std::runtime_error(std::string("CUDA error: ") + cudaGetErrorString(e_) +    \
                                     " at " + __FILE__ + ":" + std::to_string(__LINE__));      \
    } while (0)

// Every kernel launch is followed by this check, which also counts launches
// (the count is exported through cdbg_launch_count()).
#define CDBG_CHECK_LAUNCH()                 \
    do {                                    \
        ::cdbg::g_launches.fetch_add(1);    \
        CDBG_CUDA(cudaGetLastError());      \
    } while (0)

// Device-side error words.  Kernels never trap: a bounded loop that runs out,
// a table that fills up or a size that overflows a field sets a code here and
// the host turns it into an error return after the stage's synchronize.
enum dev_error : uint32_t {
    ERR_NONE = 0,
    ERR_TABLE_FULL = 1,       // open-addressing probe limit reached
    ERR_FIELD_OVERFLOW = 2,   // a value did not fit its packed field
    ERR_BAD_RECORD = 3,       // malformed serialized record
    ERR_CAPACITY = 4,         // an output buffer sized from a bound overflowed
    ERR_CHAIN_LIMIT = 5,      // a chain walk exceeded its step bound
};

__device__ __forceinline__ void set_error(uint32_t* err, uint32_t code) {
    if (err) atomicCAS(err, 0u, code);
}

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

__host__ __device__ __forceinline__ uint64_t ceil_div(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Read 64 bits of a 2-bit-packed base stream starting at base `pos`
// (base i at bits 2*(i%32) of word i/32).  `words` must have one readable
// word past the last base (streams are allocated with padding).
__device__ __forceinline__ uint64_t stream_bits64(uint64_t const* __restrict__ words, uint64_t pos) {
    const uint64_t w = pos >> 5;
    const uint32_t s = (uint32_t)(pos & 31) * 2;
    uint64_t lo = __ldg(words + w) >> s;
    if (s) lo |= __ldg(words + w + 1) << (64 - s);
    return lo;
}

// ---- small device -> host reads
// The host waits for a few bytes of device memory (a count, a flag, digit
// histograms).  With a mailbox installed for the calling thread (mapped pinned
// host memory, installed by the engine for the duration of each call), a
// one-block kernel stores the bytes into it over PCIe, and no copy engine is
// involved: a cudaMemcpyAsync would wait behind the large output copies that
// stream to the host on the engine's copy stream (tens of milliseconds each)
// and stall every batch.  Without a mailbox it is a cudaMemcpyAsync.
struct host_mailbox {
    void* h = nullptr;  // host address
    void* d = nullptr;  // device address of the same pages
    size_t bytes = 0;
    uint32_t seq = 0;   // number of the last delivery
};
extern thread_local host_mailbox* g_mailbox;
// Radix digit width of the sorts run by this host thread's current engine
// call (8 or 11 bits; a performance knob, cdbg_tuning.radix_bits).
extern thread_local int g_radix_bits;
// Device error word of this host thread's current engine call.
extern thread_local uint32_t* g_dev_err;

namespace {
constexpr size_t MAIL_DATA = 64;  // mailbox: the delivery number, then the data
constexpr int MAIL_MAX = 6;       // values of one delivery
struct mail_set {
    uint8_t const* src[MAIL_MAX];
    uint32_t n[MAIL_MAX];
    uint32_t at[MAIL_MAX];  // offset in the mailbox's data
    uint32_t count;
};
__global__ void k_mail(mail_set m, uint8_t* __restrict__ box, uint32_t seq) {
    uint8_t* data = box + MAIL_DATA;
    for (uint32_t j = 0; j < m.count; ++j) {
        uint8_t const* src = m.src[j];
        uint8_t* dst = data + m.at[j];
        if (((uintptr_t)src & 7) == 0 && (m.n[j] & 7) == 0) {
            for (uint32_t i = threadIdx.x; i < m.n[j] / 8; i += blockDim.x)
                reinterpret_cast<uint64_t*>(dst)[i] = reinterpret_cast<uint64_t const*>(src)[i];
        } else {
            for (uint32_t i = threadIdx.x; i < m.n[j]; i += blockDim.x) dst[i] = src[i];
        }
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *(volatile uint32_t*)box = seq;
}

// Device values the host waits for together: add() them, then wait().
class mail_reader {
public:
    explicit mail_reader(cudaStream_t st) : m_st(st) { m_set.count = 0; }
    template <typename T>
    mail_reader& add(T* host_dst, void const* dev_src, size_t bytes = sizeof(T)) {
        if (m_set.count == MAIL_MAX) throw std::runtime_error("mail_reader: too many values");
        m_dst[m_set.count] = host_dst;
        m_set.src[m_set.count] = static_cast<uint8_t const*>(dev_src);
        m_set.n[m_set.count] = (uint32_t)bytes;
        m_set.at[m_set.count] = (uint32_t)m_used;
        m_used += (bytes + 15) & ~size_t(15);
        ++m_set.count;
        return *this;
    }
    void wait() {
        host_mailbox* mb = g_mailbox;
        if (!mb || !mb->h || MAIL_DATA + m_used > mb->bytes) {
            for (uint32_t j = 0; j < m_set.count; ++j)
                CDBG_CUDA(cudaMemcpyAsync(m_dst[j], m_set.src[j], m_set.n[j], cudaMemcpyDeviceToHost, m_st));
            CDBG_CUDA(cudaStreamSynchronize(m_st));
            return;
        }
        const uint32_t seq = ++mb->seq;
        k_mail<<<1, m_used > 512 ? 256 : 32, 0, m_st>>>(m_set, static_cast<uint8_t*>(mb->d), seq);
        CDBG_CHECK_LAUNCH();
        // Short waits watch the delivery number; longer ones (and errors) go
        // to the driver, whose wake-up costs microseconds.
        volatile uint32_t const* flag = static_cast<volatile uint32_t const*>(mb->h);
        bool got = false;
        for (int spin = 0; spin < 20000 && !got; ++spin) {
            got = *flag == seq;
#if defined(__x86_64__)
            if (!got) __builtin_ia32_pause();
#endif
        }
        if (!got) CDBG_CUDA(cudaStreamSynchronize(m_st));
        std::atomic_thread_fence(std::memory_order_acquire);
        for (uint32_t j = 0; j < m_set.count; ++j)
            std::memcpy(m_dst[j], static_cast<uint8_t const*>(mb->h) + MAIL_DATA + m_set.at[j], m_set.n[j]);
        m_set.count = 0;
        m_used = 0;
    }

private:
    cudaStream_t m_st;
    mail_set m_set;
    void* m_dst[MAIL_MAX];
    size_t m_used = 0;
};

inline void read_small(void* host_dst, void const* dev_src, size_t n, cudaStream_t st) {
    mail_reader r(st);
    r.add(static_cast<uint8_t*>(host_dst), dev_src, n);
    r.wait();
}
}  // namespace

}  // namespace cdbg
