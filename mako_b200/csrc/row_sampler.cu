// The reference's one-row, stateful sampler object behind the C ABI: mako::gen::Sampler (src/gen/sampler.hpp:22-45)
// keeps the sampling parameters, the multiset of generated tokens and a std::mt19937_64; so does this handle, with
// the history mirrored in device memory and the uniforms produced on the host exactly as libstdc++'s
// uniform_real_distribution<float> produces them from that generator (one 64-bit draw per uniform), so that the
// same seed gives the reference's token stream. The arithmetic runs in the row pipeline kernel.
#include "row_pipeline.h"

#include <limits>
#include <mutex>
#include <new>
#include <random>
#include <vector>

extern "C" const char* mk_last_error(void);

struct mk_row_sampler {
    mk_sampler* core = nullptr;
    mk_sampling_params params{};
    uint32_t n_vocab = 0;
    int device = 0;
    std::mt19937_64 rng;
    std::vector<int32_t> history;
    int32_t* d_history = nullptr;
    size_t d_history_cap = 0;
    float* d_row = nullptr;     // staging for a host logits row
    // What a call hands the kernel and gets back, in pinned host memory the device reads and writes in place: the uniforms and the
    // draft are read while the row streams, the result is there when the stream is. (As copies of their own around the
    // launch they were most of a call: sample() of one row of 151552 columns 44 us, 37 us so.)
    struct alignas(64) Io {
        float u[2];
        int32_t token, accepted, draft;
    };
    Io* io = nullptr;
    cudaStream_t stream = nullptr;
};

namespace {

// The handle's device for the length of a call; nothing is set where it is current already.
struct OnDevice {
    int prev = -1;
    explicit OnDevice(int device)
    {
        int now = -1;
        if (cudaGetDevice(&now) == cudaSuccess && now != device && cudaSetDevice(device) == cudaSuccess)
            prev = now;
    }
    ~OnDevice()
    {
        if (prev >= 0)
            cudaSetDevice(prev);
    }
};

// Pinned memory is slow to get (2 ms and more, as long as the rest of a sampler takes), so the handles of a process share one
// page of it: 64 places, taken and given back under a lock, allocated by the first handle and freed with the last. More handles
// than places get one of their own.
constexpr int kIoPlaces = 64;
std::mutex g_io_lock;
mk_row_sampler::Io* g_io_page = nullptr;
uint64_t g_io_taken = 0;

mk_row_sampler::Io* io_alloc(size_t n)
{
    void* p = nullptr;
    return cudaHostAlloc(&p, n * sizeof(mk_row_sampler::Io), cudaHostAllocPortable) == cudaSuccess ? static_cast<mk_row_sampler::Io*>(p)
                                                                                                  : nullptr;
}

mk_row_sampler::Io* io_take()
{
    std::lock_guard<std::mutex> hold(g_io_lock);
    if (!g_io_page)
        g_io_page = io_alloc(kIoPlaces);
    if (!g_io_page || g_io_taken == ~0ull)
        return io_alloc(1);
    const int i = __builtin_ctzll(~g_io_taken);
    g_io_taken |= 1ull << i;
    return g_io_page + i;
}

void io_give(mk_row_sampler::Io* io)
{
    std::lock_guard<std::mutex> hold(g_io_lock);
    if (!g_io_page || io < g_io_page || io >= g_io_page + kIoPlaces) {
        cudaFreeHost(io);
        return;
    }
    g_io_taken &= ~(1ull << (io - g_io_page));
    if (g_io_taken == 0) {
        cudaFreeHost(g_io_page);
        g_io_page = nullptr;
    }
}

float next_uniform(std::mt19937_64& g)
{
    // what uniform_real_distribution<float>(0, total) multiplies total with (sampler.cpp:66,100)
    return std::generate_canonical<float, std::numeric_limits<float>::digits>(g);
}

int ensure_history(mk_row_sampler* r)
{
    if (r->history.size() <= r->d_history_cap)
        return MK_OK;
    size_t cap = r->d_history_cap ? r->d_history_cap * 2 : 4096;
    while (cap < r->history.size())
        cap *= 2;
    int32_t* p = nullptr;
    if (cudaMalloc((void**)&p, cap * 4) != cudaSuccess)
        return MK_ERR_CUDA;
    if (r->d_history) {
        cudaMemcpyAsync(p, r->d_history, r->d_history_cap * 4, cudaMemcpyDeviceToDevice, r->stream);
        cudaStreamSynchronize(r->stream);
        cudaFree(r->d_history);
    }
    r->d_history = p;
    r->d_history_cap = cap;
    return MK_OK;
}

const float* device_row(mk_row_sampler* r, const float* logits)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, logits) == cudaSuccess &&
        (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged))
        return logits;
    cudaGetLastError();
    cudaMemcpyAsync(r->d_row, logits, (size_t)r->n_vocab * 4, cudaMemcpyHostToDevice, r->stream);
    return r->d_row;
}

void fill_rows(mk_row_sampler* r, const float* dev_logits, mk_rows& rows)
{
    rows = mk_rows{};
    rows.logits = dev_logits;
    rows.ld = r->n_vocab;
    rows.batch = 1;
    rows.n_vocab = r->n_vocab;
    // the reference counts every accepted token; a history longer than the kernel's 16-bit counters allow would
    // need the long form of the penalty pass
    rows.n_history = (uint32_t)r->history.size();
    rows.history = r->history.empty() ? nullptr : r->d_history;
    rows.history_ld = r->history.size();
    rows.params = r->params;
}

} // namespace

extern "C" {

int mk_row_sampler_create(mk_row_sampler** out, const mk_sampling_params* p, uint32_t n_vocab, uint64_t seed, int device)
{
    if (!out || !p)
        return MK_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    mk_sampler* core = nullptr;
    if (int rc = mk_sampler_create(&core, device, n_vocab, 1))
        return rc;
    mk_row_sampler* r = new (std::nothrow) mk_row_sampler();
    if (!r) {
        mk_sampler_destroy(core);
        return MK_ERR_INVALID_ARGUMENT;
    }
    r->core = core;
    r->params = *p;
    r->n_vocab = n_vocab;
    r->device = device;
    r->rng.seed(seed);
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    bool ok = cudaMalloc((void**)&r->d_row, (size_t)n_vocab * 4) == cudaSuccess &&
              (r->io = io_take()) != nullptr &&
              cudaStreamCreateWithFlags(&r->stream, cudaStreamNonBlocking) == cudaSuccess;
    cudaSetDevice(prev);
    if (!ok) {
        mk_row_sampler_destroy(r);
        return MK_ERR_CUDA;
    }
    *out = r;
    return MK_OK;
}

void mk_row_sampler_destroy(mk_row_sampler* r)
{
    if (!r)
        return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(r->device);
    if (r->d_history) cudaFree(r->d_history);
    if (r->d_row) cudaFree(r->d_row);
    if (r->io) io_give(r->io);
    if (r->stream) cudaStreamDestroy(r->stream);
    cudaSetDevice(prev);
    mk_sampler_destroy(r->core);
    delete r;
}

int mk_row_sampler_greedy(const mk_row_sampler* r)
{
    return r && r->params.temperature <= 0.0f;
}

// Sampler::accept (sampler.cpp:15-18)
int mk_row_sampler_accept(mk_row_sampler* r, int32_t token)
{
    if (!r)
        return MK_ERR_INVALID_ARGUMENT;
    if (r->history.size() >= 65535)
        return MK_ERR_UNSUPPORTED;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(r->device);
    r->history.push_back(token);
    int rc = ensure_history(r);
    if (rc == MK_OK &&
        cudaMemcpyAsync(r->d_history + (r->history.size() - 1), &r->history.back(), 4, cudaMemcpyHostToDevice,
                        r->stream) != cudaSuccess)
        rc = MK_ERR_CUDA;
    cudaSetDevice(prev);
    return rc;
}

// Sampler::sample (sampler.cpp:75-84). logits: host or device pointer to n_vocab floats.
int mk_row_sampler_sample(mk_row_sampler* r, const float* logits, int32_t* token)
{
    if (!r || !logits || !token)
        return MK_ERR_INVALID_ARGUMENT;
    OnDevice here(r->device);
    if (!mk_row_sampler_greedy(r)) // greedy draws nothing from the generator
        r->io->u[0] = next_uniform(r->rng);
    mk_rows rows;
    fill_rows(r, device_row(r, logits), rows);
    mk_sample_out out{};
    out.token = &r->io->token;
    int rc = mk_sampler_sample_batch(r->core, &rows, r->io->u, &out, r->stream);
    if (rc == MK_OK && cudaStreamSynchronize(r->stream) != cudaSuccess)
        rc = MK_ERR_CUDA;
    if (rc == MK_OK)
        *token = *(volatile int32_t*)&r->io->token;
    return rc;
}

// Sampler::verify (sampler.cpp:86-107): one generator draw for the acceptance, one more only after a rejection.
int mk_row_sampler_verify(mk_row_sampler* r, const float* logits, int32_t draft, int32_t* accepted, int32_t* token)
{
    if (!r || !logits || !token || !accepted)
        return MK_ERR_INVALID_ARGUMENT;
    OnDevice here(r->device);
    const bool greedy = mk_row_sampler_greedy(r);
    std::mt19937_64 after_first = r->rng;
    if (!greedy) {
        r->io->u[0] = next_uniform(r->rng);
        after_first = r->rng;
        r->io->u[1] = next_uniform(r->rng);
    }
    r->io->draft = draft;
    mk_rows rows;
    fill_rows(r, device_row(r, logits), rows);
    mk_sample_out out{};
    out.token = &r->io->token;
    int rc = mk_sampler_verify_batch(r->core, &rows, &r->io->draft, r->io->u, r->io->u + 1, &out, &r->io->accepted, r->stream);
    if (rc == MK_OK && cudaStreamSynchronize(r->stream) != cudaSuccess)
        rc = MK_ERR_CUDA;
    if (rc == MK_OK) {
        *token = *(volatile int32_t*)&r->io->token;
        *accepted = *(volatile int32_t*)&r->io->accepted;
        if (!greedy && *accepted)
            r->rng = after_first; // the second draw was not consumed
    }
    return rc;
}

} // extern "C"
