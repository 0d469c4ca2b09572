// capi_internal.h -- the context object behind sb_context and helpers shared
// by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../include/speckle_b200.h"

struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
};

constexpr int SB_MAX_BANDS = 32;  // equals sbk::SB_BANDS_MAX
constexpr size_t SB_PIN_BYTES = (size_t)1 << 20;  // page-locked block of a context (OutCopies)

struct sb_context {
    int device = 0;
    int numSM = 0;
    int smMajor = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    float timing[4] = {0, 0, 0, 0};
    float stage[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    cudaEvent_t sev[16] = {};  // per-stage event pairs
    cudaStream_t copyStream = nullptr;  // host -> device image bands
    cudaEvent_t chunkEv[SB_MAX_BANDS] = {};  // band k of both images is resident
    int nsev = 0;
    int64_t launches = 0;
    std::string err;
    char* pin = nullptr;                  // SB_PIN_BYTES page-locked bytes, or null (none to be had)
    std::map<std::string, DevBuf> bufs;   // grown on demand, reused across calls
    std::map<std::string, void*> tables;  // constant tables
    size_t tableBytes = 0;                // device bytes of the tables
    cudaError_t noallocPrep = cudaSuccess;  // result of sb_noalloc_prepare at creation
    long long waitNaps = 1LL << 26;  // bounded device waits: 64 ns naps per wait (~4 s)
    int form = SB_FORM_FP32;         // transform form of the complex stage (sb_set_form)
    // launch shapes set by sb_set_tuning (0: the library default); index by
    // window: 16, 24, 32, 48, 64 -> 0..4
    int tuneCmplxThreads[5] = {0, 0, 0, 0, 0};
    int tuneCmplxCtas[5] = {0, 0, 0, 0, 0};
    int tuneTcCtas = 0;
    int tuneAmpsCtas[5] = {0, 0, 0, 0, 0};
    int lastForm = SB_FORM_FP32;     // form the last sb_strack call's complex stage ran
};

int sb_ctx_fail(sb_context* c, int code, const char* fmt, ...);
int sb_ctx_cuda(sb_context* c, cudaError_t e, const char* what);
void* sb_ctx_buf(sb_context* c, const char* name, size_t bytes, cudaError_t* err);
// Workspace for a list of cnt entries that runs *B of them at a time; size(b):
// bytes for b entries.  It has its full size for all but the shortest lists,
// because growing it from call to call stalls the other jobs of a server.
// Where the free memory does not hold that, the list's own size is tried, then
// half of it again and again down to one entry.  Sets *B to the entries of a
// chunk (equal chunks: no short last one); null: not even one entry fits.
template <typename Size>
char* sb_chunk_buf(sb_context* c, const char* name, int cnt, int* B, Size size)
{
    for (int b = cnt < 32 && cnt < *B ? cnt : *B;; b = b > cnt ? cnt : (b + 1) / 2) {
        cudaError_t e;
        char* base = (char*)sb_ctx_buf(c, name, size(b), &e);
        if (!base && b > 1) continue;
        const int chunks = (cnt + b - 1) / b;
        *B = (cnt + chunks - 1) / chunks;
        return base;
    }
}
int sb_image_to_device(sb_context* c, const sb_image* im, const char* name, const void** dptr);
// A constant table of the context: build() gives its elements (double
// precision, rounded once) when it is first asked for.  Later calls only look
// it up: evaluated on every call, the 13,440 cosines of strackw's oversampling
// kernel took 0.18 of 1.56 ms (1024 x 2048, window 64).  The upload is ordered
// with the context's kernels by its stream.
template <typename F>
const void* sb_table(sb_context* c, const std::string& key, F build)
{
    auto it = c->tables.find(key);
    if (it != c->tables.end()) return it->second;
    const auto host = build();
    const size_t bytes = host.size() * sizeof(host[0]);
    void* d = nullptr;
    if (cudaMalloc(&d, bytes) != cudaSuccess) return nullptr;
    if (cudaMemcpyAsync(d, host.data(), bytes, cudaMemcpyHostToDevice, c->stream) != cudaSuccess) {
        cudaFree(d);
        return nullptr;
    }
    c->tables[key] = d;
    c->tableBytes += bytes;
    return d;
}
const float2* tw_table(sb_context* c, int N);
const float2* tau_table(sb_context* c, int W);
// Twiddles of a batched line transform of N1 N2 points in step order
// (fft_batch.cuh).
const float2* batch_tw_table(sb_context* c, int N1, int N2);
// Loads the allocation-free entry point's kernels and its file-scope workspace
// on the current device (noalloc.cu).
cudaError_t sb_noalloc_prepare();

// Arrays carved from one buffer, 16-byte aligned: first the sizes, then the
// pointers.
class Packed {
    size_t bytes_ = 0;

public:
    size_t add(size_t bytes)
    {
        const size_t at = bytes_;
        bytes_ += (bytes + 15) / 16 * 16;
        return at;
    }
    size_t bytes() const { return bytes_; }
};

// The output copies of one call.  A copy into pageable memory occupies the
// host for about 10 us whatever its size and the next one starts only then, so
// the copies of a small call go to the context's page-locked block back to
// back and are moved on by the host after one synchronisation.  What no longer
// fits into the block (1 MB; there the bytes cost more than the calls) is
// copied straight to its destination, as are grids that stay on the device.
// Sources that follow one another on the device (Packed) go as one copy: each
// takes 3.5 us on the device.  Host results of 256 x 512, window 32: 81 us
// copied one by one, 25 back to back, 15 as one; a batch of 24 tiles (123
// arrays): 5.1, 3.8 and 3.3 ms for the whole call.
class OutCopies {
    struct Part {
        void* dst;
        size_t at, bytes;
    };
    sb_context* c_;
    std::vector<Part> parts_;
    const char* src_ = nullptr;  // the copy being put together: len_ bytes of src_
    size_t len_ = 0, used_ = 0;  // to pin + used_

    cudaError_t flush()
    {
        if (!len_) return cudaSuccess;
        const cudaError_t e = cudaMemcpyAsync(c_->pin + used_, src_, len_, cudaMemcpyDeviceToHost, c_->stream);
        used_ += (len_ + 15) / 16 * 16;
        len_ = 0;
        return e;
    }

public:
    explicit OutCopies(sb_context* c) : c_(c) {}
    int add(void* dst, const void* src, size_t bytes, bool onDevice = false)
    {
        const char* p = (const char*)src;
        cudaError_t e = cudaSuccess;
        if (onDevice) {
            e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, c_->stream);
        } else {
            const bool next = len_ && p >= src_ + len_ && p < src_ + len_ + 16;
            if (!next) e = flush();
            const size_t off = next ? (size_t)(p - src_) : 0;
            if (e != cudaSuccess) {
            } else if (!c_->pin || used_ + off + bytes > SB_PIN_BYTES) {
                e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c_->stream);
            } else {
                if (!next) src_ = p;
                len_ = off + bytes;
                parts_.push_back({dst, used_ + off, bytes});
            }
        }
        return sb_ctx_cuda(c_, e, "cudaMemcpyAsync(output)");
    }
    // Waits for the stream; the destinations are then written.
    int finish(const char* what)
    {
        cudaError_t e = flush();
        if (e == cudaSuccess) e = cudaEventRecord(c_->ev[3], c_->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c_->stream);
        if (e != cudaSuccess) return sb_ctx_cuda(c_, e, what);
        for (const Part& q : parts_) memcpy(q.dst, c_->pin + q.at, q.bytes);
        return SB_OK;
    }
};
