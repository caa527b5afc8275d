// Batched input value checks: one launch evaluates every finiteness / range /
// structure check that input validation needs and marks each failed check, so
// the host waits once instead of synchronising once per check (the reference's
// _validation.py evaluates each with its own torch reduction and host read).
// Also the small host <-> device transfers of the explicit operators: counts
// read back and constants written, neither stopping the stream.
//
// The operators' checks are marked by plain byte stores into pinned host
// memory. A call whose inputs are valid then writes nothing at all, and needs
// neither the memset of a device word nor the copy that brings it back: one
// launch and one event. These calls are bound by their host time: a fitting step
// of 2,000 primitives (4 views of 64^2 and a 32^3 volume, four checked calls)
// took 978 us with a device word, torch events and copies from pageable memory
// for the extents, 676 us with the entries below and cheaper handles in the
// loader, of which 290 us are kernels.
#include "common.cuh"

#include <string.h>

namespace r2s {

constexpr uint32_t kMaxChecks = 32;

// Check c runs on blocks [first[c], first[c + 1]).
struct CheckList {
    r2s_value_check item[kMaxChecks];
    uint32_t first[kMaxChecks + 1];
    uint32_t count;
};

template <typename S>
__device__ __forceinline__ bool element_fails(const S* data, uint64_t i, uint32_t kind) {
    switch (kind) {
        case R2S_CHECK_FINITE:
            return !isfinite(data[i]);
        case R2S_CHECK_ZERO_ROW4: {
            const S* row = data + 4 * i;
            return row[0] == S(0) && row[1] == S(0) && row[2] == S(0) && row[3] == S(0);
        }
        case R2S_CHECK_POSITIVE:
            return data[i] <= S(0);
        case R2S_CHECK_NONNEGATIVE:
            return data[i] < S(0);
        case R2S_CHECK_FOCAL: {
            const S* k = data + 9 * i;
            return k[0] <= S(0) || k[4] <= S(0);
        }
        case R2S_CHECK_PINHOLE: {
            const S* k = data + 9 * i;
            return k[1] != S(0) || k[3] != S(0) || k[6] != S(0) || k[7] != S(0) || k[8] != S(1);
        }
        case R2S_CHECK_HOMOGENEOUS_ROW: {
            const S* m = data + 16 * i;
            return !(m[12] == S(0) && m[13] == S(0) && m[14] == S(0) && m[15] == S(1));
        }
        default:
            return true;
    }
}

// 16-byte vectors of S for the finiteness scan.
template <typename S> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };

__device__ __forceinline__ bool any_nonfinite(const float4& v) {
    return !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
}
__device__ __forceinline__ bool any_nonfinite(const double2& v) { return !(isfinite(v.x) && isfinite(v.y)); }

// Where a failed check is marked: a bit of a device word, or a byte of pinned host memory.
struct WordMark {
    uint32_t* word;
    __device__ __forceinline__ void set(uint32_t bit) const { atomicOr(word, 1u << bit); }
};
struct HostMark {
    uint8_t* bytes;  // every writer stores the same 1
    __device__ __forceinline__ void set(uint32_t bit) const { *static_cast<volatile uint8_t*>(bytes + bit) = 1; }
};

// Each check has the blocks its own elements need (launch_checks); a block
// looks its check up in the table. The finiteness check of 16-byte-aligned data
// (the image and volume adjoints, hundreds of MB) reads 16-byte vectors, four
// in flight per thread; the other checks read element by element. (A grid as
// wide as the longest check for every check spent most of its blocks on
// nothing: the four calls of a fitting step of 100,000 Beta primitives, 32
// views of 384^2 and a 192^3 volume took 52 us, and take 22.)
template <typename S, typename Mark>
__global__ void check_values_kernel(CheckList list, Mark mark) {
    uint32_t c = 0;
    while (c + 1 < list.count && blockIdx.x >= list.first[c + 1]) ++c;
    const r2s_value_check chk = list.item[c];
    const S* data = static_cast<const S*>(chk.data);
    const uint64_t tid = uint64_t(blockIdx.x - list.first[c]) * blockDim.x + threadIdx.x;
    const uint64_t stride = uint64_t(list.first[c + 1] - list.first[c]) * blockDim.x;
    bool bad = false;
    if (chk.kind == R2S_CHECK_FINITE && (reinterpret_cast<uintptr_t>(data) & 15u) == 0u) {
        using V = typename Vec16<S>::type;
        constexpr uint64_t kPer = sizeof(V) / sizeof(S);
        const V* vec = reinterpret_cast<const V*>(data);
        const uint64_t nv = chk.count / kPer;
        uint64_t i = tid;
        for (; i + 3 * stride < nv; i += 4 * stride) {
            const V a = vec[i], b = vec[i + stride], d = vec[i + 2 * stride], e = vec[i + 3 * stride];
            bad |= any_nonfinite(a) | any_nonfinite(b) | any_nonfinite(d) | any_nonfinite(e);
        }
        for (; i < nv; i += stride) bad |= any_nonfinite(vec[i]);
        for (uint64_t t = nv * kPer + tid; t < chk.count; t += stride) bad |= !isfinite(data[t]);
    } else {
        for (uint64_t i = tid; i < chk.count; i += stride) bad |= element_fails(data, i, chk.kind);
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31u) == 0u) mark.set(chk.bit);
}

struct Constants {
    double value[R2S_MAX_CONSTANTS];
};

template <typename S>
__global__ void write_constants_kernel(Constants c, uint32_t n, S* __restrict__ dst) {
    if (threadIdx.x < n) dst[threadIdx.x] = S(c.value[threadIdx.x]);
}

// Validates the table and copies it into kernel parameters, without empty checks.
int read_checks(const r2s_value_check* checks, uint32_t n_checks, CheckList& list) {
    R2S_REQUIRE(n_checks <= kMaxChecks, R2S_ERR_UNSUPPORTED, "at most 32 checks per call");
    R2S_REQUIRE(n_checks == 0 || checks != nullptr, R2S_ERR_ARGUMENT, "checks must be non-null");
    list.count = 0;
    for (uint32_t c = 0; c < n_checks; ++c) {
        R2S_REQUIRE(checks[c].bit < 32u, R2S_ERR_ARGUMENT, "check bit must be below 32");
        R2S_REQUIRE(checks[c].kind <= R2S_CHECK_HOMOGENEOUS_ROW, R2S_ERR_ARGUMENT, "unknown check kind");
        R2S_REQUIRE(checks[c].count == 0 || checks[c].data != nullptr, R2S_ERR_ARGUMENT, "check data is null");
        if (checks[c].count != 0) list.item[list.count++] = checks[c];
    }
    return R2S_OK;
}

template <typename Mark>
int launch_checks(int dtype, CheckList& list, Mark mark, cudaStream_t st) {
    if (list.count == 0) return R2S_OK;
    // One pass of a thread's four loads per block, up to eight blocks a SM.
    const uint64_t threads = 256, per_vector = dtype == R2S_F32 ? 4 : 2, most = 1184;
    list.first[0] = 0;
    for (uint32_t c = 0; c < list.count; ++c) {
        const uint64_t per_block = 4 * threads * (list.item[c].kind == R2S_CHECK_FINITE ? per_vector : 1);
        const uint64_t blocks = (list.item[c].count + per_block - 1) / per_block;
        list.first[c + 1] = list.first[c] + uint32_t(blocks < most ? blocks : most);
    }
    const unsigned grid = list.first[list.count];
    R2S_DISPATCH(dtype, check_values_kernel<S><<<grid, unsigned(threads), 0, st>>>(list, mark));
    return check_launch("check_values");
}

// Creates *done and records it on st; nothing is left behind on failure.
int record_done(void** done, cudaStream_t st) {
    cudaEvent_t event = nullptr;
    if (cudaEventCreateWithFlags(&event, cudaEventDisableTiming) != cudaSuccess)
        return fail(R2S_ERR_CUDA, "event creation failed");
    if (cudaEventRecord(event, st) != cudaSuccess) {
        cudaEventDestroy(event);
        return fail(R2S_ERR_CUDA, "event record failed");
    }
    *done = event;
    return R2S_OK;
}

}  // namespace r2s

using namespace r2s;

extern "C" {

int r2s_check_values(int dtype, const r2s_value_check* checks, uint32_t n_checks, uint32_t* flags, void* stream) {
    R2S_REQUIRE(flags != nullptr, R2S_ERR_ARGUMENT, "flags must be non-null");
    CheckList list{};
    R2S_TRY(read_checks(checks, n_checks, list));
    cudaStream_t st = as_stream(stream);
    if (cudaMemsetAsync(flags, 0, sizeof(uint32_t), st) != cudaSuccess) return fail(R2S_ERR_CUDA, "memset failed");
    return launch_checks(dtype, list, WordMark{flags}, st);
}

int r2s_check_values_host(int dtype, const r2s_value_check* checks, uint32_t n_checks, uint8_t* host_flags,
                          void** done, void* stream) {
    R2S_REQUIRE(host_flags != nullptr && done != nullptr, R2S_ERR_ARGUMENT, "host_flags and done must be non-null");
    CheckList list{};
    R2S_TRY(read_checks(checks, n_checks, list));
    void* mapped = nullptr;
    if (cudaHostGetDevicePointer(&mapped, host_flags, 0) != cudaSuccess) {
        cudaGetLastError();
        return fail(R2S_ERR_ARGUMENT, "host_flags must be pinned host memory");
    }
    memset(host_flags, 0, kMaxChecks);
    cudaStream_t st = as_stream(stream);
    R2S_TRY(launch_checks(dtype, list, HostMark{static_cast<uint8_t*>(mapped)}, st));
    const int status = record_done(done, st);
    // The caller may free the flags once this has failed, so the launched kernel must not outlive it.
    if (status != R2S_OK) cudaStreamSynchronize(st);
    return status;
}

int r2s_read_count(const int64_t* count, int64_t* host, void** done, void* stream) {
    R2S_REQUIRE(count != nullptr && host != nullptr && done != nullptr, R2S_ERR_ARGUMENT, "null argument");
    cudaStream_t st = as_stream(stream);
    if (cudaMemcpyAsync(host, count, sizeof(int64_t), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return fail(R2S_ERR_CUDA, "count copy failed");
    const int status = record_done(done, st);
    if (status != R2S_OK) cudaStreamSynchronize(st);
    return status;
}

int r2s_wait_done(void* done) {
    R2S_REQUIRE(done != nullptr, R2S_ERR_ARGUMENT, "done must be non-null");
    const cudaError_t status = cudaEventSynchronize(static_cast<cudaEvent_t>(done));
    cudaEventDestroy(static_cast<cudaEvent_t>(done));
    if (status != cudaSuccess) return fail(R2S_ERR_CUDA, cudaGetErrorString(status));
    return R2S_OK;
}

int r2s_write_constants(int dtype, const double* values, uint32_t n, void* dst, void* stream) {
    R2S_REQUIRE(n <= R2S_MAX_CONSTANTS, R2S_ERR_UNSUPPORTED, "too many constants");
    if (n == 0) return R2S_OK;
    R2S_REQUIRE(values != nullptr && dst != nullptr, R2S_ERR_ARGUMENT, "null argument");
    Constants c{};
    for (uint32_t i = 0; i < n; ++i) c.value[i] = values[i];
    R2S_DISPATCH(dtype, write_constants_kernel<S><<<1, 32, 0, as_stream(stream)>>>(c, n, static_cast<S*>(dst)));
    return check_launch("write_constants");
}

}  // extern "C"
