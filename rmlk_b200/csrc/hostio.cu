// Small transfers between the host and the device without the copy engines.
//
// A decode step of one request moves a few hundred bytes in and half a megabyte out.  Through cudaMemcpyAsync every input costs
// 6 us of host time and a stop of the stream while the copy engine takes over, and a pageable read of 512 KB takes 48 us.  The
// kernels here run in the stream's own order, launched under their predecessor's tail like every other kernel of the library: one of
// them fetches all inputs of a run from pinned memory, the other writes an output to pinned memory chunk by chunk, each chunk
// announced by a flag, so that the host copies a chunk out while the next one crosses the bus.
#include "hostio.h"

namespace rmlk {

struct UploadJobs {
    UploadJob job[UPLOAD_MAX_JOBS];
};

__global__ void __launch_bounds__(256) upload_kernel(const __grid_constant__ UploadJobs jobs) {
    dep_sync();
    const UploadJob& j = jobs.job[blockIdx.y];
    const uint32_t units = j.bytes / 16;
    const uint4* src = static_cast<const uint4*>(j.src);
    uint4* dst = static_cast<uint4*>(j.dst);
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < units; i += gridDim.x * 256) dst[i] = src[i];
    if (blockIdx.x == 0 && threadIdx.x < j.bytes % 16)
        static_cast<uint8_t*>(j.dst)[units * 16 + threadIdx.x] = static_cast<const uint8_t*>(j.src)[units * 16 + threadIdx.x];
}

int host_upload(cudaStream_t st, int n, const UploadJob* jobs) {
    UploadJobs p = {};
    uint32_t most = 0;
    for (int i = 0; i < n; i++) {
        p.job[i] = jobs[i];
        most = most > jobs[i].bytes ? most : jobs[i].bytes;
    }
    const unsigned blocks = most <= 4096 ? 1 : (most / 16 + 255) / 256;
    launch_dep(upload_kernel, dim3(blocks < 64 ? blocks : 64, n), dim3(256), 0, st, p);
    RMLK_CHECK_LAUNCH("upload_kernel");
    return RMLK_OK;
}

template <typename T>
__device__ __forceinline__ void copy_chunk(const uint8_t* src, uint8_t* dst, uint32_t n) {
    const uint32_t units = n / sizeof(T);
    for (uint32_t i = threadIdx.x; i < units; i += 512) reinterpret_cast<T*>(dst)[i] = reinterpret_cast<const T*>(src)[i];
    if (threadIdx.x < n % sizeof(T)) dst[units * sizeof(T) + threadIdx.x] = src[units * sizeof(T) + threadIdx.x];
}

// Few CTAs that take the chunks in turn: enough to fill the bus, and the chunks arrive one after the other instead of all at the end,
// so that the host's copy of one overlaps the transfer of the next.
constexpr unsigned DOWNLOAD_CTAS = 8;
__global__ void __launch_bounds__(512) download_kernel(const uint8_t* __restrict__ src, size_t bytes, uint8_t* dst, uint32_t* flags, uint32_t seq) {
    dep_sync();
    for (size_t c = blockIdx.x, at = c * DOWNLOAD_CHUNK; at < bytes; c += gridDim.x, at = c * DOWNLOAD_CHUNK) {
        const uint32_t n = static_cast<uint32_t>(bytes - at < DOWNLOAD_CHUNK ? bytes - at : DOWNLOAD_CHUNK);
        if (reinterpret_cast<uintptr_t>(src) % 16 == 0) copy_chunk<uint4>(src + at, dst + at, n);
        else if (reinterpret_cast<uintptr_t>(src) % 4 == 0) copy_chunk<uint32_t>(src + at, dst + at, n);
        else copy_chunk<uint8_t>(src + at, dst + at, n);
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence_system();
            *reinterpret_cast<volatile uint32_t*>(flags + c) = seq;
        }
    }
}

int host_download(cudaStream_t st, const void* src, size_t bytes, void* dst, uint32_t* flags, uint32_t seq, bool all_at_once) {
    const unsigned ctas = all_at_once ? 32 : DOWNLOAD_CTAS;
    const unsigned chunks = static_cast<unsigned>((bytes + DOWNLOAD_CHUNK - 1) / DOWNLOAD_CHUNK);
    launch_dep(download_kernel, dim3(chunks < ctas ? chunks : ctas), dim3(512), 0, st, static_cast<const uint8_t*>(src), bytes,
               static_cast<uint8_t*>(dst), flags, seq);
    RMLK_CHECK_LAUNCH("download_kernel");
    return RMLK_OK;
}

}  // namespace rmlk
