// Small transfers between the host and the device without the copy engines (hostio.cu).
#pragma once

#include "common.cuh"

namespace rmlk {

constexpr int UPLOAD_MAX_JOBS = 16;
struct UploadJob {
    const void* src;  // pinned host memory, 16-byte aligned
    void* dst;        // device, 16-byte aligned
    uint32_t bytes;
};
// Up to 16 copies pinned host -> device as one kernel.
int host_upload(cudaStream_t st, int n, const UploadJob* jobs);

// all_at_once: nobody copies the chunks on as they arrive.
// Device -> pinned host in chunks of DOWNLOAD_CHUNK bytes; flags[i] (pinned host) becomes `seq` when chunk i has arrived.
constexpr size_t DOWNLOAD_CHUNK = 16384;
int host_download(cudaStream_t st, const void* src, size_t bytes, void* dst, uint32_t* flags, uint32_t seq, bool all_at_once);

}  // namespace rmlk
