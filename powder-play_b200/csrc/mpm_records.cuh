// mpm_records.cuh -- particle records between the host and the device: the
// reference's 20-word record (src/lib/mpm/kernels/layout.ts:385-437) packed
// from and unpacked into the SoA slots by kernels, and the staged copies that
// carry the records across PCIe.
#pragma once

#include <mutex>

#include "mpm_kernels.cuh"

namespace mpm {

constexpr uint32_t RECORD_WORDS = 20;
constexpr unsigned RECORD_THREADS = 128;
// records moved through the device workspace at a time (88 MB of workspace
// at most per solver, whatever its particle count)
constexpr uint32_t RECORD_SLAB = 1u << 20;

// Slot of every original index that a slot holds (the others keep what they
// had); *corrupt is set when a slot names an index >= total.
__global__ void k_record_slots(const uint32_t *orig, uint32_t n, uint32_t total, uint32_t *slot_of, uint32_t *corrupt);

// The records of original indices request[k] (NULL: first + k), k < count, to
// out (20 words each) and their object ids to ids (NULL: skipped).  An index
// that none of the n slots holds writes model 0xffffffff and sets *missing.
__global__ void k_pack_records(ParticleBuffers b, uint32_t n, const Material *mats, const uint32_t *bonded, const uint32_t *obj,
                               const uint32_t *slot_of, const uint32_t *request, uint32_t first, uint32_t count,
                               float *out, uint32_t *ids, uint32_t *missing);

// The records of all slots to out + 20 * original index (every index has a
// slot); *corrupt as k_record_slots.
__global__ void k_pack_all_records(ParticleBuffers b, uint32_t n, const Material *mats, const uint32_t *bonded,
                                   const uint32_t *obj, float *out, uint32_t *ids, uint32_t *corrupt);

// Sets *unknown when a record holds an unsupported model, an invalid bonded
// marker or a material that is not in the table (the host then looks closer).
__global__ void k_check_records(const float *records, uint32_t count, const Material *mats, uint32_t n_mats,
                                uint32_t *unknown);

// Unpacks checked records into slots slot_base + k as original indices
// orig_base + k; slot_of (NULL: skipped) receives the slot of each index.
__global__ void k_unpack_records(const float *records, uint32_t count, const Material *mats, uint32_t n_mats,
                                 ParticleBuffers b, uint32_t *bonded, uint32_t *slot_of, uint32_t slot_base,
                                 uint32_t orig_base);

// The pinned staging of a device's transfers, shared by its solvers: eight
// chunks of 1 MiB, allocated when first needed and given back with the last
// solver (one solver's own would cost its creation 0.7 ms for a small one and
// 10 ms for a large one).  Each of up to four host threads takes two chunks:
// while the copy engine moves one, the thread copies the other from or to the
// caller's memory.  One transfer uses the chunks at a time; a second that
// comes meanwhile does not wait for it but copies pageable memory directly.
class RecordStage {
public:
    static RecordStage &of(int device);
    void retain();   // a solver of the device starts
    void release();  // and ends

    // Device to host: `bytes` from src; the first split bytes go to dst0, the
    // rest to dst1.  Returns when the caller's memory is written.
    cudaError_t copy_out(cudaStream_t stream, const void *src, size_t bytes, void *dst0, size_t split, void *dst1);
    // Host to device: returns when the caller's memory has been read.
    cudaError_t copy_in(cudaStream_t stream, void *dst, const void *src, size_t bytes);
    // At most CHUNK bytes of pinned memory for kernels of `stream` to read or
    // write, or NULL when a transfer is under way; lend_end, after the kernels
    // are queued (or done), ends the loan.
    void *lend(size_t bytes);
    cudaError_t lend_end(cudaStream_t stream);

    static constexpr size_t CHUNK = 1u << 20;

private:
    static constexpr int WORKERS = 4, PER_WORKER = 2, CHUNKS = WORKERS * PER_WORKER;
    explicit RecordStage(int device) : device_(device) {}
    cudaError_t reserve(int chunks);
    int workers_for(size_t bytes) const;
    int device_;
    std::mutex busy_;  // held during a transfer
    std::mutex users_lock_;
    int users_ = 0;
    unsigned char *chunk_[CHUNKS] = {};
    cudaEvent_t done_[CHUNKS] = {};  // the last copy or kernel that used the chunk
};

}  // namespace mpm
