// mpm_records.cu -- packing and unpacking of the 20-word particle record on
// the device and its staged copies (mpm_records.cuh).
//
// What bounds a read or a write of all particles is the host side: 84 bytes a
// particle over PCIe (54 GB/s into pinned memory) and into the caller's
// pages, which a core writes at 5 GB/s when it touches them first.  The
// kernels move 84 bytes of SoA state and 84 bytes of record per particle: 36 us
// to pack a million.  One million particles on a B200 and its host: read
// 34.9 -> 6.0 ms, write 21.8 -> 2.8 ms; 1,600: read 181 -> 50 us, write 52-105
// -> 40 us; the first figure with the nine SoA arrays copied to or from
// pageable vectors and one core assembling the records.  A read by index packs
// what was asked for (before, every read moved all particles: a scene of a
// batch of 24 1,873 -> 51 us).
#include <algorithm>
#include <cstring>
#include <map>
#include <system_error>
#include <thread>

#include "mpm_records.cuh"

namespace mpm {

namespace {

// One record through shared memory, 5 float4 per thread: a thread's record is
// 80 bytes, so a warp's 128-bit accesses at a stride of 5 float4 touch every
// bank once per quarter warp, and the records leave (or arrive) as the
// contiguous run of the CTA.
struct RecordTile {
    float4 q[RECORD_THREADS * 5];
};

__device__ __forceinline__ void build_record(const ParticleBuffers &b, const Material *mats, const uint32_t *bonded,
                                             uint32_t slot, uint32_t index, float4 (&q)[5])
{
    const float2 x = b.pos[slot], v = b.vel[slot];
    q[0] = make_float4(x.x, x.y, v.x, v.y);
    q[1] = b.C[slot];
    q[2] = b.F[slot];
    const Material m = mats[b.mat[slot]];
    q[3] = make_float4(b.pvol[slot], __uint_as_float(m.model), m.lambda, m.mu);
    // a Neo-Hookean particle keeps its damage in the parameter's word
    q[4] = make_float4(m.density, b.vol[slot], m.model == MODEL_NEO_HOOKEAN ? b.damage[slot] : m.param,
                       __uint_as_float(bonded[index]));
}

// The table's entry of a record (its model, lambda, mu, density and
// parameter by their bits, the first that matches), n_mats when it has none.
__device__ __forceinline__ uint32_t find_material(const Material *mats, uint32_t n_mats, uint32_t model, float lambda,
                                                  float mu, float density, float param)
{
    const uint32_t l = __float_as_uint(lambda), u = __float_as_uint(mu), d = __float_as_uint(density);
    const uint32_t p = model == MODEL_NEO_HOOKEAN ? 0u : __float_as_uint(param);
    for (uint32_t k = 0; k < n_mats; ++k) {
        const Material &t = mats[k];
        if (t.model == model && __float_as_uint(t.lambda) == l && __float_as_uint(t.mu) == u &&
            __float_as_uint(t.density) == d && __float_as_uint(t.param) == p)
            return k;
    }
    return n_mats;
}

}  // namespace

__global__ void __launch_bounds__(RECORD_THREADS) k_record_slots(const uint32_t *orig, uint32_t n, uint32_t total,
                                                                uint32_t *slot_of, uint32_t *corrupt)
{
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    const uint32_t i = orig[d];
    if (i < total)
        slot_of[i] = d;
    else
        *corrupt = 1u;
}

__global__ void __launch_bounds__(RECORD_THREADS) k_pack_records(ParticleBuffers b, uint32_t n, const Material *mats,
                                                                const uint32_t *bonded, const uint32_t *obj,
                                                                const uint32_t *slot_of, const uint32_t *request,
                                                                uint32_t first, uint32_t count, float *out,
                                                                uint32_t *ids, uint32_t *missing)
{
    __shared__ RecordTile tile;
    const uint32_t k0 = blockIdx.x * RECORD_THREADS, k = k0 + threadIdx.x;
    if (k < count) {
        const uint32_t i = request ? request[k] : first + k;
        const uint32_t slot = slot_of[i];
        float4 q[5] = {};
        if (slot < n && b.orig[slot] == i) {
            build_record(b, mats, bonded, slot, i, q);
        } else {
            q[3].y = __uint_as_float(0xffffffffu);
            *missing = 1u;
        }
#pragma unroll
        for (int u = 0; u < 5; ++u) tile.q[threadIdx.x * 5 + u] = q[u];
        if (ids) ids[k] = obj[i];
    }
    __syncthreads();
    const uint32_t quads = min(count - k0, RECORD_THREADS) * 5u;
    float4 *dst = reinterpret_cast<float4 *>(out) + (size_t)k0 * 5;
    for (uint32_t t = threadIdx.x; t < quads; t += RECORD_THREADS) dst[t] = tile.q[t];
}

__global__ void __launch_bounds__(RECORD_THREADS) k_pack_all_records(ParticleBuffers b, uint32_t n,
                                                                    const Material *mats, const uint32_t *bonded,
                                                                    const uint32_t *obj, float *out, uint32_t *ids,
                                                                    uint32_t *corrupt)
{
    __shared__ RecordTile tile;
    __shared__ uint32_t index[RECORD_THREADS];
    const uint32_t d0 = blockIdx.x * RECORD_THREADS, d = d0 + threadIdx.x;
    if (d < n) {
        const uint32_t i = b.orig[d];
        index[threadIdx.x] = i;
        if (i < n) {
            float4 q[5];
            build_record(b, mats, bonded, d, i, q);
#pragma unroll
            for (int u = 0; u < 5; ++u) tile.q[threadIdx.x * 5 + u] = q[u];
            if (ids) ids[i] = obj[i];
        } else {
            *corrupt = 1u;
        }
    }
    __syncthreads();
    const uint32_t quads = min(n - d0, RECORD_THREADS) * 5u;
    // 5 neighbouring threads write one record's 80 bytes
    for (uint32_t t = threadIdx.x; t < quads; t += RECORD_THREADS) {
        const uint32_t i = index[t / 5u];
        if (i < n) reinterpret_cast<float4 *>(out)[(size_t)i * 5 + t % 5u] = tile.q[t];
    }
}

__global__ void __launch_bounds__(RECORD_THREADS) k_check_records(const float *records, uint32_t count,
                                                                 const Material *mats, uint32_t n_mats,
                                                                 uint32_t *unknown)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const float4 a = reinterpret_cast<const float4 *>(records)[(size_t)k * 5 + 3];
    const float4 b = reinterpret_cast<const float4 *>(records)[(size_t)k * 5 + 4];
    const uint32_t model = __float_as_uint(a.y);
    if (model > MODEL_FIXED_COROTATED || __float_as_uint(b.w) > 3u ||
        find_material(mats, n_mats, model, a.z, a.w, b.x, b.z) == n_mats)
        *unknown = 1u;
}

__global__ void __launch_bounds__(RECORD_THREADS) k_unpack_records(const float *records, uint32_t count,
                                                                  const Material *mats, uint32_t n_mats,
                                                                  ParticleBuffers b, uint32_t *bonded,
                                                                  uint32_t *slot_of, uint32_t slot_base,
                                                                  uint32_t orig_base)
{
    __shared__ RecordTile tile;
    const uint32_t k0 = blockIdx.x * RECORD_THREADS, k = k0 + threadIdx.x;
    const uint32_t quads = min(count - k0, RECORD_THREADS) * 5u;
    const float4 *src = reinterpret_cast<const float4 *>(records) + (size_t)k0 * 5;
    for (uint32_t t = threadIdx.x; t < quads; t += RECORD_THREADS) tile.q[t] = __ldcs(src + t);
    __syncthreads();
    if (k >= count) return;
    float4 q[5];
#pragma unroll
    for (int u = 0; u < 5; ++u) q[u] = tile.q[threadIdx.x * 5 + u];
    const uint32_t slot = slot_base + k, index = orig_base + k, model = __float_as_uint(q[3].y);
    b.pos[slot] = make_float2(q[0].x, q[0].y);
    b.vel[slot] = make_float2(q[0].z, q[0].w);
    b.C[slot] = q[1];
    b.F[slot] = q[2];
    b.pvol[slot] = q[3].x;
    b.damage[slot] = model == MODEL_NEO_HOOKEAN ? q[4].z : 0.0f;
    b.vol[slot] = q[4].y;
    b.mat[slot] = find_material(mats, n_mats, model, q[3].z, q[3].w, q[4].x, q[4].z);
    b.orig[slot] = index;
    bonded[index] = __float_as_uint(q[4].w);
    if (slot_of) slot_of[index] = slot;
}

// ----------------------------------------------------------------- host ---

RecordStage &RecordStage::of(int device)
{
    // never destroyed: the chunks are freed with the last solver, and at
    // process exit the driver may already be gone
    static std::mutex lock;
    static std::map<int, RecordStage *> &stages = *new std::map<int, RecordStage *>();
    std::lock_guard<std::mutex> hold(lock);
    RecordStage *&s = stages[device];
    if (!s) s = new RecordStage(device);
    return *s;
}

void RecordStage::retain()
{
    std::lock_guard<std::mutex> hold(users_lock_);
    ++users_;
}

void RecordStage::release()
{
    std::lock_guard<std::mutex> hold(users_lock_);
    if (--users_ > 0) return;
    std::lock_guard<std::mutex> idle(busy_);
    for (int k = 0; k < CHUNKS; ++k) {
        if (done_[k]) cudaEventSynchronize(done_[k]);
        if (done_[k]) cudaEventDestroy(done_[k]);
        if (chunk_[k]) cudaFreeHost(chunk_[k]);
        done_[k] = nullptr;
        chunk_[k] = nullptr;
    }
}

// Allocates the first `chunks` chunks (with busy_ held).
cudaError_t RecordStage::reserve(int chunks)
{
    for (int k = 0; k < chunks; ++k) {
        cudaError_t e = cudaSuccess;
        if (!done_[k]) e = cudaEventCreateWithFlags(&done_[k], cudaEventDisableTiming);
        if (e == cudaSuccess && !chunk_[k])
            e = cudaHostAlloc(reinterpret_cast<void **>(&chunk_[k]), CHUNK, cudaHostAllocPortable);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Host threads for a transfer: one per 2 MiB.
int RecordStage::workers_for(size_t bytes) const
{
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    return (int)std::min<size_t>({(size_t)WORKERS, (size_t)cores, std::max<size_t>(1, bytes / (2 * CHUNK))});
}

namespace {

// Runs job(0) .. job(workers - 1), the first on this thread and the others on
// threads of their own (on this one where a thread cannot be started).
template <class Job>
void run_workers(int workers, const Job &job)
{
    std::thread threads[8];
    int started = 1;
    for (; started < workers; ++started) {
        try {
            threads[started] = std::thread(job, started);
        } catch (const std::system_error &) {
            break;
        }
    }
    job(0);
    for (int w = started; w < workers; ++w) job(w);
    for (int w = 1; w < started; ++w) threads[w].join();
}

}  // namespace

cudaError_t RecordStage::copy_out(cudaStream_t stream, const void *src, size_t bytes, void *dst0, size_t split,
                                  void *dst1)
{
    if (bytes == 0) return cudaSuccess;
    std::unique_lock<std::mutex> hold(busy_, std::try_to_lock);
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    const int workers = workers_for(bytes);
    if (!hold.owns_lock()) {
        const size_t head = std::min(bytes, split);
        cudaError_t e = cudaMemcpyAsync(dst0, src, head, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess && bytes > head)
            e = cudaMemcpyAsync(dst1, (const unsigned char *)src + head, bytes - head, cudaMemcpyDeviceToHost, stream);
        return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
    }
    cudaError_t e = reserve((int)std::min<size_t>(chunks, (size_t)workers * PER_WORKER));
    if (e != cudaSuccess) return e;
    cudaError_t failed[WORKERS] = {};
    run_workers(workers, [&](int w) {
        cudaError_t err = cudaSetDevice(device_);
        auto issue = [&](size_t c, int k) {
            const size_t at = c * CHUNK, n = std::min(CHUNK, bytes - at);
            // the chunk's last copy may belong to another stream
            cudaError_t r = cudaEventSynchronize(done_[k]);
            if (r == cudaSuccess)
                r = cudaMemcpyAsync(chunk_[k], (const unsigned char *)src + at, n, cudaMemcpyDeviceToHost, stream);
            return r == cudaSuccess ? cudaEventRecord(done_[k], stream) : r;
        };
        // chunk c of the transfer goes through slot c mod (workers * 2)
        const size_t slots = (size_t)workers * PER_WORKER;
        for (int u = 0; u < PER_WORKER && err == cudaSuccess; ++u) {
            const size_t c = (size_t)w + (size_t)u * workers;
            if (c < chunks) err = issue(c, (int)(c % slots));
        }
        for (size_t c = w; c < chunks && err == cudaSuccess; c += workers) {
            const int k = (int)(c % slots);
            err = cudaEventSynchronize(done_[k]);
            if (err != cudaSuccess) break;
            const size_t at = c * CHUNK, n = std::min(CHUNK, bytes - at);
            const size_t head = at >= split ? 0 : std::min(n, split - at);
            if (head) std::memcpy((unsigned char *)dst0 + at, chunk_[k], head);
            if (n > head) std::memcpy((unsigned char *)dst1 + (at + head - split), chunk_[k] + head, n - head);
            if (c + slots < chunks) err = issue(c + slots, k);
        }
        failed[w] = err;
    });
    for (int w = 0; w < workers; ++w)
        if (failed[w] != cudaSuccess) return failed[w];
    return cudaSuccess;
}

cudaError_t RecordStage::copy_in(cudaStream_t stream, void *dst, const void *src, size_t bytes)
{
    if (bytes == 0) return cudaSuccess;
    std::unique_lock<std::mutex> hold(busy_, std::try_to_lock);
    if (!hold.owns_lock()) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    const int workers = workers_for(bytes);
    const size_t slots = (size_t)workers * PER_WORKER;
    cudaError_t e = reserve((int)std::min(chunks, slots));
    if (e != cudaSuccess) return e;
    cudaError_t failed[WORKERS] = {};
    run_workers(workers, [&](int w) {
        cudaError_t err = cudaSetDevice(device_);
        for (size_t c = w; c < chunks && err == cudaSuccess; c += workers) {
            const int k = (int)(c % slots);
            const size_t at = c * CHUNK, n = std::min(CHUNK, bytes - at);
            err = cudaEventSynchronize(done_[k]);  // the copy that last used this chunk
            if (err != cudaSuccess) break;
            std::memcpy(chunk_[k], (const unsigned char *)src + at, n);
            err = cudaMemcpyAsync((unsigned char *)dst + at, chunk_[k], n, cudaMemcpyHostToDevice, stream);
            if (err == cudaSuccess) err = cudaEventRecord(done_[k], stream);
        }
        failed[w] = err;
    });
    for (int w = 0; w < workers; ++w)
        if (failed[w] != cudaSuccess) return failed[w];
    return cudaSuccess;
}

void *RecordStage::lend(size_t bytes)
{
    if (bytes > CHUNK || !busy_.try_lock()) return nullptr;
    if (reserve(1) == cudaSuccess && cudaEventSynchronize(done_[0]) == cudaSuccess) return chunk_[0];
    cudaGetLastError();
    busy_.unlock();
    return nullptr;
}

cudaError_t RecordStage::lend_end(cudaStream_t stream)
{
    const cudaError_t e = cudaEventRecord(done_[0], stream);
    busy_.unlock();
    return e;
}

}  // namespace mpm
