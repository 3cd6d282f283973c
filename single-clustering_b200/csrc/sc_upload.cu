// sc_upload.cu — copies between large pageable host buffers and the device.
//
// A pageable cudaMemcpyAsync is staged by the CUDA driver through its own pinned
// buffers by one thread, about 10 GB/s here. For the graph arrays (hundreds
// of MB) that copy is most of an end-to-end call, so large uploads go through
// the context's own pinned staging instead: STAGE_LANES host threads each copy
// STAGE_CHUNK-byte chunks of the source into their two pinned buffers and queue
// each chunk's DMA on their own stream, so host copies, transfers and the other
// lanes overlap. The context's stream then waits for every lane.
//
// Results come back the same way in reverse (Download). There the first touch of
// the caller's fresh arrays, page by page, is most of the time, and the lanes
// share it: a 1M x 50, k = 15 kNN build (330 MB of results) took 179 ms with
// plain pageable copies and the roots of the distances on one host thread, 85 ms
// with 8 lanes, the roots on the device and the CSR coming back while the graph
// is built.
#include <thread>

#include "sc_prims.cuh"

namespace sc {

struct Staging {
    cudaStream_t stream[STAGE_LANES] = {};
    cudaEvent_t done[STAGE_LANES][2] = {};  // the last DMA out of each buffer
    unsigned char* buf[STAGE_LANES][2] = {};
};

namespace {

void destroy(Staging* s) {
    for (int l = 0; l < STAGE_LANES; ++l) {
        if (s->stream[l]) cudaStreamSynchronize(s->stream[l]);
        for (int b = 0; b < 2; ++b) {
            if (s->done[l][b]) cudaEventDestroy(s->done[l][b]);
            if (s->buf[l][b]) cudaFreeHost(s->buf[l][b]);
        }
        if (s->stream[l]) cudaStreamDestroy(s->stream[l]);
    }
    delete s;
}

Staging* staging_of(Ctx& c) {
    if (c.staging) return c.staging;
    Staging* s = new Staging();
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < STAGE_LANES && e == cudaSuccess; ++l) {
        e = cudaStreamCreateWithFlags(&s->stream[l], cudaStreamNonBlocking);
        for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
            e = cudaEventCreateWithFlags(&s->done[l][b], cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaHostAlloc((void**)&s->buf[l][b], STAGE_CHUNK, cudaHostAllocDefault);
        }
    }
    if (e != cudaSuccess) {
        destroy(s);
        throw_cuda(e, "pinned staging set-up", __FILE__, __LINE__);
    }
    c.staging = s;
    return s;
}

}  // namespace

void release_staging(Ctx& c) {
    if (c.staging) destroy(c.staging);
    c.staging = nullptr;
}

void upload(Ctx& c, void* dst, const void* src, size_t bytes) {
    if (bytes < STAGE_MIN_BYTES) {
        if (bytes) SC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c.stream));
        return;
    }
    Staging* s = staging_of(c);
    // dst may come from a stream-ordered allocation on the context's stream
    cudaEvent_t ready;
    SC_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ready, c.stream);
    for (int l = 0; l < STAGE_LANES && e == cudaSuccess; ++l) e = cudaStreamWaitEvent(s->stream[l], ready, 0);
    cudaEventDestroy(ready);
    if (e != cudaSuccess) throw_cuda(e, "staged upload set-up", __FILE__, __LINE__);

    const size_t nchunks = (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK;
    cudaError_t lane_err[STAGE_LANES];
    auto lane = [&](int l) {
        cudaError_t le = cudaSetDevice(c.device);
        int which = 0;
        for (size_t k = (size_t)l; k < nchunks && le == cudaSuccess; k += STAGE_LANES) {
            const size_t off = k * STAGE_CHUNK;
            const size_t len = bytes - off < STAGE_CHUNK ? bytes - off : STAGE_CHUNK;
            unsigned char* b = s->buf[l][which];
            le = cudaEventSynchronize(s->done[l][which]);  // this buffer's previous DMA has finished
            if (le != cudaSuccess) break;
            std::memcpy(b, (const unsigned char*)src + off, len);
            le = cudaMemcpyAsync((unsigned char*)dst + off, b, len, cudaMemcpyHostToDevice, s->stream[l]);
            if (le == cudaSuccess) le = cudaEventRecord(s->done[l][which], s->stream[l]);
            which ^= 1;
        }
        lane_err[l] = le;
    };
    std::thread workers[STAGE_LANES - 1];
    for (int l = 1; l < STAGE_LANES; ++l) {
        try {
            workers[l - 1] = std::thread(lane, l);
        } catch (...) {
            lane(l);  // no thread to be had: this thread copies the lane's chunks itself
        }
    }
    lane(0);
    for (int t = 0; t < STAGE_LANES - 1; ++t)
        if (workers[t].joinable()) workers[t].join();
    for (int l = 0; l < STAGE_LANES; ++l)
        if (lane_err[l] != cudaSuccess) throw_cuda(lane_err[l], "staged upload", __FILE__, __LINE__);
    // the context's stream continues once every lane's DMAs are done
    for (int l = 0; l < STAGE_LANES; ++l) {
        cudaEvent_t fin;
        SC_CUDA(cudaEventCreateWithFlags(&fin, cudaEventDisableTiming));
        e = cudaEventRecord(fin, s->stream[l]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(c.stream, fin, 0);
        cudaEventDestroy(fin);
        if (e != cudaSuccess) throw_cuda(e, "staged upload join", __FILE__, __LINE__);
    }
}

// ------------------------------------------------------------ downloads
struct Download::State {
    struct Seg {
        unsigned char* dst;
        const unsigned char* src;
        size_t bytes;
    };
    std::vector<Seg> segs;
    std::thread workers[STAGE_LANES];
    cudaError_t err[STAGE_LANES] = {};
};

Download::Download(Ctx& ctx) : c(ctx), st(new State()) {}

Download::~Download() { join(); }

void Download::join() {
    for (std::thread& t : st->workers)
        if (t.joinable()) t.join();
}

void Download::add(void* dst, const void* src, size_t bytes) {
    if (dst && bytes) st->segs.push_back({(unsigned char*)dst, (const unsigned char*)src, bytes});
}

void Download::start() {
    size_t total = 0;
    for (const State::Seg& s : st->segs) total += s.bytes;
    if (!c.staged_downloads || total < DOWNLOAD_MIN_BYTES) {
        for (const State::Seg& s : st->segs)
            SC_CUDA(cudaMemcpyAsync(s.dst, s.src, s.bytes, cudaMemcpyDeviceToHost, c.stream));
        return;
    }
    Staging* sg = staging_of(c);
    cudaEvent_t ready;  // what the context's stream has queued so far writes the sources
    SC_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    cudaError_t e = cudaEventRecord(ready, c.stream);
    for (int l = 0; l < STAGE_LANES && e == cudaSuccess; ++l) e = cudaStreamWaitEvent(sg->stream[l], ready, 0);
    cudaEventDestroy(ready);
    if (e != cudaSuccess) throw_cuda(e, "staged download set-up", __FILE__, __LINE__);
    State* s = st.get();
    const int device = c.device;
    // chunk k of the segments' concatenated chunks goes to lane k mod STAGE_LANES;
    // a lane copies one buffer out to the caller while the other one fills
    auto lane = [s, sg, device](int l) {
        cudaError_t le = cudaSetDevice(device);
        struct Chunk {
            unsigned char* dst = nullptr;
            size_t len = 0;
        } pending[2];
        int which = 0;
        auto drain = [&](int b) {
            if (!pending[b].dst) return;
            const cudaError_t de = cudaEventSynchronize(sg->done[l][b]);
            if (de == cudaSuccess) std::memcpy(pending[b].dst, sg->buf[l][b], pending[b].len);
            else if (le == cudaSuccess) le = de;
            pending[b].dst = nullptr;
        };
        size_t k = 0;
        for (const State::Seg& seg : s->segs) {
            for (size_t off = 0; off < seg.bytes && le == cudaSuccess; off += STAGE_CHUNK, ++k) {
                if (k % STAGE_LANES != (size_t)l) continue;
                const size_t len = seg.bytes - off < STAGE_CHUNK ? seg.bytes - off : STAGE_CHUNK;
                drain(which);
                if (le != cudaSuccess) break;
                le = cudaMemcpyAsync(sg->buf[l][which], seg.src + off, len, cudaMemcpyDeviceToHost, sg->stream[l]);
                if (le == cudaSuccess) le = cudaEventRecord(sg->done[l][which], sg->stream[l]);
                if (le == cudaSuccess) pending[which] = Chunk{seg.dst + off, len};
                which ^= 1;
                drain(which);
            }
        }
        drain(0);
        drain(1);
        s->err[l] = le;
    };
    for (int l = 0; l < STAGE_LANES; ++l) {
        try {
            st->workers[l] = std::thread(lane, l);
        } catch (...) {
            lane(l);  // no thread to be had: this thread copies the lane's chunks itself
        }
    }
}

void Download::finish() {
    join();
    for (cudaError_t e : st->err)
        if (e != cudaSuccess) throw_cuda(e, "staged download", __FILE__, __LINE__);
    sync(c);
}

namespace {
__global__ void k_widen_labels(const uint32_t* __restrict__ a, uint64_t n, uint64_t* b) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        b[i] = a[i];
}
}  // namespace

void download_labels(Ctx& c, const uint32_t* d_labels, uint64_t n, uint64_t* host_out) {
    if (n == 0) return;
    DBuf<uint64_t> wide(c, n);
    k_widen_labels<<<grid_for(n, 256), 256, 0, c.stream>>>(d_labels, n, wide.get());
    SC_LAUNCH_CHECK();
    c.launches++;
    Download dl(c);
    dl.add(host_out, wide.get(), n * sizeof(uint64_t));
    dl.start();
    dl.finish();
}

}  // namespace sc
