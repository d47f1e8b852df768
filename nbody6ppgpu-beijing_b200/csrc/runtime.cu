// runtime.cu -- device selection, stream, status word and error policy shared
// by the gpunb_* / gpupot_ / irr_simd_* entry points of libnb6b200.
//
// Device choice mirrors GPUNB_devinit (gpunb.velocity.cu:575-627): the
// GPU_LIST environment variable (space-separated ids) is honoured, first id
// wins since this library drives one GPU per process; NB_GPU_DEVICE is an
// explicit override; otherwise device (irank % device_count), as the
// single-GPU build does (gpunb.gpu.cu:574).
//
// Error policy: the reference asserts and aborts on bad input (NAN_CHECK,
// ni range, gpunb.velocity.cu:40,751,802).  This library does the same by
// default.  nb6_set_abort_on_error_(0) switches to "record and return": the
// call does no work and nb6_last_status_() reports the code.
#include "nb6_common.cuh"
#include "copy_pool.h"

#include <string.h>

static int g_device = -1;
static int g_num_sms = 0;
static cudaStream_t g_stream = nullptr;
static int *g_dev_status = nullptr;
static int *g_status_host = nullptr;   // pinned copy, filled by nb6_status_fetch
static bool g_status_fetched = false;
static bool g_uva = false;
static int g_host_status = 0;
static int g_abort_on_error = 1;
static bool g_abort_env_read = false;

static void read_abort_env() {
    if (g_abort_env_read) return;
    g_abort_env_read = true;
    const char *e = getenv("NB6_ABORT_ON_ERROR");
    if (e) g_abort_on_error = atoi(e) != 0;
}

void nb6_set_host_status(int code) {
    if (g_host_status == 0) g_host_status = code;
}

void nb6_fatal(int code) {
    read_abort_env();
    nb6_set_host_status(code);
    if (g_abort_on_error) {
        fprintf(stderr, "libnb6b200: fatal error code %d, aborting\n", code);
        abort();
    }
}

void nb6_devinit_once(int irank) {
    if (g_device >= 0) return;
    read_abort_env();
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count <= 0) {
        fprintf(stderr, "libnb6b200: no CUDA device visible\n");
        nb6_fatal(NB6_ERR_CUDA);
        return;
    }
    int dev = (irank >= 0 ? irank : 0) % count;
    if (const char *gl = getenv("GPU_LIST")) {
        char buf[256];
        strncpy(buf, gl, sizeof(buf) - 1);
        buf[sizeof(buf) - 1] = 0;
        char *p = strtok(buf, " ,");
        if (p) dev = atoi(p) % count;
    }
    if (const char *nd = getenv("NB_GPU_DEVICE")) dev = atoi(nd) % count;
    g_device = dev;
    NB6_CUDA_CHECK(cudaSetDevice(dev));
    NB6_CUDA_CHECK(cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev));
    NB6_CUDA_CHECK(cudaStreamCreateWithFlags(&g_stream, cudaStreamNonBlocking));
    NB6_CUDA_CHECK(cudaMalloc((void **)&g_dev_status, sizeof(int)));
    NB6_CUDA_CHECK(cudaMemset(g_dev_status, 0, sizeof(int)));
    NB6_CUDA_CHECK(cudaMallocHost((void **)&g_status_host, sizeof(int)));
    *g_status_host = 0;
    int uva = 0;
    NB6_CUDA_CHECK(cudaDeviceGetAttribute(&uva, cudaDevAttrUnifiedAddressing, dev));
    g_uva = uva != 0;
    if (getenv("NB6_VERBOSE")) {
        cudaDeviceProp prop;
        cudaGetDeviceProperties(&prop, dev);
        fprintf(stderr, "# libnb6b200 GPU initialization - rank: %d; device: %d %s; SMs %d\n",
                irank, dev, prop.name, g_num_sms);
    }
}

int nb6_device_id() { return g_device; }
static CopyPool g_pool;
static int g_open_libs = 0;

CopyPool &nb6_copy_pool() {
    g_pool.start(CopyPool::default_parts());
    return g_pool;
}
void nb6_lib_opened() { ++g_open_libs; }
void nb6_lib_closed() {
    if (--g_open_libs <= 0) {
        g_open_libs = 0;
        g_pool.stop();
    }
}

int nb6_num_sms() { return g_num_sms; }
cudaStream_t nb6_stream() { return g_stream; }
int *nb6_dev_status() { return g_dev_status; }

bool nb6_uva() { return g_uva; }

// ----------------------------------------------------------------------------
// Host arrays on their way to the device.  The callers' arrays are pageable;
// a copy from pageable memory goes through the driver's staging on one thread
// (16 GB/s) with some 10 us per call.  Blocks of up to STAGE_MAX bytes are
// copied into one pinned block that a kernel reads over the bus in place (no
// copy to launch); larger ones pass through a ring of pinned chunks, filled
// by the copy threads while the chunks before are uploaded.  Measured on the
// host: gpunb_send_ of 1,024 bodies 36 -> 7 us, of 16,384 47 -> 33 us, of
// 996,147 (56 MB) 3,950 -> 1,560 us.
// ----------------------------------------------------------------------------
static constexpr size_t STAGE_MAX = 512u << 10, POOL_MIN = 256u << 10;
static constexpr size_t CHUNK_MIN = 512u << 10, CHUNK_MAX = 4u << 20;
static constexpr int RING = 3;
static HostBuf<unsigned char> g_stage, g_ring[RING];
static cudaEvent_t g_ring_ev[RING] = {};
static int g_ring_next = 0;
static bool g_stage_busy = false;   // a kernel may still read g_stage

// Bytes [lo, hi) of the block into `to` (the place of byte lo).
static void copy_range(unsigned char *to, const Nb6Seg *seg, int nseg, size_t lo, size_t hi) {
    for (int k = 0; k < nseg; ++k) {
        const size_t a = lo > seg[k].off ? lo : seg[k].off;
        const size_t end = seg[k].off + seg[k].len, b = hi < end ? hi : end;
        if (a < b) memcpy(to + (a - lo), static_cast<const unsigned char *>(seg[k].src) + (a - seg[k].off), b - a);
    }
}

static void copy_range_pool(unsigned char *to, const Nb6Seg *seg, int nseg, size_t lo, size_t hi) {
    if (hi - lo < POOL_MIN) {
        copy_range(to, seg, nseg, lo, hi);
        return;
    }
    CopyPool &pool = nb6_copy_pool();
    const size_t np = (size_t)pool.parts(), len = hi - lo;
    pool.run([&](int p) {
        const size_t a = len * (size_t)p / np, b = len * ((size_t)p + 1) / np;
        copy_range(to + a, seg, nseg, lo + a, lo + b);
    });
}

const void *nb6_stage(const Nb6Seg *seg, int nseg, size_t bytes) {
    if (bytes > STAGE_MAX || !g_uva) return nullptr;
    if (g_stage_busy) NB6_CUDA_CHECK(cudaStreamSynchronize(g_stream));
    g_stage.reserve(STAGE_MAX);
    copy_range_pool(g_stage.ptr, seg, nseg, 0, bytes);
    g_stage_busy = true;
    return g_stage.ptr;
}

void nb6_upload(void *dst, const Nb6Seg *seg, int nseg, size_t bytes, cudaStream_t st) {
    size_t chunk = (bytes / 4 + 4095) / 4096 * 4096;
    chunk = chunk < CHUNK_MIN ? CHUNK_MIN : chunk > CHUNK_MAX ? CHUNK_MAX : chunk;
    for (size_t lo = 0; lo < bytes; lo += chunk) {
        const size_t hi = lo + chunk < bytes ? lo + chunk : bytes;
        const int r = g_ring_next;
        g_ring_next = (g_ring_next + 1) % RING;
        if (!g_ring_ev[r]) NB6_CUDA_CHECK(cudaEventCreateWithFlags(&g_ring_ev[r], cudaEventDisableTiming));
        else NB6_CUDA_CHECK(cudaEventSynchronize(g_ring_ev[r]));
        g_ring[r].reserve(chunk);
        copy_range_pool(g_ring[r].ptr, seg, nseg, lo, hi);
        NB6_CUDA_CHECK(cudaMemcpyAsync(static_cast<unsigned char *>(dst) + lo, g_ring[r].ptr, hi - lo,
                                       cudaMemcpyHostToDevice, st));
        NB6_CUDA_CHECK(cudaEventRecord(g_ring_ev[r], st));
    }
}

// Enqueue a copy of the device status word into pinned host memory; the
// next nb6_check_dev_status after a sync of `st` reads that copy instead of
// doing a synchronous copy of its own.
void nb6_status_fetch(cudaStream_t st) {
    NB6_CUDA_CHECK(cudaMemcpyAsync(g_status_host, g_dev_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    g_status_fetched = true;
}

// The pinned word itself, for a kernel that posts the status word as its last
// act in place of that copy.
int *nb6_status_post() {
    g_status_fetched = true;
    return g_status_host;
}

float nb6_span_ms(const DevSpan *s, cudaStream_t st) {
    DevSpan h{};
    NB6_CUDA_CHECK(cudaStreamSynchronize(st));
    NB6_CUDA_CHECK(cudaMemcpy(&h, s, sizeof(h), cudaMemcpyDeviceToHost));
    return h.t1 > h.t0 ? 1e-6f * (float)(h.t1 - h.t0) : 0.0f;
}

// Read (and clear) the device status word; call after a stream sync.
int nb6_check_dev_status() {
    int st = 0;
    g_stage_busy = false;
    if (g_status_fetched) {
        st = *(volatile int *)g_status_host;
        g_status_fetched = false;
    } else {
        NB6_CUDA_CHECK(cudaMemcpy(&st, g_dev_status, sizeof(int), cudaMemcpyDeviceToHost));
    }
    if (st != 0) {
        NB6_CUDA_CHECK(cudaMemset(g_dev_status, 0, sizeof(int)));
        fprintf(stderr, "libnb6b200: device reported status %d\n", st);
        nb6_fatal(st);
    }
    return st;
}

extern "C" {

// Extension entry points (no reference counterpart): error policy + status.
void nb6_set_abort_on_error_(int *flag) {
    g_abort_env_read = true;
    g_abort_on_error = (*flag != 0);
}

int nb6_last_status_() {
    int s = g_host_status;
    g_host_status = 0;
    return s;
}

int nb6_device_() { return g_device; }

}  // extern "C"
