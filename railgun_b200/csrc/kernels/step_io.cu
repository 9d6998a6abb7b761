// A decode step's way in and out: the packed step from page-locked host memory into the step's device buffer, and the
// tokens it chose back, by kernels of the step's graph.
//
// What bounds them: latency.  The packed step is 0.5 to 130 KB, a few microseconds of PCIe; as copy nodes of the graph the
// same bytes cost a hand-over to a copy engine and back in front of the first kernel and behind the last, where a kernel
// costs its launch and one round trip over the bus and the kernel behind it starts as any other (alone, one after another: 1.2 KB
// 2.5 us, as a copy 3.6; 132 KB 6.5, as a copy 11.8).  With the host packing the next step meanwhile (below) and the argmax of
// sampling.cu: a step of 1B-sized layers for one request 695 to 676 us, for 64 1,242 to 1,200; a question of 1,999 tokens and
// 16 steps of three 2,048-wide layers 4,721 to 4,489.
//
// The host may write the buffer again once every block has read its part, long before the step is done: the last block to
// finish copies the step's number, which the host wrote beside the buffer, to where the host looks for it.
#include "common.cuh"

#define STEP_IN_THREADS 256

// seq[0]: the number of the step in the buffer (host -> device); seq[1]: the last one read (device -> host).
// done[0]: blocks that have read their part, zero before and after; done[1]: the step's number, from block 0 (every block
// asking the host for the same number cost 1 us a block).  Numbers before `first` stay as they are on the device.
__global__ void step_in_kernel(const int* __restrict__ host, int* __restrict__ dev, int first, int n,
                               volatile int* seq, unsigned* done) {
    pdl_wait();
    pdl_trigger();
    int step = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0 && seq != nullptr) step = seq[0];          // under way together with the block's other reads
    const int quads = (n + 3) >> 2;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += gridDim.x * blockDim.x) {
        if (4 * i >= first && 4 * i + 4 <= n) {
            ((int4*)dev)[i] = __ldcv((const int4*)host + i);
        } else {
            for (int j = max(4 * i, first); j < min(4 * i + 4, n); ++j) dev[j] = __ldcv(host + j);
        }
    }
    if (seq == nullptr) return;
    __syncthreads();                                       // every number of this block has been read (and is on its way to dev)
    if (threadIdx.x == 0) {
        if (gridDim.x == 1) {
            seq[1] = step;
        } else {
            if (blockIdx.x == 0) *(volatile unsigned*)(done + 1) = (unsigned)step;
            __threadfence();
            if (atomicAdd(done, 1u) == gridDim.x - 1) {
                __threadfence();
                done[0] = 0u;
                seq[1] = (int)*(volatile unsigned*)(done + 1);
            }
        }
    }
}

__global__ void step_out_kernel(const int* __restrict__ dev, int* __restrict__ host, int n) {
    pdl_wait();
    pdl_trigger();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) host[i] = dev[i];
}

// The result of a step that a graph replays, to where the step's packed buffer says (0: nowhere): a tensor of its own per step,
// as a step launched one kernel at a time returns.  What bounds it: its launch as the graph's last node (a result of 5 x 500
// numbers), or its bytes.  A copy behind the graph instead: a step of 22 small kernels 130 us, 120 with this.
__global__ void step_result_kernel(const float* __restrict__ src, const unsigned long long* __restrict__ where, size_t n) {
    float* dst = reinterpret_cast<float*>(*where);                 // the step's description: in place before the step's first kernel
    pdl_wait();
    pdl_trigger();
    if (dst == nullptr) return;
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    if ((((uintptr_t)src | (uintptr_t)dst) & 15u) == 0) {
        for (size_t i = first; i < n >> 2; i += step) reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
        for (size_t i = (n & ~(size_t)3) + first; i < n; i += step) dst[i] = src[i];
    } else {
        for (size_t i = first; i < n; i += step) dst[i] = src[i];
    }
}

// What the GPU calls a page-locked host address.
static int device_address(void* host, void** dev) {
    *dev = nullptr;
    return host == nullptr ? 0 : (int)cudaHostGetDevicePointer(dev, host, 0);
}

// host, dev: 16-byte aligned; host and seq (null: no step numbers) page-locked host memory.
extern "C" int rg_step_in(void* host, int* dev, int first, int n, void* seq, unsigned* done, void* stream) {
    if (n <= 0) return 0;
    if (first < 0 || ((uintptr_t)host | (uintptr_t)dev) & 15u || (seq != nullptr && done == nullptr)) return RG_ERR_UNSUPPORTED;
    void *h, *s;
    int e = device_address(host, &h);
    if (e) return e;
    e = device_address(seq, &s);
    if (e) return e;
    // one 16-byte request a thread, all under way at once, up to 64 blocks (256 KB; 64 KB of the bus's 50 GB/s are 1.3 us); a
    // larger step is a few requests a thread one after another
    const int blocks = min(64, (n + 4 * STEP_IN_THREADS - 1) / (4 * STEP_IN_THREADS));
    return rg_launch(step_in_kernel, dim3(blocks), dim3(STEP_IN_THREADS), 0, (cudaStream_t)stream, 1, (const int*)h, dev, first, n,
                     (volatile int*)s, done);
}

extern "C" int rg_step_out(const int* dev, void* host, int n, void* stream) {
    if (n <= 0) return 0;
    void* h;
    const int e = device_address(host, &h);
    if (e) return e;
    return rg_launch(step_out_kernel, dim3(1), dim3(min(512, (n + 31) / 32 * 32)), 0, (cudaStream_t)stream, 1, dev, (int*)h, n);
}

// where: 8-byte aligned, on the device: the address of n floats, or 0.
extern "C" int rg_step_result(const float* src, const void* where, long long n, void* stream) {
    if (n <= 0) return 0;
    if ((uintptr_t)where & 7u) return RG_ERR_UNSUPPORTED;
    const long long blocks = (n + 1023) / 1024;
    return rg_launch(step_result_kernel, dim3((unsigned)(blocks < 592 ? blocks : 592)), dim3(256), 0, (cudaStream_t)stream, 1, src,
                     (const unsigned long long*)where, (size_t)n);
}
