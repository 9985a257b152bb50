// Grid-wide sums and barriers inside one cooperative launch, shared by the one-launch solvers.
#pragma once

#include "pm_common.cuh"

namespace pm
{

constexpr int kGridMaxThreads = 1024;
constexpr int kGridMaxCtas = 160;            // most CTAs of a launch that waits for itself
constexpr unsigned kBarrierPolls = 1u << 25; // a barrier gives up after this many polls (some 20 s)

struct alignas(16) Packet
{
    double value;
    unsigned long long epoch;
};

// Grid barriers carry the dots.  Every CTA stores its partial sums, each with the barrier's number
// as one 16-byte packet, into a mailbox of every other CTA and polls its own, so a sum costs one
// trip through L2 and no line is polled by two CTAs (148 CTAs polling one shared set of packets
// slowed the stores down: 4 us a barrier against 1.5).  Packets alternate between two sets: a CTA
// reaches barrier e + 2 only after every CTA has read the packets of e.
__device__ __forceinline__ void packet_store(Packet* at, double value, unsigned long long epoch)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(at),
                 "l"(__double_as_longlong(value)), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ void packet_load(const Packet* at, double& value, unsigned long long& epoch)
{
    unsigned long long bits;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(bits), "=l"(epoch)
                 : "l"(at)
                 : "memory");
    value = __longlong_as_double(static_cast<long long>(bits));
}

struct GridShared // of one CTA
{
    double local[2][kGridMaxThreads / 32]; // the warps' sums
    double grid[2][(kGridMaxCtas + 31) / 32];
    int failed;
};

struct GridSync
{
    Packet* mail; // [2][CTA][CTA][2], epochs below this launch's before it
    int* timed_out; // device flag: a barrier gave up
    GridShared* sh;
    unsigned long long epoch;
};

// Grid sums of K per-thread values, the same bits in every CTA; false when a CTA gave up waiting.
// publish: writes before it are visible after it to plain (coherent) loads of every CTA.
template <int K>
__device__ __forceinline__ bool grid_sum(GridSync& g, double (&mine)[K], double (&total)[K], bool publish)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const unsigned ctas = gridDim.x;
    g.epoch += 1;
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const double s = warp_sum(mine[k]);
        if (lane == 0)
            g.sh->local[k][warp] = s;
    }
    __syncthreads();
    if (ctas == 1) // the CTA's own barriers order everything
    {
#pragma unroll
        for (int k = 0; k < K; ++k)
            total[k] = warp_sum(lane < warps ? g.sh->local[k][lane] : 0.0);
        __syncthreads();
        return true;
    }
    const unsigned peer = threadIdx.x;
    if (warp * 32 < ctas) // one thread per peer
    {
        double s[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
            s[k] = warp_sum(lane < warps ? g.sh->local[k][lane] : 0.0);
        if (publish)
            __threadfence();
        double from[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
            from[k] = 0.0;
        if (peer < ctas)
        {
            Packet* const set = g.mail + size_t(g.epoch & 1) * 2 * ctas * ctas;
            Packet* const out = set + (size_t(peer) * ctas + blockIdx.x) * 2;
            const Packet* const in = set + (size_t(blockIdx.x) * ctas + peer) * 2;
#pragma unroll
            for (int k = 0; k < K; ++k)
                packet_store(out + k, s[k], g.epoch);
            unsigned polls = 0;
#pragma unroll
            for (int k = 0; k < K; ++k)
            {
                unsigned long long seen;
                do
                    packet_load(in + k, from[k], seen);
                while (seen != g.epoch && ++polls < kBarrierPolls);
            }
            if (polls >= kBarrierPolls)
            {
                atomicExch(g.timed_out, 1);
                g.sh->failed = 1;
            }
        }
        if (publish)
            __threadfence();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            const double sum = warp_sum(from[k]);
            if (lane == 0)
                g.sh->grid[k][warp] = sum;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        double sum = 0.0;
        for (unsigned w = 0; w * 32 < ctas; ++w)
            sum += g.sh->grid[k][w];
        total[k] = sum;
    }
    return g.sh->failed == 0;
}

__device__ __forceinline__ bool grid_barrier(GridSync& g)
{
    double none[1] = {0.0}, total[1];
    return grid_sum<1>(g, none, total, true);
}

// The mailboxes of one workspace and the number below which all its barriers lie so far, zeroed once.  Every
// launch takes numbers of its own.  One that may be captured takes them on the device, through grid_next_launch
// in a kernel queued before it: it is replayed with the same arguments, and packets of the replay before must not
// pass for its own.  A workspace whose solves wait on the host, and so are never captured, takes next_launch().
constexpr size_t kGridPackets = 4 * size_t(kGridMaxCtas) * kGridMaxCtas;
constexpr unsigned long long kGridEpochs = 1ull << 34; // more than the barriers of any solve (three per iteration)

// an atomic without a result, which the kernel does not wait for
__device__ __forceinline__ void grid_next_launch(unsigned long long* epoch) { atomicAdd(epoch, kGridEpochs); }

struct GridMail
{
    DeviceBuffer buffer;
    Packet* packets() const { return static_cast<Packet*>(buffer.ptr); }
    unsigned long long* epoch() const { return reinterpret_cast<unsigned long long*>(packets() + kGridPackets); }
    unsigned long long launches = 0;
    unsigned long long next_launch() { return ++launches * kGridEpochs; }
    void open(cudaStream_t stream, const char* owner)
    {
        buffer.bind(stream, owner);
        if (!buffer.ptr)
        {
            const size_t bytes = (kGridPackets + 1) * sizeof(Packet);
            buffer.ensure(bytes, stream, owner);
            PM_CUDA(cudaMemsetAsync(buffer.ptr, 0, bytes, stream));
        }
    }
};

// More than the default 48 KB of shared memory, static arrays included.  The limit is the function's, not the
// launch's: `most` is the same in every call for a kernel, so that no thread lowers another's.
inline void allow_smem(const void* kernel, size_t most)
{
    if (most > 40 * 1024)
        PM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)));
}

// A launch whose CTAs wait for one another; false where the device will not hold all of them at once (a
// context with fewer SMs than the device has): the caller then takes its kernels one by one.
inline bool launch_resident(const void* kernel, unsigned ctas, unsigned threads, void** args, size_t smem,
                            cudaStream_t stream)
{
    const cudaError_t launched = cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(threads), args, smem, stream);
    if (launched == cudaErrorCooperativeLaunchTooLarge)
    {
        cudaGetLastError(); // not the next launch's error
        return false;
    }
    check_cuda(launched, "cooperative launch");
    PM_LAUNCH_CHECK();
    return true;
}

} // namespace pm
