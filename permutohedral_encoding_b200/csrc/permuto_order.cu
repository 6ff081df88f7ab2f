// Spatial order of a batch of points.
//
// The lattice kernels are bound by random accesses: every point touches D+1 table entries per level.
// Neighbouring points share most of them on every level whose cells are wider than the distance
// between points, but a batch of independent samples puts no neighbours into the same warp.  This
// file sorts the points along a space-filling curve first, so that the 32 points of a warp (and the
// 256 of a block) lie close together: gathers of a level then fall into few lines of L1, and the
// reductions of a warp merge before they reach L2.  Results do not depend on the order; every kernel
// writes its rows to the point's own index, which travels in the record.
//
// A counting sort over curve cells:
//   (counters cleared)
//   order_count_kernel     cell of every point, its arrival number inside the cell (atomic counter)
//   order_scan_kernel      exclusive sums over each group of kScanBins cells, plus the group's place
//   order_scatter_kernel   record {coordinates, index} to cell base + arrival number
// Only neighbouring cells have to stay together, so groups take their place in the order they arrive
// (one atomic on a cursor) and no sum over all cells is needed.  Batches above kChunk points are
// sorted chunk by chunk: the records of a chunk (64 MB) and the rows it touches stay within reach of
// L2 and of the address translation caches.
#include <cstdint>
#include <cuda_runtime.h>

#include "permuto_b200.h"
#include "permuto_internal.h"

namespace permuto {
namespace {

#ifndef PERMUTO_CHUNK_BITS
#define PERMUTO_CHUNK_BITS 22
#endif
#ifndef PERMUTO_CELL_POINTS_BITS
#define PERMUTO_CELL_POINTS_BITS 3
#endif
constexpr int kChunkBits = PERMUTO_CHUNK_BITS;
constexpr int kCellBits = PERMUTO_CELL_POINTS_BITS;  // about 2^kCellBits points per cell
constexpr int kScanBins = 1024;     // cells per block of the scan
constexpr int kThreads = 256;
constexpr int kPerThread = 4;       // points per thread, so that a batch of 2^20 is one wave of blocks
constexpr int kPerBlock = kThreads * kPerThread;
constexpr int kNibbles = 6;         // a cell coordinate has at most 24 bits

struct OrderArgs {
    const float* positions;
    int64_t stride_n, stride_d;
    uint32_t n;
    int bits;            // cells per chunk: 2^bits, at least kScanBins
    uint32_t* cursors;   // one per chunk: records handed out
    uint32_t* counters;  // 2^bits per chunk
    uint2* arrival;      // per point: cell, arrival number
    float4* records;
};

template <int D>
__device__ __forceinline__ void load(const OrderArgs& a, int64_t n, float (&pos)[D]) {
#pragma unroll
    for (int i = 0; i < D; ++i) pos[i] = __ldg(a.positions + n * a.stride_n + i * a.stride_d);
}

// sum over the block of M values per thread; every thread gets it
template <int M>
__device__ __forceinline__ void block_sum(float (&v)[M], float* scratch) {
    constexpr int kWarps = kThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < M; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if (lane == 0) scratch[warp * M + i] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < M; ++i) {
        v[i] = scratch[i];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) v[i] += scratch[w * M + i];
    }
    __syncthreads();
}

// Cell of a point: `bits` halvings of the batch's extent, each of the dimension whose cells are widest
// at that moment -- cells stay near cubes whatever the aspect of the batch, flat dimensions get none --
// and the coordinate bits interleaved in that sequence.  Every block derives the grid of its chunk
// from the same 256 points, with the same result.
template <int D>
__global__ void __launch_bounds__(kThreads) order_count_kernel(const OrderArgs a) {
    __shared__ float scratch[kThreads / 32 * (D + 1)];
    __shared__ float lo[D], inv_cell[D];
    __shared__ int halvings[D];
    __shared__ uint8_t key_bit[D][24];                // of a dimension's k-th halving
    __shared__ uint32_t spread[D][kNibbles][16];      // coordinate nibble -> its key bits
    const uint32_t first = blockIdx.x * (uint32_t)kPerBlock;
    const uint32_t chunk = first >> kChunkBits;
    const uint32_t chunk_begin = chunk << kChunkBits;
    const uint32_t chunk_n = min(a.n - chunk_begin, 1u << kChunkBits);

    float s[D];
    load<D>(a, (int64_t)chunk_begin + (int64_t)((uint64_t)threadIdx.x * chunk_n / kThreads), s);
    float x[kPerThread][D];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        const uint32_t n = first + k * kThreads + threadIdx.x;
        load<D>(a, min(n, a.n - 1u), x[k]);
    }
    {
        bool ok = true;  // what is not finite does not take part
#pragma unroll
        for (int i = 0; i < D; ++i) ok = ok && fabsf(s[i]) < 1e30f;
        float sum[D + 1], dev[D];
#pragma unroll
        for (int i = 0; i < D; ++i) sum[i] = ok ? s[i] : 0.f;
        sum[D] = ok ? 1.f : 0.f;
        block_sum<D + 1>(sum, scratch);
        const float inv = 1.f / fmaxf(sum[D], 1.f);
#pragma unroll
        for (int i = 0; i < D; ++i) dev[i] = ok ? fabsf(s[i] - sum[i] * inv) : 0.f;
        block_sum<D>(dev, scratch);
        if (threadIdx.x == 0) {
            float cell[D];
            int halved[D];
#pragma unroll
            for (int i = 0; i < D; ++i) {
                // 4.4 mean absolute deviations hold a uniform box with a margin; what lies outside
                // goes to the edge cells
                cell[i] = fmaxf(4.4f * dev[i] * inv, 1e-30f);
                lo[i] = sum[i] * inv - 0.5f * cell[i];
                halved[i] = 0;
            }
            for (int b = a.bits - 1; b >= 0; --b) {
                int best = 0;
                float widest = cell[0];
#pragma unroll
                for (int i = 1; i < D; ++i)
                    if (cell[i] > widest) {
                        widest = cell[i];
                        best = i;
                    }
#pragma unroll
                for (int i = 0; i < D; ++i)
                    if (i == best) {
                        cell[i] *= 0.5f;
                        key_bit[i][halved[i]++] = (uint8_t)b;
                    }
            }
#pragma unroll
            for (int i = 0; i < D; ++i) {
                halvings[i] = halved[i];
                inv_cell[i] = 1.f / cell[i];
            }
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < D * kNibbles * 16; e += kThreads) {
        const int dim = e / (kNibbles * 16), nibble = e / 16 % kNibbles, v = e % 16;
        uint32_t r = 0u;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int k = halvings[dim] - 1 - (4 * nibble + t);  // the top bit is halving 0
            if ((v >> t & 1) && k >= 0) r |= 1u << key_bit[dim][k];
        }
        spread[dim][nibble][v] = r;
    }
    __syncthreads();
    uint32_t key[kPerThread];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        key[k] = chunk << a.bits;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const int h = halvings[i];
            const float top = (float)((1 << h) - 1);
            const int c = (int)fminf(fmaxf((x[k][i] - lo[i]) * inv_cell[i], 0.f), top);  // NaN: cell 0
            for (int nibble = 0; 4 * nibble < h; ++nibble) key[k] |= spread[i][nibble][c >> (4 * nibble) & 15];
        }
    }
    uint32_t arrived[kPerThread];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        const uint32_t n = first + k * kThreads + threadIdx.x;
        if (n < a.n) arrived[k] = atomicAdd(a.counters + key[k], 1u);
    }
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        const uint32_t n = first + k * kThreads + threadIdx.x;
        if (n < a.n) a.arrival[n] = make_uint2(key[k], arrived[k]);
    }
}

__global__ void __launch_bounds__(256) order_scan_kernel(const OrderArgs a) {
    __shared__ uint32_t warp_sum[8];
    __shared__ uint32_t place;
    cudaGridDependencySynchronize();
    const uint32_t base = blockIdx.x * kScanBins + threadIdx.x * 4u;
    const uint4 v = *reinterpret_cast<const uint4*>(a.counters + base);
    const uint32_t mine = v.x + v.y + v.z + v.w;
    uint32_t run = mine;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += t;
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    uint32_t before = run - mine, total = 0u;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) before += warp_sum[w];
        total += warp_sum[w];
    }
    if (threadIdx.x == 0) {
        const uint32_t chunk = base >> a.bits;
        place = (chunk << kChunkBits) + atomicAdd(a.cursors + chunk, total);
    }
    __syncthreads();
    before += place;
    *reinterpret_cast<uint4*>(a.counters + base) = make_uint4(before, before + v.x, before + v.x + v.y, before + v.x + v.y + v.z);
}

template <int D>
__global__ void __launch_bounds__(kThreads) order_scatter_kernel(const OrderArgs a) {
    const uint32_t first = blockIdx.x * (uint32_t)kPerBlock + threadIdx.x;
    float x[kPerThread][D];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) load<D>(a, min(first + k * kThreads, a.n - 1u), x[k]);
    cudaGridDependencySynchronize();
    uint2 at[kPerThread];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) at[k] = a.arrival[min(first + k * kThreads, a.n - 1u)];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) at[k].y += a.counters[at[k].x];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        const uint32_t n = first + k * kThreads;
        if (n >= a.n) break;
        if (D <= 3) {
            a.records[at[k].y] = make_float4(x[k][0], x[k][1], D == 3 ? x[k][D - 1] : 0.f, __uint_as_float(n));
        } else {
            float r[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < D; ++i) r[i] = x[k][i];
            r[7] = __uint_as_float(n);
            asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(a.records + 2 * (size_t)at[k].y),
                         "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7])
                         : "memory");
        }
    }
}

int order_bits(uint32_t n) {
    int bits = 10;  // kScanBins
    while (bits < kChunkBits - kCellBits && ((uint64_t)(1 << kCellBits) << bits) < n) ++bits;
    return bits;
}
uint32_t order_chunks(uint32_t n) { return ((n - 1u) >> kChunkBits) + 1u; }

size_t align256(size_t x) { return (x + 255) / 256 * 256; }
size_t record_bytes(int pos_dim) { return pos_dim <= 3 ? 16 : 32; }
size_t cursor_bytes(uint32_t n) { return align256(sizeof(uint32_t) * order_chunks(n)); }
size_t counter_bytes(uint32_t n) { return (sizeof(uint32_t) * order_chunks(n)) << order_bits(n); }

// launched while the kernel before it drains; the kernel waits for it itself
template <class K>
cudaError_t launch_early(K kernel, unsigned blocks, unsigned threads, const OrderArgs& a, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int D>
cudaError_t launch(const OrderArgs& a, cudaStream_t st) {
    const unsigned points = (a.n + kPerBlock - 1) / kPerBlock;
    cudaError_t e = cudaMemsetAsync(a.cursors, 0, cursor_bytes(a.n) + counter_bytes(a.n), st);
    if (e != cudaSuccess) return e;
    order_count_kernel<D><<<points, kThreads, 0, st>>>(a);
    e = launch_early(order_scan_kernel, (order_chunks(a.n) << a.bits) / kScanBins, 256, a, st);
    if (e != cudaSuccess) return e;
    e = launch_early(order_scatter_kernel<D>, points, kThreads, a, st);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace
}  // namespace permuto

extern "C" {

int64_t permuto_order_bytes(int32_t pos_dim, int64_t nr_positions) {
    using namespace permuto;
    if (pos_dim < 2 || pos_dim > 7 || nr_positions < 1 || nr_positions > (int64_t)0x7fffffff) return 0;
    const uint32_t n = (uint32_t)nr_positions;
    return (int64_t)(align256(n * record_bytes(pos_dim)) + align256(n * sizeof(uint2)) + cursor_bytes(n) + counter_bytes(n));
}

int permuto_order_pays(const permuto_config* cfg, int64_t nr_positions, int32_t with_gradients) {
    (void)with_gradients;
    return cfg && nr_positions >= (1 << 18) ? 1 : 0;
}

int permuto_order_points(const permuto_config* cfg, const permuto_inputs* in, void* order, int64_t order_bytes, void* stream) {
    using namespace permuto;
    if (!cfg || !in || !in->positions || !order)
        return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "cfg, in, positions and order must not be NULL");
    const int64_t need = permuto_order_bytes(cfg->pos_dim, in->nr_positions);
    if (need == 0) return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: pos_dim must be 2..7 and nr_positions in 1..2^31-1");
    if (order_bytes < need || (reinterpret_cast<uintptr_t>(order) & 255u) != 0)
        return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: needs %lld bytes on a 256-byte boundary", (long long)need);
    OrderArgs a;
    a.positions = in->positions;
    a.stride_n = in->pos_stride_n;
    a.stride_d = in->pos_stride_d;
    a.n = (uint32_t)in->nr_positions;
    a.bits = order_bits(a.n);
    char* at = static_cast<char*>(order);
    a.records = reinterpret_cast<float4*>(at);
    at += align256(a.n * record_bytes(cfg->pos_dim));
    a.arrival = reinterpret_cast<uint2*>(at);
    at += align256(a.n * sizeof(uint2));
    a.cursors = reinterpret_cast<uint32_t*>(at);
    at += cursor_bytes(a.n);
    a.counters = reinterpret_cast<uint32_t*>(at);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    switch (cfg->pos_dim) {
        case 2: e = launch<2>(a, st); break;
        case 3: e = launch<3>(a, st); break;
        case 4: e = launch<4>(a, st); break;
        case 5: e = launch<5>(a, st); break;
        case 6: e = launch<6>(a, st); break;
        default: e = launch<7>(a, st); break;
    }
    return e == cudaSuccess ? PERMUTO_OK : set_error(PERMUTO_ERR_CUDA, "permuto_order_points launch: %s", cudaGetErrorString(e));
}

}  // extern "C"
