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
//   order_clear_kernel     zero counters
//   order_count_kernel     cell of every point, its arrival number inside the cell (atomic counter)
//   order_scan_kernel      exclusive sums over each group of kScanBins cells, plus the group's place
//   order_scatter_kernel   record {coordinates, index} to cell base + arrival number
// Only neighbouring cells have to stay together, so groups take their place in the order they arrive
// (one atomic on a cursor) and no sum over all cells is needed.  Large batches are sorted chunk by
// chunk, so that the records and counters of a chunk (32 and 4 MB) stay in L2.
//
// What bounds it: the counters' returning atomics (about 92 G/s) and the scattered 16-byte records; 32 us
// for 2^20 points (34 with a separate clear and a serial grid), 520-540 us for 2^24, where reading and writing its data once would take 5 and 75 us.
// Tried: counting with reductions and taking the places in the scatter kernel (34 -> 38 us, 2^24 points
// 520 -> 432), counters 16 or 32 bytes apart (no change).
#include <cstdint>
#include <cuda_runtime.h>

#include "permuto_b200.h"
#include "permuto_internal.h"

namespace permuto {
namespace {

constexpr int kChunkBits = 21;      // points per chunk; 2^20 / 2^22 / 2^23 / 2^24 points: order 461 / 568 / 675 / 772 us
                                    // against 520, but the forward after it 3160 / 3085 / 3064 / 3018 against 3080
constexpr int kCellBits = 1;        // about two points per cell: more share counters, whose atomics then collide
                                    // (8 / 32 / 128 / 512 points per cell, 2^20 points: 34 / 37 / 39 / 72 us).  1 / 2 / 4
                                    // / 8 points out of a cold L2: order 43 / 42 / 42 / 42, table gradient after it 304 /
                                    // 305 / 305 / 309; 2^24 points, order 552 / 534 / 527 / 523
constexpr int kScanBins = 1024;     // cells per block of the scan
constexpr int kThreads = 256;
constexpr int kPerThread = 4;       // consecutive points of a thread: whole 16-byte vectors of any row length
constexpr int kPerBlock = kThreads * kPerThread;
constexpr int kNibbles = 6;         // a cell coordinate has at most 24 bits

struct OrderArgs {
    const float* positions;
    int64_t stride_n, stride_d;
    uint32_t n;
    int bits;            // cells per chunk: 2^bits, at least kScanBins
    int rounds;          // tiles of kPerBlock points per block
    int vec_ok;          // contiguous rows on a 16-byte boundary
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

// the kPerThread points from n on; where the batch ends, its last point again
template <int D>
__device__ __forceinline__ void load_points(const OrderArgs& a, uint32_t n, float (&x)[kPerThread][D]) {
    if (a.vec_ok && n + kPerThread <= a.n) {
        const float4* src = reinterpret_cast<const float4*>(a.positions) + (size_t)n / kPerThread * D;
        float v[kPerThread * D];
#pragma unroll
        for (int q = 0; q < D; ++q) {
            const float4 f = __ldg(src + q);
            v[4 * q] = f.x;
            v[4 * q + 1] = f.y;
            v[4 * q + 2] = f.z;
            v[4 * q + 3] = f.w;
        }
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
#pragma unroll
            for (int i = 0; i < D; ++i) x[k][i] = v[k * D + i];
        }
    } else {
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) load<D>(a, min(n + k, a.n - 1u), x[k]);
    }
}

__device__ __forceinline__ float warp_sum_all(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// clears the counters and cursors while the blocks of the count kernel already work out their grid
__global__ void __launch_bounds__(256) order_clear_kernel(uint4* words, uint32_t n) {
    cudaTriggerProgrammaticLaunchCompletion();
    for (uint32_t i = blockIdx.x * 1024u + threadIdx.x, end = min(n, blockIdx.x * 1024u + 1024u); i < end; i += 256u)
        words[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Cell of a point: `bits` halvings of the batch's extent, each of the dimension whose cells are widest
// at that moment -- cells stay near cubes whatever the aspect of the batch, flat dimensions get none --
// and the coordinate bits interleaved in that sequence.  Every block derives the grid of its chunk
// from the same 256 points, with the same result.
template <int D>
__global__ void __launch_bounds__(kThreads) order_count_kernel(const OrderArgs a) {
    constexpr int kWarps = kThreads / 32;
    __shared__ float part[2 * D][kWarps];
    __shared__ float lo[D], width[D], inv_cell[D];
    __shared__ int halvings[D];
    __shared__ uint8_t key_bit[D][24];                // of a dimension's k-th halving
    __shared__ uint32_t spread[D][kNibbles][16];      // coordinate nibble -> its key bits
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t first = blockIdx.x * (uint32_t)a.rounds * kPerBlock;
    const uint32_t chunk = first >> kChunkBits;
    const uint32_t chunk_begin = chunk << kChunkBits;
    const uint32_t chunk_n = min(a.n - chunk_begin, 1u << kChunkBits);

    float s[D];
    load<D>(a, (int64_t)chunk_begin + (int64_t)((uint64_t)t * chunk_n / kThreads), s);
    float x[kPerThread][D];
    load_points<D>(a, first + t * kPerThread, x);
    {
        bool ok = true;  // what is not finite does not take part
#pragma unroll
        for (int i = 0; i < D; ++i) ok = ok && fabsf(s[i]) < 1e30f;
        const float inv = 1.f / fmaxf((float)__popc(__ballot_sync(0xffffffffu, ok)), 1.f);
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const float mean = warp_sum_all(ok ? s[i] : 0.f) * inv;
            const float dev = warp_sum_all(ok ? fabsf(s[i] - mean) : 0.f) * inv;
            if (lane == 0) {
                part[i][warp] = mean;
                part[D + i][warp] = dev;
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
        // mean, and mean absolute deviation (inside a warp's samples plus of its mean), over the warps
        float mean[D], dev[D];
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const float m = lane < kWarps ? part[i][lane] : 0.f, d = lane < kWarps ? part[D + i][lane] : 0.f;
            mean[i] = warp_sum_all(m) * (1.f / kWarps);
            dev[i] = warp_sum_all(lane < kWarps ? d + fabsf(m - mean[i]) : 0.f) * (1.f / kWarps);
        }
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < D; ++i) {
                // 4.4 mean absolute deviations hold a uniform box with a margin; what lies outside
                // goes to the edge cells
                width[i] = fmaxf(4.4f * dev[i], 1e-30f);
                lo[i] = mean[i] - 0.5f * width[i];
                halvings[i] = 0;
            }
        }
    }
    __syncthreads();
    // Halving k of dimension i splits cells of width[i] / 2^k.  Its place in the sequence is the number of
    // halvings of wider cells, counted from the widths' exponents and mantissas (all places at once: taking
    // the widest dimension `bits` times in one thread was a microsecond of every block).
    if (t < D * 24) {
        const int i = t / 24, k = t % 24, mine = __float_as_int(width[i]);
        int place = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            const int other = __float_as_int(width[j]);
            const int a0 = other & 0x7fffff, b0 = mine & 0x7fffff;
            place += max(0, (other >> 23) - (mine >> 23) + k + ((a0 > b0 || (a0 == b0 && j < i)) ? 1 : 0));
        }
        if (place < a.bits) {
            key_bit[i][k] = (uint8_t)(a.bits - 1 - place);
            atomicMax(&halvings[i], k + 1);
        }
    }
    __syncthreads();
    if (t < D) inv_cell[t] = ldexpf(1.f / width[t], halvings[t]);
    for (int e = t; e < D * kNibbles * 16; e += kThreads) {
        const int dim = e / (kNibbles * 16), nibble = e / 16 % kNibbles, v = e % 16;
        uint32_t r = 0u;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int k = halvings[dim] - 1 - (4 * nibble + b);  // the top bit is halving 0
            if ((v >> b & 1) && k >= 0) r |= 1u << key_bit[dim][k];
        }
        spread[dim][nibble][v] = r;
    }
    __syncthreads();
    cudaGridDependencySynchronize();  // the counters are cleared
#pragma unroll 1
    for (int round = 0; round < a.rounds; ++round) {
        const uint32_t n = first + round * (uint32_t)kPerBlock + t * kPerThread;
        if (n >= a.n) return;
        if (round > 0) load_points<D>(a, n, x);
        uint32_t key[kPerThread], arrived[kPerThread];
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) key[k] = chunk << a.bits;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const int h = halvings[i];
            const float top = (float)((1 << h) - 1), l = lo[i], ic = inv_cell[i];
            int c[kPerThread];
#pragma unroll
            for (int k = 0; k < kPerThread; ++k) c[k] = (int)fminf(fmaxf((x[k][i] - l) * ic, 0.f), top);  // NaN: cell 0
            for (int nibble = 0; 4 * nibble < h; ++nibble) {
#pragma unroll
                for (int k = 0; k < kPerThread; ++k) key[k] |= spread[i][nibble][c[k] >> (4 * nibble) & 15];
            }
        }
#pragma unroll
        for (int k = 0; k < kPerThread; ++k)
            if (n + k < a.n) arrived[k] = atomicAdd(a.counters + key[k], 1u);
        if (n + kPerThread <= a.n) {
            uint4* dst = reinterpret_cast<uint4*>(a.arrival + n);
            dst[0] = make_uint4(key[0], arrived[0], key[1], arrived[1]);
            dst[1] = make_uint4(key[2], arrived[2], key[3], arrived[3]);
        } else {
#pragma unroll
            for (int k = 0; k < kPerThread; ++k)
                if (n + k < a.n) a.arrival[n + k] = make_uint2(key[k], arrived[k]);
        }
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
    const uint32_t n = (blockIdx.x * (uint32_t)kThreads + threadIdx.x) * kPerThread;
    if (n >= a.n) return;
    float x[kPerThread][D];
    load_points<D>(a, n, x);
    cudaGridDependencySynchronize();
    uint2 at[kPerThread];
    if (n + kPerThread <= a.n) {
        const uint4* src = reinterpret_cast<const uint4*>(a.arrival + n);
        const uint4 u = src[0], v = src[1];
        at[0] = make_uint2(u.x, u.y);
        at[1] = make_uint2(u.z, u.w);
        at[2] = make_uint2(v.x, v.y);
        at[3] = make_uint2(v.z, v.w);
    } else {
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) at[k] = a.arrival[min(n + k, a.n - 1u)];
    }
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) at[k].y += a.counters[at[k].x];
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        if (n + k >= a.n) break;
        if (D <= 3) {
            a.records[at[k].y] = make_float4(x[k][0], x[k][1], D == 3 ? x[k][D - 1] : 0.f, __uint_as_float(n + k));
        } else {
            float r[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < D; ++i) r[i] = x[k][i];
            r[7] = __uint_as_float(n + k);
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
bool order_sizes_ok(int32_t pos_dim, int64_t n) { return pos_dim >= 2 && pos_dim <= 7 && n >= 1 && n <= (int64_t)0x7fffffff; }

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
    const unsigned counting = (points + a.rounds - 1) / a.rounds;
    const uint32_t words = (uint32_t)((cursor_bytes(a.n) + counter_bytes(a.n)) / sizeof(uint4));
    order_clear_kernel<<<(words + 1023u) / 1024u, 256, 0, st>>>(reinterpret_cast<uint4*>(a.cursors), words);
    cudaError_t e = launch_early(order_count_kernel<D>, counting, kThreads, a, st);
    if (e != cudaSuccess) return e;
    e = launch_early(order_scan_kernel, (order_chunks(a.n) << a.bits) / kScanBins, 256, a, st);
    if (e != cudaSuccess) return e;
    e = launch_early(order_scatter_kernel<D>, points, kThreads, a, st);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace
}  // namespace permuto

extern "C" {

int64_t permuto_order_record_bytes(int32_t pos_dim, int64_t nr_positions) {
    using namespace permuto;
    if (!order_sizes_ok(pos_dim, nr_positions)) return 0;
    return nr_positions * (int64_t)record_bytes(pos_dim) + pos_dim;
}

int64_t permuto_order_scratch_bytes(int32_t pos_dim, int64_t nr_positions) {
    using namespace permuto;
    if (!order_sizes_ok(pos_dim, nr_positions)) return 0;
    const uint32_t n = (uint32_t)nr_positions;
    return (int64_t)(align256(n * sizeof(uint2)) + cursor_bytes(n) + counter_bytes(n));
}

int64_t permuto_order_bytes(int32_t pos_dim, int64_t nr_positions) {
    using namespace permuto;
    if (!order_sizes_ok(pos_dim, nr_positions)) return 0;
    return (int64_t)align256((size_t)nr_positions * record_bytes(pos_dim)) + permuto_order_scratch_bytes(pos_dim, nr_positions);
}

// Where the order's own time comes back: the number of levels from which on it is used, by what follows it.  A
// line lies where neither independent points nor ray samples (half in order already) get slower than on the
// kernels of the build that knew no order ("before").  us without -> with the order, itself included:
//  features only, F = 2: 2^19 points 24 levels 156 -> 141 (pos_dim 2: 115 -> 98), rays 121 -> 135 (before 147), 16
//    levels 115 -> 106, but rays 90 -> 100 (before 97); 2^20: 24 levels 293 -> 250, rays 228 -> 240 (before 282), 16
//    levels 211 -> 186, rays 161 -> 180 (before 172), 12 levels 148 -> 150; pos_dim 6, 16 levels 369 -> 371.
//    F = 4, 2^20 points 174 -> 178.
//  table gradient (without -> with, walked in strands), F = 2: 2^17: 16 levels 104 -> 86, rays 87 -> 82, pos_dim 4 118 -> 104, 6
//    155 -> 144; 12 levels 73 -> 72, rays 64 -> 70 (3 * 2^16: 16 levels 131 -> 108, rays 111 -> 102, pos_dim 7 232 -> 226).  2^18: 12
//    levels 122 -> 100, rays 95 -> 97, 8 levels 77 -> 68, rays 67 -> 69; pos_dim 4, 8 / 4 levels 97 -> 85 / 61 -> 64, pos_dim 6 125 -> 115 /
//    79 -> 83.  2^19: 8 levels 126 -> 102, rays 112 -> 102; 4 levels 85 -> 75, rays 65 -> 74, pos_dim 6 120 -> 138.  2^20: 4 levels 140 -> 122, rays
//    120 -> 122, pos_dim 6 212 -> 232.
//    F = 4: 2^18: 8 levels 94 -> 77, rays 82 -> 76, 4 levels 58 -> 59, rays 50 -> 59; pos_dim 4 / 6, 8 levels 110 -> 94 / 140 -> 137 (pos_dim 5,
//    12 levels 186 -> 186).  2^19: pos_dim 6, 8 levels 246 -> 226, 4 levels 139 -> 162.  F = 8: 2^18: 6 levels 118 -> 90, rays 95 -> 88, pos_dim
//    4 / 6 148 -> 119 / 187 -> 194, 4 levels rays 75 -> 76.  2^19: 4 levels 159 -> 113, rays 121 -> 104, pos_dim 6 247 -> 229, 6 levels 305 -> 325.  2^20: pos_dim
//    6, 4 / 6 levels 407 -> 416 / 574 -> 485.
//  position gradient, alone or with the table's, F = 2: 2^18: both, 16 levels 198 -> 194, 12 levels 148 -> 152; pos_dim 4,
//    24 levels 345 -> 356.  2^19: 12 levels 265 -> 248, rays 210 -> 236 (before 263), 8 levels 146 -> 156; pos_dim 6, 12 /
//    16 levels 462 -> 492 / 620 -> 631 (2^20: 1185 -> 1167).  F = 4: 2^19: 16 levels 414 -> 408, rays 359 -> 397 (before 402);
//    pos_dim 4 503 -> 510, 2^20 949 -> 932; pos_dim 6 1330 -> 1366.  F = 8: 8 levels 341 -> 276, pos_dim 6 534 -> 533, 4
//    levels rays 138 -> 164 (before 150).
int permuto_order_pays(const permuto_config* cfg, int64_t nr_positions, int32_t purpose) {
    if (!cfg || nr_positions > (int64_t)0x7fffffff) return 0;
    const int F = cfg->nr_feat_per_level, d = cfg->pos_dim;
    const bool n18 = nr_positions >= 1 << 18, n19 = nr_positions >= 1 << 19, n20 = nr_positions >= 1 << 20;
    int levels = 0;  // never
    if (purpose == PERMUTO_ORDER_FEATURES) {
        if (F == 2 && (d <= 5 ? n19 : n20)) levels = 18;
    } else if (purpose == PERMUTO_ORDER_TABLE_GRAD) {
        if (F == 2) levels = n20 ? (d <= 3 ? 4 : 8) : (n19 ? 8 : (n18 ? (d <= 3 ? 10 : 8) : (nr_positions >= 3 << 16 ? 16 : 0)));
        if (F == 4) levels = n19 || (n18 && d <= 5) ? 8 : 0;
        if (F == 8) levels = n19 ? (d <= 5 ? 4 : (n20 ? 6 : 8)) : (n18 && d <= 4 ? 6 : 0);
    } else {
        if (F == 2 && n18) levels = n19 ? (d <= 5 ? 12 : 16) : (d <= 3 ? 16 : 0);
        if (F == 4 && n19) levels = d <= 3 || (d <= 5 && n20) ? 12 : 0;
        if (F == 8 && n19) levels = 8;
    }
    return levels > 0 && cfg->nr_levels >= levels ? 1 : 0;
}

int permuto_order_points(const permuto_config* cfg, const permuto_inputs* in, void* order, int64_t order_bytes, void* stream) {
    using namespace permuto;
    if (!cfg || !in || !order) return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "cfg, in, positions and order must not be NULL");
    const int64_t need = permuto_order_bytes(cfg->pos_dim, in->nr_positions);
    if (need == 0) return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: pos_dim must be 2..7 and nr_positions in 1..2^31-1");
    if (order_bytes < need) return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: needs %lld bytes on a 256-byte boundary", (long long)need);
    void* scratch = static_cast<char*>(order) + align256((size_t)in->nr_positions * record_bytes(cfg->pos_dim));
    return permuto_order_records(cfg, in, order, scratch, stream);
}

int permuto_order_records(const permuto_config* cfg, const permuto_inputs* in, void* records, void* scratch, void* stream) {
    using namespace permuto;
    if (!cfg || !in || !in->positions || !records || !scratch)
        return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "cfg, in, positions and order must not be NULL");
    if (!order_sizes_ok(cfg->pos_dim, in->nr_positions))
        return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: pos_dim must be 2..7 and nr_positions in 1..2^31-1");
    if (((reinterpret_cast<uintptr_t>(records) | reinterpret_cast<uintptr_t>(scratch)) & 255u) != 0)
        return set_error(PERMUTO_ERR_INVALID_ARGUMENT, "order: records and scratch need a 256-byte boundary");
    OrderArgs a;
    a.positions = in->positions;
    a.stride_n = in->pos_stride_n;
    a.stride_d = in->pos_stride_d;
    a.n = (uint32_t)in->nr_positions;
    a.bits = order_bits(a.n);
    // a block's grid of cells serves several tiles once there are more tiles than resident blocks
    a.rounds = 1;
    while (a.rounds < 8 && a.n / kPerBlock / (2 * a.rounds) >= 1024) a.rounds *= 2;
    a.vec_ok = in->pos_stride_d == 1 && in->pos_stride_n == cfg->pos_dim && (reinterpret_cast<uintptr_t>(in->positions) & 15u) == 0;
    a.records = static_cast<float4*>(records);
    char* at = static_cast<char*>(scratch);
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
