// Lattice kernels for one pos_dim (compile with -DPERMUTO_DIM=2..7), sm_100a.
//
// Work decomposition shared by all kernels: one thread owns one point and walks levels in steps
// of LPS levels.  blockIdx.x walks point tiles, blockIdx.y walks passes of `levels_per_pass`
// levels, and blocks are dispatched x-fastest, so the whole grid sweeps the points once per
// pass: the slices of the value table (and of its gradient) that are live at any time are those
// of one pass, which stay L2-resident.  A step covers LPS = 8 / F levels of F features each,
// i.e. 8 consecutive floats of a feature row = one 32-byte sector, moved with a single 256-bit
// access (ld/st.global.v8.f32, new on sm_100), directly in the final [N, F*L] layout -- no
// transposed intermediate.  F = 2 is the reference's only supported width; F = 4 and 8 (which
// the reference lists as not yet implemented, Encoding.cuh:140-143) make every table access a
// 16- or 32-byte one, i.e. half or all of the sector the memory system moves anyway (measured on
// B200 over an L2-resident region: 16-byte random gathers run at three quarters of the rate of
// 8-byte ones, 16-byte vector reductions at the same rate as 8-byte ones; a 32-byte access is two
// 16-byte ones).
//
// What each kernel replaces in the reference (paths relative to its root):
//   forward_kernel          kernels/permutohedral_encoding/EncodingGPU.cuh:68-256
//   backward_kernel         EncodingGPU.cuh:259-414 (table) and :530-769 (positions), fused
//   double_backward_kernel  EncodingGPU.cuh:1016-1257 and :1260-1493, fused
#include <cuda_fp16.h>

#include "permuto_geometry.cuh"
#include "permuto_internal.h"

#ifndef PERMUTO_DIM
#error "compile with -DPERMUTO_DIM=<2..7>"
#endif

namespace permuto {
namespace {

constexpr int D = PERMUTO_DIM;
#ifndef PERMUTO_THREADS
#define PERMUTO_THREADS 256
#endif
// Resident blocks per SM the register allocator must leave room for.  Measured on B200: the
// gather+scatter kernels ran at 64-71 registers (36-46 % of the warps an SM can hold) and gain a
// few per cent when capped at 64; the gather-only position-gradient kernel gains 10 % at 51.
#ifndef PERMUTO_MIN_BLOCKS
#define PERMUTO_MIN_BLOCKS 4
#endif
#ifndef PERMUTO_MIN_BLOCKS_GATHER_ONLY
#define PERMUTO_MIN_BLOCKS_GATHER_ONLY (PERMUTO_DIM <= 4 ? 5 : 4)  // 5 spills and loses from pos_dim 5 up
#endif
// The forward kernel is bound by the LSU pipe, not by instruction-level parallelism: at 60
// registers (what a cap of 64 invites) it runs 4 % slower than at 32 with twice the resident warps.
#ifndef PERMUTO_MIN_BLOCKS_FORWARD
#define PERMUTO_MIN_BLOCKS_FORWARD (PERMUTO_DIM <= 3 ? 8 : (PERMUTO_DIM <= 5 ? 6 : 4))
#endif
constexpr int kThreads = PERMUTO_THREADS;
// wider table entries keep more addends live per vertex: leave them more registers
constexpr int min_blocks(int feats, bool gather_only) {
    return feats == 8 ? 2
                      : (feats == 4 || D >= 6) ? 3
                                               : (gather_only ? PERMUTO_MIN_BLOCKS_GATHER_ONLY : PERMUTO_MIN_BLOCKS);
}
constexpr unsigned kFullMask = 0xffffffffu;

// A point's coordinates.  Rows of 2 or 4 contiguous floats on an aligned base are one 8- or
// 16-byte load (consecutive threads then read consecutive vectors); every other case -- odd
// pos_dim, strided or transposed positions -- takes one 4-byte load per coordinate, which for
// contiguous rows still touches each 128-byte line from a single warp instruction group.
__device__ __forceinline__ void load_pos(const Problem& p, int64_t n, float (&pos)[D]) {
    if ((D == 2 || D == 4) && p.pos_vec_ok) {
        if (D == 2) {
            const float2 t = __ldg(reinterpret_cast<const float2*>(p.positions) + n);
            pos[0] = t.x;
            pos[D - 1] = t.y;
        } else {
            const float4 t = __ldg(reinterpret_cast<const float4*>(p.positions) + n);
            pos[0] = t.x;
            pos[1 % D] = t.y;
            pos[2 % D] = t.z;
            pos[3 % D] = t.w;
        }
        return;
    }
    const float* src = p.positions + n * p.pos_stride_n;
#pragma unroll
    for (int i = 0; i < D; ++i) pos[i] = __ldg(src + i * p.pos_stride_d);
}

// Hash modulo the capacity (EncodingGPU.cuh:34-36): a mask when it is a power of two, else the remainder
// from the quotient estimate h * floor(2^32 / capacity) / 2^32, which is at most one too small.
__device__ __forceinline__ uint32_t to_slot(const Problem& p, uint32_t h) {
    if (p.cap_is_pow2) return h & (p.capacity - 1u);
    const uint32_t r = h - __umulhi(h, p.cap_magic) * p.capacity;
    return min(r, r - p.capacity);  // r - capacity wraps around to a larger number when r is the remainder
}
__device__ __forceinline__ void to_slots(const Problem& p, const Simplex<D>& s, uint32_t (&slot)[D + 1]) {
    uint32_t h[D + 1];
    vertex_hashes<D>(s, h);
#pragma unroll
    for (int q = 0; q <= D; ++q) slot[q] = to_slot(p, h[q]);
}

// Vertices of the walk (q = 0..D) renumbered by the reference's remainder r = q - s modulo D+1, under
// which a lattice point keeps its number in every simplex it belongs to.
template <class T>
__device__ __forceinline__ void to_remainders(int s, T (&v)[D + 1]) {
    constexpr bool kPow2 = ((D + 1) & D) == 0;
    const int by = kPow2 ? (s & D) : (s < 0 ? s + D + 1 : s);
#pragma unroll
    for (int bit = 1; bit <= D; bit <<= 1) {
        T t[D + 1];
#pragma unroll
        for (int r = 0; r <= D; ++r) t[r] = (by & bit) ? v[(r + bit) % (D + 1)] : v[r];
#pragma unroll
        for (int r = 0; r <= D; ++r) v[r] = t[r];
    }
}

// and back to the numbers of the walk
template <class T>
__device__ __forceinline__ void from_remainders(int s, T (&v)[D + 1]) {
    to_remainders(s == 0 ? 0 : (s < 0 ? -s : D + 1 - s), v);
}

// ---- level constants in shared memory ---------------------------------------------------------
// A level's weight, shift and scale are 2D+1 floats that every thread of a block reads: staged once
// per block they cost a point two to four 16-byte shared loads per level instead of 2D+1 global ones
// (7 of the 11 load instructions of a level at pos_dim 3).
constexpr int kRecord = (2 * D + 2 + 3) / 4 * 4;  // weight, shift, scale, reach
constexpr int kStage = 32;  // levels staged at a time

__device__ __forceinline__ void stage_levels(const Problem& p, int begin, int end, float* table) {
    for (int i = threadIdx.x; i < (end - begin) * kRecord; i += blockDim.x) {
        const int l = begin + i / kRecord, c = i % kRecord;
        float v = 0.f;
        if (c == 0) v = __ldg(p.anneal + l);
        else if (c <= D) v = __ldg(p.shift + l * D + c - 1);
        else if (c <= 2 * D) v = __ldg(p.scale + l * D + c - 1 - D);
        else if (c == 2 * D + 1) v = exact_reach<D>(p.shift + l * D, p.scale + l * D);
        table[i] = v;
    }
}
__device__ __forceinline__ void load_level(const float* table, int i, LevelConst<D>& lc) {
    float v[kRecord];
#pragma unroll
    for (int j = 0; j < kRecord / 4; ++j) {
        const float4 t = reinterpret_cast<const float4*>(table + i * kRecord)[j];
        v[4 * j] = t.x;
        v[4 * j + 1] = t.y;
        v[4 * j + 2] = t.z;
        v[4 * j + 3] = t.w;
    }
    lc.weight = v[0];
    lc.reach = v[2 * D + 1];
#pragma unroll
    for (int j = 0; j < D; ++j) {
        lc.shift[j] = v[1 + j];
        lc.scale[j] = v[1 + D + j];
    }
}

// ---- F consecutive floats (one table entry, or one level of a feature row) ------------------
template <int F>
__device__ __forceinline__ void load_feats(const float* __restrict__ src, float (&v)[F]) {
    if (F == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(src));
        v[0] = t.x;
        v[1] = t.y;
    } else {
#pragma unroll
        for (int q = 0; q < F / 4; ++q) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(src) + q);
            v[4 * q + 0] = t.x;
            v[4 * q + 1] = t.y;
            v[4 * q + 2] = t.z;
            v[4 * q + 3] = t.w;
        }
    }
}
template <int F>
__device__ __forceinline__ void store_feats(float* dst, const float (&v)[F]) {
    if (F == 2) {
        *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
    } else {
#pragma unroll
        for (int q = 0; q < F / 4; ++q)
            reinterpret_cast<float4*>(dst)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
}

// 8 consecutive floats of a feature row (or one 8-feature table entry), 32-byte aligned
__device__ __forceinline__ void load8(const float* src, float (&v)[8]) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(src));
}
__device__ __forceinline__ void store8(float* dst, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// Point number i of the sweep and the row it belongs to: i itself, or, when the batch has been put
// into spatial order, the i-th record {coordinates, row} (16 bytes up to pos_dim 3, else 32).  The row is
// an index into every row-shaped operand, so it is held inside the batch whatever the buffer contains.
__device__ __forceinline__ int64_t load_point(const Problem& p, int64_t i, float (&pos)[D]) {
    if (p.order == nullptr) {
        load_pos(p, i, pos);
        return i;
    }
    if (D <= 3) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p.order) + i);
        pos[0] = t.x;
        pos[1] = t.y;
        if (D == 3) pos[D - 1] = t.z;
        return (int64_t)min(__float_as_uint(t.w), (uint32_t)p.n_points - 1u);
    }
    float r[8];
    load8(reinterpret_cast<const float*>(p.order) + 8 * i, r);
#pragma unroll
    for (int j = 0; j < D; ++j) pos[j] = r[j];
    return (int64_t)min(__float_as_uint(r[7]), (uint32_t)p.n_points - 1u);
}

// Aligned gather of one table entry (all F features) through the read-only path.  HALF: the
// table is stored as fp16 (storage only -- every product and sum below stays fp32), so an entry is
// 2F bytes: one 4-, 8- or 16-byte load.  Random accesses are bound by operations per second, not
// bytes, so a 4-feature fp16 entry (8 bytes) costs what a 2-feature fp32 entry costs, and the
// table takes half the room in L2.
template <int F, bool HALF>
__device__ __forceinline__ void gather(const void* __restrict__ table, int level, uint32_t capacity, uint32_t slot,
                                       float (&v)[F]) {
    const size_t entry = (size_t)level * capacity + slot;
    if (HALF) {
        const __half2* src = reinterpret_cast<const __half2*>(table) + entry * (F / 2);
        if (F == 2) {
            const unsigned raw = __ldg(reinterpret_cast<const unsigned*>(src));
            const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&raw));
            v[0] = t.x;
            v[1] = t.y;
        } else if (F == 4) {
            const uint2 raw = __ldg(reinterpret_cast<const uint2*>(src));
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
            const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
            v[0] = a.x;
            v[1] = a.y;
            v[2 % F] = b.x;
            v[3 % F] = b.y;
        } else {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src));
            const unsigned w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[q]));
                v[(2 * q) % F] = t.x;
                v[(2 * q + 1) % F] = t.y;
            }
        }
    } else {
        const float* src = reinterpret_cast<const float*>(table) + entry * F;
        if (F == 8) {
            asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=f"(v[0]), "=f"(v[1]), "=f"(v[2 % F]), "=f"(v[3 % F]), "=f"(v[4 % F]), "=f"(v[5 % F]),
                           "=f"(v[6 % F]), "=f"(v[7 % F])
                         : "l"(src));
        } else {
            load_feats<F>(src, v);
        }
    }
}

// vector reduction of one table-gradient entry: 8 bytes (F = 2) or 16 bytes (F = 4) per L2
// atomic -- both run at the same operation rate -- and two 16-byte ones for F = 8
template <int F>
__device__ __forceinline__ void red_add(float* level_base, uint32_t slot, const float (&x)[F]) {
    float* p = level_base + (size_t)slot * F;
    if (F == 2) {
        asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x[0]), "f"(x[1]) : "memory");
    } else {
#pragma unroll
        for (int q = 0; q < F / 4; ++q)
            asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * q), "f"(x[4 * q]),
                         "f"(x[4 * q + 1]), "f"(x[4 * q + 2]), "f"(x[4 * q + 3])
                         : "memory");
    }
}

// Row segment of point n starting at level l0: LPS levels of F floats.  One 32-byte vector access
// when the segment is a whole, aligned 8-float group; else per-level accesses.
template <int F, int LPS>
__device__ __forceinline__ void load_row_segment(const Problem& p, const float* rows, int64_t n, int l0,
                                                 float (&v)[F * LPS]) {
    const float* src = rows + n * p.width + F * l0;
    if (F * LPS == 8 && p.rows_vec8_ok && l0 + LPS <= p.level_end) {
        load8(src, reinterpret_cast<float(&)[8]>(v));
    } else {
#pragma unroll
        for (int k = 0; k < LPS; ++k) {
            float t[F];
#pragma unroll
            for (int f = 0; f < F; ++f) t[f] = 0.f;
            if (l0 + k < p.level_end) load_feats<F>(src + F * k, t);
#pragma unroll
            for (int f = 0; f < F; ++f) v[F * k + f] = t[f];
        }
    }
}
template <int F, int LPS>
__device__ __forceinline__ void store_row_segment(const Problem& p, float* rows, int64_t n, int l0,
                                                  const float (&v)[F * LPS]) {
    float* dst = rows + n * p.width + F * l0;
    if (F * LPS == 8 && p.rows_vec8_ok && l0 + LPS <= p.level_end) {
        store8(dst, reinterpret_cast<const float(&)[8]>(v));
    } else {
#pragma unroll
        for (int k = 0; k < LPS; ++k) {
            if (l0 + k < p.level_end) {
                float t[F];
#pragma unroll
                for (int f = 0; f < F; ++f) t[f] = v[F * k + f];
                store_feats<F>(dst + F * k, t);
            }
        }
    }
}

// Rows that do not start on a 32-byte boundary (level counts that are no multiple of four at F = 2, of two
// at F = 4): the row's values, handed over 8 at a time, go out as whole 32-byte sectors shifted by the
// row's misalignment, and only the ends of the row as 8-byte pieces.  Four 8-byte stores per step touch
// every sector four times (18 levels, 2^19 points: forward 134 -> 118 us, in spatial order 108 -> 91).
struct ShiftedRow {
    float* at;       // sector the next 8 values start in
    int m;           // values of that sector before them, 0, 2, 4 or 6
    int left;        // values still held in `held` when the row ends
    bool first;
    float held[8];   // the last 8 values, rotated by m: the first m are still to be written

    __device__ __forceinline__ explicit ShiftedRow(float* row) {
        m = (int)((reinterpret_cast<uintptr_t>(row) >> 2) & 7u);
        at = row - m;
        left = 0;
        first = true;
#pragma unroll
        for (int i = 0; i < 8; ++i) held[i] = 0.f;
    }
    __device__ __forceinline__ void push(const float (&v)[8], int valid) {
        float a[8], r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = (m & 4) ? v[(i + 4) & 7] : v[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = (m & 2) ? a[(i + 6) & 7] : a[i];
        float out[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = i < m ? held[i] : r[i];
        left = m + valid - 8;
        if (left >= 0 && (!first || m == 0)) {
            store8(at, out);
        } else {
#pragma unroll
            for (int q = 0; q < 8; q += 2)
                if ((!first || q >= m) && q < m + valid) *reinterpret_cast<float2*>(at + q) = make_float2(out[q], out[q + 1]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) held[i] = r[i];
        at += 8;
        first = false;
    }
    __device__ __forceinline__ void finish() {
#pragma unroll
        for (int q = 0; q < 8; q += 2)
            if (q < left) *reinterpret_cast<float2*>(at + q) = make_float2(held[q], held[q + 1]);
    }
};

// ------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------
// One step of a point's feature row: LPS levels of F features (8 floats) starting at level l0;
// levels at or beyond `end` give zeros (EncodingGPU.cuh:130-254 for one level).
template <int F, int LPS, bool HALF>
__device__ __forceinline__ void encode_step(const Problem& p, const float* levels, const float (&pos)[D], float largest,
                                            int l0, int end, float (&out)[F * LPS]) {
#pragma unroll
    for (int k = 0; k < LPS; ++k) {
        const int l = l0 + k;
        float acc[F];
#pragma unroll
        for (int f = 0; f < F; ++f) acc[f] = 0.f;
        if (l < end) {  // uniform over the block
            LevelConst<D> lc;
            load_level(levels, k, lc);
            if (lc.weight != 0.0f) {  // a closed coarse-to-fine window contributes exact zeros
                Simplex<D> s;
                locate_simplex<D>(pos, largest, lc, s);
                uint32_t slot[D + 1];
                to_slots(p, s, slot);
                float v[D + 1][F];
#pragma unroll
                for (int q = 0; q <= D; ++q) gather<F, HALF>(p.table, l, p.capacity, slot[q], v[q]);
                float w[D + 1];
                vertex_weights<D>(s, lc.weight * (1.0f / (D + 1)), w);  // EncodingGPU.cuh:234
#pragma unroll
                for (int q = 0; q <= D; ++q) {
#pragma unroll
                    for (int f = 0; f < F; ++f) acc[f] = fmaf(v[q][f], w[q], acc[f]);
                }
            }
        }
#pragma unroll
        for (int f = 0; f < F; ++f) out[F * k + f] = acc[f];
    }
}

// SHIFTED: rows off the 32-byte grid, written by a ShiftedRow.  Its held values spill at the occupancy of
// the plain kernel, which costs more than the warps (17 levels, 2^19 points, 8 / 6 / 5 / 4 blocks per SM:
// 149 / 126 / 115 / 115 us).
constexpr int forward_blocks(int feats, bool shifted) {
    return feats == 2 ? (shifted ? (D <= 5 ? 5 : 4) : PERMUTO_MIN_BLOCKS_FORWARD) : min_blocks(feats, false);
}
template <int F, int LPS, bool HALF, bool SHIFTED>
__global__ void __launch_bounds__(kThreads, forward_blocks(F, SHIFTED)) forward_kernel(const ForwardArgs a) {
    const Problem& p = a.p;
    __shared__ __align__(16) float levels[kStage * kRecord];
    const int64_t i_raw = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool active = i_raw < p.n_points;
    const int pass_begin = p.level_begin + (int)blockIdx.y * p.levels_per_pass;
    const int pass_end = min(pass_begin + p.levels_per_pass, p.level_end);

    float pos[D];
    const int64_t n = load_point(p, active ? i_raw : p.n_points - 1, pos);  // idle threads shadow the last point
    const float largest = largest_coordinate<D>(pos);
    ShiftedRow row(a.features + n * p.width + F * pass_begin);  // used by SHIFTED only

#pragma unroll 1
    for (int begin = pass_begin; begin < pass_end; begin += kStage) {
        const int end = min(begin + kStage, pass_end);
        if (begin != pass_begin) __syncthreads();
        stage_levels(p, begin, end, levels);
        __syncthreads();
        const int nsteps = (end - begin + LPS - 1) / LPS;
        // without an order, blocks start at different steps as in the scatter kernels (1 %)
        int step = (!SHIFTED && p.order == nullptr) ? (int)(blockIdx.x % (unsigned)nsteps) : 0;
#pragma unroll 1
        for (int it = 0; it < nsteps; ++it) {
            const int l0 = begin + step * LPS;
            step = (step + 1 == nsteps) ? 0 : step + 1;
            float out[F * LPS];
            encode_step<F, LPS, HALF>(p, levels + (l0 - begin) * kRecord, pos, largest, l0, end, out);
            if (SHIFTED) {
                if (active) row.push(reinterpret_cast<const float(&)[8]>(out), F * min(LPS, end - l0));
            } else if (active) {
                store_row_segment<F, LPS>(p, a.features, n, l0, out);
            }
        }
    }
    if (SHIFTED && active) row.finish();

    // raw points appended after the lattice levels (EncodingGPU.cuh:105-121)
    if (active && p.extra_levels > 0 && blockIdx.y == 0 && p.level_begin == 0) {
        float* dst = a.features + n * p.width + F * p.nr_levels;
        for (int c = 0; c < F * p.extra_levels; ++c) {
            float v = 0.f;
#pragma unroll
            for (int i = 0; i < D; ++i) v = (c == i) ? pos[i] * p.points_scaling : v;
            dst[c] = v;
        }
    }
}

// ------------------------------------------------------------------------------------------
// forward fused with the consumer's first linear layer (tcgen05 + TMEM)
// ------------------------------------------------------------------------------------------
// The users of the encoding feed the [N, F*L] feature row straight into a small MLP (reference:
// examples/train_toy_example.py:18-26, README.md:39-40).  Here a block of 128 threads encodes 128
// points, passes the 128 x K feature tile (K = F*(L+extra), rounded to tf32) through shared memory
// 8 columns at a time and multiplies it by the layer's weight [H, K] on the tensor cores: K/8
// tcgen05.mma of shape 128 x H x 8 (kind::tf32, fp32 accumulate) issued by one thread, accumulator
// in tensor memory, read back with tcgen05.ld (thread t holds row t) and written as [N, H] with
// the bias added.  The 192 B/point feature row and the separate GEMM's read of it never touch HBM.
//
// Shared-memory operand layout (K-major, no swizzle -- the canonical layout of the tcgen05
// matrix descriptor): 8 rows x 16 bytes form a contiguous 128-byte core matrix; the core
// matrices of consecutive 4-column groups follow each other (leading byte offset 128) and those
// of consecutive 8-row groups are a fixed number of bytes apart (stride byte offset).
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 64-bit shared-memory matrix descriptor: start address, leading / stride byte offsets (all in
// units of 16 bytes), descriptor version 1 (Blackwell), no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t leading_bytes, uint32_t stride_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(leading_bytes >> 4) << 16) |
           ((uint64_t)(stride_bytes >> 4) << 32) | (1ull << 46);
}

// 32-bit instruction descriptor for kind::tf32: D = fp32 (bits 4-5 = 1), A and B = tf32 (bits 7-9
// and 10-12 = 2), both K-major (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24
__device__ __forceinline__ uint32_t instr_desc_tf32(int m, int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ float to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// the mbarrier receives one arrival when every tcgen05.mma issued so far by this thread is done
__device__ __forceinline__ void commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

// Bounded wait for phase `parity` of an mbarrier: false when the limit ran out (the caller then
// reports it and skips its output instead of spinning for ever).
__device__ __forceinline__ bool wait_bounded(uint32_t mbar, uint32_t parity) {
    for (int it = 0; it < (1 << 20); ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

}  // namespace umma

constexpr int kTileRows = 128;  // points per block = rows of one tcgen05.mma
#ifndef PERMUTO_FUSED_RING
#define PERMUTO_FUSED_RING 2
#endif
constexpr int kRing = PERMUTO_FUSED_RING;  // 128 x 8 slices in flight between the threads and the tensor core
constexpr uint32_t kSliceBytes = kTileRows * 8 * 4;  // one slice: 128 rows x 8 tf32 = 4 KB

// The A operand of every product is never whole in shared memory: 8 columns of the 128-row tile
// (a K = 8 slice of the product) are written into a ring of kRing slices and consumed by one
// tcgen05.mma right away, accumulating in tensor memory.  That keeps a block at 8 KB + the
// weights instead of 128 x K x 4 bytes, so that shared memory neither limits the resident blocks
// nor eats the L1 capacity the coarse levels' gathers live on.
struct SliceRing {
    unsigned char* base;   // kRing slices
    uint64_t* free_bar;    // one mbarrier per slice: arrives when the MMA that read it is done
    uint32_t base_addr;
    uint32_t row_off;      // this thread's row inside a slice
    int pushed;            // slices written so far (all layers)
    bool ok;               // no bounded wait has run out

    // Write this thread's 8 values of the next slice; when the whole block has, thread 0 issues
    // D[128 x n] (+)= slice[128 x 8] * B[n x 8]^T and commits to the slice's barrier.
    // Block-uniform control flow: every thread of the block calls it.
    __device__ __forceinline__ void push(const float (&v)[8], uint32_t tmem_d, uint32_t b_addr, uint32_t b_stride,
                                         uint32_t idesc, bool accumulate) {
        const int slot = pushed % kRing;
        // the MMA that read this slice kRing pushes ago must be done before it is overwritten
        if (pushed >= kRing) ok = umma::wait_bounded(umma::smem_u32(&free_bar[slot]), (uint32_t)((pushed / kRing - 1) & 1)) && ok;
        unsigned char* dst = base + (size_t)slot * kSliceBytes + row_off;
        *reinterpret_cast<float4*>(dst) =
            make_float4(umma::to_tf32(v[0]), umma::to_tf32(v[1]), umma::to_tf32(v[2]), umma::to_tf32(v[3]));
        *reinterpret_cast<float4*>(dst + 128) =
            make_float4(umma::to_tf32(v[4]), umma::to_tf32(v[5]), umma::to_tf32(v[6]), umma::to_tf32(v[7]));
        // the block's writes -> visible to the tensor core (async proxy); then one thread issues the slice's MMA
        // (and what the threads have read from tensor memory is ordered before it may be overwritten)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            umma::mma_tf32(tmem_d, umma::smem_desc(base_addr + (uint32_t)slot * kSliceBytes, 128u, 256u),
                           umma::smem_desc(b_addr, 128u, b_stride), idesc, accumulate);
            umma::commit(umma::smem_u32(&free_bar[slot]));  // covers every MMA issued so far
        }
        ++pushed;
    }

    // Wait until every MMA issued so far is done (the last commit covers them all); the result is
    // made block-uniform, because tcgen05.ld afterwards must be executed by whole warps.
    __device__ __forceinline__ bool drain() {
        const int last = pushed - 1;
        ok = umma::wait_bounded(umma::smem_u32(&free_bar[last % kRing]), (uint32_t)((last / kRing) & 1)) && ok;
        ok = __syncthreads_and(ok) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return ok;
    }
};

// weight [rows, cols] row-major in global memory -> shared memory in the K-major operand layout
// with `chunks` 16-byte column groups per row, rounded to tf32; columns beyond `cols` are zero
__device__ __forceinline__ void stage_weight(unsigned char* tile, const float* __restrict__ weight, int rows, int cols,
                                             int chunks) {
    const uint32_t stride = (uint32_t)chunks * 128u;
    const bool vec = (cols % 4 == 0) && ((reinterpret_cast<uintptr_t>(weight) & 15u) == 0);
    for (int e = threadIdx.x; e < rows * chunks; e += kTileRows) {
        const int n = e / chunks, kc = e - n * chunks;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* src = weight + (size_t)n * cols + 4 * kc;
        if (vec && 4 * kc + 3 < cols) {
            w = __ldg(reinterpret_cast<const float4*>(src));
        } else {
            if (4 * kc + 0 < cols) w.x = __ldg(src + 0);
            if (4 * kc + 1 < cols) w.y = __ldg(src + 1);
            if (4 * kc + 2 < cols) w.z = __ldg(src + 2);
            if (4 * kc + 3 < cols) w.w = __ldg(src + 3);
        }
        *reinterpret_cast<float4*>(tile + (size_t)(n >> 3) * stride + (size_t)kc * 128 + (n & 7) * 16) =
            make_float4(umma::to_tf32(w.x), umma::to_tf32(w.y), umma::to_tf32(w.z), umma::to_tf32(w.w));
    }
}

// 16 consecutive accumulator columns of this thread's row (tensor-memory lane = row)
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));  // all 32 lanes of the warp take part
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Packed fp32 pairs: one instruction, the IEEE result in each half.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// torch.nn.GELU() of two values: x * Phi(x) = max(x, 0) - |x| * Q(t) * exp(-x^2 / 2), t = 1 / (1 + p |x|).
// Q is the degree-6 polynomial (no constant term) with the smallest largest error of erfc against
// erfcx(x) * exp(-x^2) on [0, 6], p = 0.4 / sqrt(2): 2.8e-8 before rounding, 2.4e-7 absolute in fp32 with
// the approximate reciprocal and exponential (the form through 1 + erf had 4.7e-7).  About ten issue
// slots a value instead of 25: a hidden layer was mostly this.
__device__ __forceinline__ void gelu2(float& x, float& y) {
    const uint64_t v = pack2(x, y);
    const float ax = fminf(fabsf(x), 1e18f), ay = fminf(fabsf(y), 1e18f);  // infinity times zero otherwise
    const uint64_t a = pack2(ax, ay);
    float dx, dy, sx, sy;
    unpack2(fma2(a, pack2(0.282842712f, 0.282842712f), pack2(1.f, 1.f)), dx, dy);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(dx));
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(dy));
    const uint64_t t = pack2(dx, dy);
    uint64_t q = fma2(t, pack2(-0.100129196f, -0.100129196f), pack2(0.354571956f, 0.354571956f));
    q = fma2(t, q, pack2(-0.1854512479f, -0.1854512479f));
    q = fma2(t, q, pack2(0.2341349315f, 0.2341349315f));
    q = fma2(t, q, pack2(0.08091262737f, 0.08091262737f));
    q = fma2(t, q, pack2(0.1159609153f, 0.1159609153f));
    q = mul2(t, q);
    unpack2(mul2(mul2(v, pack2(-0.72134752f, -0.72134752f)), v), sx, sy);  // -x^2 / 2 * log2(e)
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(sx));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(sy));
    const uint64_t m = mul2(pack2(-ax, -ay), pack2(sx, sy));
    unpack2(fma2(m, q, pack2(fmaxf(x, 0.f), fmaxf(y, 0.f))), x, y);
}

// HMAX = 0: the encoding followed by ONE linear layer (out = features @ W^T + b).
// HMAX = 32 / 64: a whole small MLP behind the encoding; hidden widths are multiples of 16 up to
// HMAX (a thread holds its row of hidden activations in registers between two layers).
// Resident blocks per SM: ten of the one-layer kernel, and six of the small MLP, whose row of 32 hidden
// activations would spill at eight (pos_dim 4: 469 -> 400 us); more blocks also leave too little L1 beside
// their shared memory for the gathers (one layer at eleven or twelve: 285 -> 297 us on 10^6 ray samples).
constexpr int fused_blocks(int feats, int hmax) { return feats == 2 && hmax <= 32 ? (hmax ? 6 : 10) : 4; }
template <int F, int LPS, bool HALF, int HMAX>
__global__ void __launch_bounds__(kTileRows, fused_blocks(F, HMAX))
forward_mlp_kernel(const ForwardLinearArgs a) {
    const Problem& p = a.p;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t slice_free[kRing];
    __shared__ uint32_t tmem_base;

    const int t = threadIdx.x;
    const int warp = t >> 5;
    const int H0 = a.layer[0].out_features;
    const uint32_t tmem_cols = (uint32_t)a.tmem_cols;  // a power of two >= 32 (host-computed)

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(umma::smem_u32(&tmem_base)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (t == 0) {
#pragma unroll
        for (int i = 0; i < kRing; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(umma::smem_u32(&slice_free[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // shared memory: the slice ring, then the weight of every layer that runs on the tensor core
    unsigned char* tile_w = smem_raw + kRing * kSliceBytes;
    const int chunks0 = a.k_pad / 4;
    float* levels = reinterpret_cast<float*>(smem_raw + a.levels_offset);  // behind the weights
    float* biases = levels + p.nr_levels * kRecord;  // one layer after the other, zeros where there is none
    float* narrow = nullptr;                         // weight rows of a narrow last layer
    {
        int at = 0;
        for (int i = 0; i < a.nr_layers; ++i) {
            const MlpLayer& ly = a.layer[i];
            const int padded = (ly.out_features + 3) / 4 * 4;
            for (int k = t; k < padded; k += kTileRows) biases[at + k] = ly.bias && k < ly.out_features ? __ldg(ly.bias + k) : 0.f;
            at += padded;
        }
        const MlpLayer& ly = a.layer[a.nr_layers - 1];
        if (HMAX > 0 && ly.out_features % 16 != 0) {
            narrow = biases + at;
            for (int k = t; k < ly.out_features * ly.in_features; k += kTileRows) narrow[k] = __ldg(ly.weight + k);
        }
    }
    stage_levels(p, 0, p.nr_levels, levels);
    stage_weight(tile_w, a.layer[0].weight, H0, p.width, chunks0);
    if (HMAX > 0) {
        unsigned char* next = tile_w + (size_t)H0 * a.k_pad * 4;
        for (int i = 1; i < a.nr_layers; ++i) {
            const MlpLayer& ly = a.layer[i];
            if (ly.out_features % 16 != 0) break;  // a narrow last layer is evaluated in registers
            stage_weight(next, ly.weight, ly.out_features, ly.in_features, ly.in_features / 4);
            next += (size_t)ly.out_features * ly.in_features * 4;
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    SliceRing ring;
    ring.base = smem_raw;
    ring.free_bar = slice_free;
    ring.base_addr = umma::smem_u32(smem_raw);
    ring.row_off = (uint32_t)(t >> 3) * 256u + (uint32_t)(t & 7) * 16u;  // 8-row groups 256 bytes apart
    ring.pushed = 0;
    ring.ok = true;

    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);  // tensor-memory lane = 32*warp + lane = row t
    bool ok = true;
    // A block walks over tiles of 128 points: what stands above -- tensor memory, barriers, weights -- is
    // set up once per resident block, not once per tile (355 -> 307 us on 10^6 ray samples).
    const int64_t tiles = (p.n_points + kTileRows - 1) / kTileRows;
#pragma unroll 1
    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        // ---- layer 0: this thread's point -> row t of every slice ----------------------------------
        const int64_t i_raw = tile * kTileRows + t;
        const bool active = i_raw < p.n_points;
        int64_t n;
        {
            float pos[D];
            n = load_point(p, active ? i_raw : p.n_points - 1, pos);  // idle rows shadow the last point and are not stored
            const float largest = largest_coordinate<D>(pos);
            const int lattice_cols = F * p.nr_levels;
            // a column past the lattice levels: a concatenated raw coordinate (EncodingGPU.cuh:105-121) or padding
            auto tail_value = [&](int c) -> float {
                float v = 0.f;
                const int i = c - lattice_cols;
#pragma unroll
                for (int j = 0; j < D; ++j) v = (i == j && c < p.width) ? pos[j] * p.points_scaling : v;
                return v;
            };
            const int nsteps = (p.nr_levels + LPS - 1) / LPS;  // steps that hold lattice levels
            const int ksteps = a.k_pad / 8;                    // all steps: one tcgen05.mma each
            const uint32_t idesc = umma::instr_desc_tf32(kTileRows, H0);
            const uint32_t addr_w = umma::smem_u32(tile_w);
#pragma unroll 1
            for (int s = 0; s < ksteps; ++s) {
                float out[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) out[i] = 0.f;
                if (s < nsteps) encode_step<F, LPS, HALF>(p, levels + s * LPS * kRecord, pos, largest, s * LPS, p.nr_levels, out);
                if (8 * s + 8 > lattice_cols) {  // block-uniform: only the last step(s) reach past the lattice levels
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int c = 8 * s + i;
                        out[i] = (c >= lattice_cols) ? tail_value(c) : out[i];
                    }
                }
                ring.push(out, tmem, addr_w + (uint32_t)s * 256u, (uint32_t)chunks0 * 128u, idesc, s > 0);
            }
        }

        int last = 0;          // layer whose accumulators are in tensor memory
        const float* bias = biases;  // of that layer

        // ---- hidden layers: accumulators -> registers (+bias, activation) -> slices -> next product ----
        if (HMAX > 0) {
            constexpr int HM = HMAX > 0 ? HMAX : 16;
            uint32_t w_addr = umma::smem_u32(tile_w) + (uint32_t)H0 * (uint32_t)a.k_pad * 4u;
            for (int i = 1; i < a.nr_layers; ++i) {
                const MlpLayer& ly = a.layer[i];
                const int width = ly.in_features;  // = out_features of layer i-1, a multiple of 16 up to HMAX
                ok = ring.drain() && ok;
                float h[HM];
                const int kind = a.activation;
#pragma unroll
                for (int c = 0; c < HM / 16; ++c) {
                    if (16 * c < width) {
                        float v[16];
                        tmem_load16(lane_base + 16u * c, v);
#pragma unroll
                        for (int k = 0; k < 16; k += 4) {
                            const float4 b = *reinterpret_cast<const float4*>(bias + 16 * c + k);
                            unpack2(add2(pack2(v[k], v[k + 1]), pack2(b.x, b.y)), v[k], v[k + 1]);
                            unpack2(add2(pack2(v[k + 2], v[k + 3]), pack2(b.z, b.w)), v[k + 2], v[k + 3]);
                        }
                        // one uniform branch per group, not one per element
                        if (kind == PERMUTO_ACT_GELU) {
#pragma unroll
                            for (int k = 0; k < 16; k += 2) gelu2(v[k], v[k + 1]);
                        } else if (kind == PERMUTO_ACT_RELU) {
#pragma unroll
                            for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k], 0.f);
                        }
#pragma unroll
                        for (int k = 0; k < 16; ++k) h[16 * c + k] = v[k];
                    }
                }
                bias += width;  // a multiple of 16
                if (ly.out_features % 16 != 0) {
                    // narrow last layer (e.g. one output): plain fp32 dot products in registers
                    if (active && ok) {
                        for (int o = 0; o < ly.out_features; ++o) {
                            float acc = bias[o];
                            const float4* w = reinterpret_cast<const float4*>(narrow + o * width);
#pragma unroll
                            for (int k = 0; k < HM; k += 4) {
                                if (k < width) {
                                    const float4 u = w[k / 4];
                                    acc = fmaf(h[k], u.x, acc);
                                    acc = fmaf(h[k + 1], u.y, acc);
                                    acc = fmaf(h[k + 2], u.z, acc);
                                    acc = fmaf(h[k + 3], u.w, acc);
                                }
                            }
                            a.out[n * ly.out_features + o] = acc;
                        }
                    }
                    last = -1;  // everything is written
                    break;
                }
                // the product goes to the columns it came from: every row is in registers when the block meets
                // in the first push, before its MMA is issued
                const uint32_t idesc = umma::instr_desc_tf32(kTileRows, ly.out_features);
#pragma unroll
                for (int j = 0; j < HM / 8; ++j) {
                    if (8 * j < width) {
                        float v[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = h[8 * j + k];
                        ring.push(v, tmem, w_addr + (uint32_t)j * 256u, (uint32_t)(width / 4) * 128u, idesc, j > 0);
                    }
                }
                w_addr += (uint32_t)ly.out_features * (uint32_t)width * 4u;
                last = i;
            }
        }

        // ---- last tensor-core layer: accumulators + bias -> out[N, out_features] -------------------------
        if (last >= 0) {
            ok = ring.drain() && ok;
            const int H = a.layer[last].out_features;
            if (ok) {
                float* dst = a.out + n * H;
                for (int c = 0; c < H; c += 16) {
                    float v[16];
                    tmem_load16(lane_base + (uint32_t)c, v);
                    if (active) {
#pragma unroll
                        for (int h8 = 0; h8 < 2; ++h8) {
                            float o[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) o[k] = v[8 * h8 + k] + bias[c + 8 * h8 + k];
                            if (a.out_vec8_ok) {
                                store8(dst + c + 8 * h8, o);
                            } else {
                                reinterpret_cast<float4*>(dst + c + 8 * h8)[0] = make_float4(o[0], o[1], o[2], o[3]);
                                reinterpret_cast<float4*>(dst + c + 8 * h8)[1] = make_float4(o[4], o[5], o[6], o[7]);
                            }
                        }
                    }
                }
            }
        }
    }
    if (!ok && a.status && t == 0) atomicExch(a.status, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

// ------------------------------------------------------------------------------------------
// scatter-add of the d+1 table-gradient entries of one level, colliding lanes merged first
// ------------------------------------------------------------------------------------------
// On coarse levels the 32 points of a warp hit a handful of slots; sending 32 same-address
// reductions to L2 serialises there (2.0-3.6 ms per backward instead of 0.47 on the training
// shape).  match.any groups the lanes by slot, a pointer-jumping suffix sum over each group's
// lanes (log2 of the largest group rounds) leaves the group total in its lowest lane, and only
// that lane issues the vector reduction.  The summation order is fixed by the lane order, so a
// warp's contribution is deterministic.
//
// The d+1 vertices are merged together, round by round, not one after the other: a round is a
// chain match/shuffle -> add -> shuffle whose latency nothing else in the warp can hide, and the
// d+1 chains are independent of each other.  (With the vertices merged one after the other the
// coarse half of the levels took as long as the fine half, although it sends a quarter of the
// reductions to L2.)
//
// Merging pays only while a warp's 32 points share slots: per warp and vertex the number of
// distinct slots on the training shape is 6, 7, 9, 15, 22, 38, 63, 96, 116, 124 of 128 for levels
// 0..9 and 128 from level 11 on, and match.any itself is slowest when all keys differ.  The
// match of vertex 0 doubles as the probe: when it finds more than kMergeBelow distinct slots the
// level is scattered directly and -- collisions only get rarer towards finer levels -- the warp
// stops probing until its walk over the levels restarts at the coarsest one.
//
// Blocks start their walk over the steps of a pass at different steps (block index modulo the
// number of steps), so that at any moment the blocks in flight work on different levels instead
// of all sending their reductions to the few hot slots of the same coarse level (2-4 % on the
// scatter kernels).
#ifndef PERMUTO_MERGE_BELOW
#define PERMUTO_MERGE_BELOW 24
#endif
#ifndef PERMUTO_STAGGER
#define PERMUTO_STAGGER 1
#endif
constexpr int kMergeBelow = PERMUTO_MERGE_BELOW;
constexpr bool kStagger = PERMUTO_STAGGER != 0;

// per-thread state of the scatter of one warp
struct Scatter {
    unsigned lane;
    bool active;  // this lane owns a point
    bool probe;   // warp-uniform: keep testing levels for mergeable collisions
};

// Vertices merged side by side: all of them up to pos_dim 4; beyond that half at a time, which
// keeps the d+1 partial sums, group masks and chain pointers within the register budget.
#ifndef PERMUTO_MERGE_CHUNK
#define PERMUTO_MERGE_CHUNK (PERMUTO_DIM <= 4 ? PERMUTO_DIM + 1 : (PERMUTO_DIM + 2) / 2)
#endif
constexpr int kMergeChunk = PERMUTO_MERGE_CHUNK;

// vertices [R0, R0 + CNT) of one level: segmented suffix sums over the lanes of every group,
// then one reduction per group from its lowest lane.  group[0] is passed in when R0 == 0.
template <int F, int R0, int CNT>
__device__ __forceinline__ void merge_vertices(const Scatter& sc, float* level_base, const uint32_t (&slot)[D + 1],
                                               float (&add)[D + 1][F], unsigned group0) {
    const unsigned lane = sc.lane;
    const uint32_t idle = 0xffffffffu - lane;  // idle lanes match nobody
    const unsigned below = (1u << lane) - 1u;
    unsigned group[CNT];
    int next[CNT];  // next higher lane of the same group, -1 at the end of the chain
    int largest = 0;
#pragma unroll
    for (int c = 0; c < CNT; ++c) {
        group[c] = (R0 == 0 && c == 0) ? group0 : __match_any_sync(kFullMask, sc.active ? slot[R0 + c] : idle);
        largest = max(largest, __popc(group[c]));
        const unsigned above = group[c] & (0xfffffffeu << lane);
        next[c] = above ? (__ffs(above) - 1) : -1;
    }
    largest = __reduce_max_sync(kFullMask, largest);
    for (int span = 1; span < largest; span <<= 1) {  // warp-uniform trip count
#pragma unroll
        for (int c = 0; c < CNT; ++c) {
            const int src = next[c] >= 0 ? next[c] : (int)lane;
            float x2[F];
#pragma unroll
            for (int f = 0; f < F; ++f) x2[f] = __shfl_sync(kFullMask, add[R0 + c][f], src);
            const int n2 = __shfl_sync(kFullMask, next[c], src);
            if (next[c] >= 0) {
#pragma unroll
                for (int f = 0; f < F; ++f) add[R0 + c][f] += x2[f];
                next[c] = n2;
            }
        }
    }
    if (sc.active) {
#pragma unroll
        for (int c = 0; c < CNT; ++c)
            if ((group[c] & below) == 0u) red_add<F>(level_base, slot[R0 + c], add[R0 + c]);
    }
}

template <int F, int R0>
__device__ __forceinline__ void merge_from(const Scatter& sc, float* level_base, const uint32_t (&slot)[D + 1],
                                           float (&add)[D + 1][F], unsigned group0) {
    if constexpr (R0 <= D) {
        constexpr int CNT = (D + 1 - R0) < kMergeChunk ? (D + 1 - R0) : kMergeChunk;
        merge_vertices<F, R0, CNT>(sc, level_base, slot, add, group0);
        merge_from<F, R0 + CNT>(sc, level_base, slot, add, group0);
    }
}

// adds w[q] * g[f] to entry slot[q] of the level for every vertex q; `s` renumbers the vertices by remainder
template <int F>
__device__ __forceinline__ void scatter_level(Scatter& sc, float* level_base, int s, uint32_t (&slot)[D + 1],
                                              float (&w)[D + 1], const float (&g)[F]) {
    float add[D + 1][F];
    if (sc.probe) {
        to_remainders(s, slot);
        const unsigned lane = sc.lane;
        const unsigned group0 = __match_any_sync(kFullMask, sc.active ? slot[0] : 0xffffffffu - lane);
        const int distinct = __popc(__ballot_sync(kFullMask, (group0 & ((1u << lane) - 1u)) == 0u));
        to_remainders(s, w);
        if (distinct <= kMergeBelow) {
#pragma unroll
            for (int r = 0; r <= D; ++r) {
#pragma unroll
                for (int f = 0; f < F; ++f) add[r][f] = w[r] * g[f];
            }
            merge_from<F, 0>(sc, level_base, slot, add, group0);
            return;
        }
        sc.probe = false;
    }
    if (sc.active) {
#pragma unroll
        for (int r = 0; r <= D; ++r) {
#pragma unroll
            for (int f = 0; f < F; ++f) add[r][f] = w[r] * g[f];
            red_add<F>(level_base, slot[r], add[r]);
        }
    }
}

// d loss / d barycentric weight of every vertex, times the level weight (EncodingGPU.cuh:1187-1218)
__device__ __forceinline__ void second_order_weights(const Simplex<D>& s, const LevelConst<D>& lc, const float (&dpg)[D],
                                                     float (&dBw)[D + 1]) {
    float gsd[D], dE[D + 1];  // d loss / d elevated
#pragma unroll
    for (int i = 0; i < D; ++i) gsd[i] = dpg[i] * lc.scale[i];
#pragma unroll
    for (int j = 0; j <= D; ++j) dE[j] = 0.f;
#pragma unroll
    for (int i = 0; i < D; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) dE[j] += gsd[i];
    }
#pragma unroll
    for (int i = 0; i < D; ++i) dE[i + 1] -= gsd[i] * (float)(i + 1);
#pragma unroll
    for (int i = 0; i <= D; ++i) dE[i] *= 1.0f / (D + 1);
    to_ranks(s, dE);  // the gaps of dE in rank order
#pragma unroll
    for (int m = 1; m <= D; ++m) dBw[m] = (dE[D - m] - dE[D + 1 - m]) * lc.weight;
    dBw[0] = (dE[D] - dE[0]) * lc.weight;
}

// ------------------------------------------------------------------------------------------
// first-order backward: table gradient (scatter) and/or position gradient (gather)
// ------------------------------------------------------------------------------------------
template <int F, int LPS, bool TABLE, bool POS, bool HALF>
__global__ void __launch_bounds__(kThreads, min_blocks(F, !TABLE))
backward_kernel(const BackwardArgs a) {
    const Problem& p = a.p;
    __shared__ __align__(16) float levels[kStage * kRecord];
    const int64_t i_raw = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool active = i_raw < p.n_points;
    const int pass_begin = p.level_begin + (int)blockIdx.y * p.levels_per_pass;
    const int pass_end = min(pass_begin + p.levels_per_pass, p.level_end);
    const unsigned lane = threadIdx.x & 31u;
    constexpr float kInv = 1.0f / (D + 1);

    float pos[D];
    const int64_t n = load_point(p, active ? i_raw : p.n_points - 1, pos);  // idle lanes shadow the last point
    const float largest = largest_coordinate<D>(pos);

    float dpos[D];
#pragma unroll
    for (int i = 0; i < D; ++i) dpos[i] = 0.f;
    Scatter sc{lane, active, a.aggregate != 0};

#pragma unroll 1
    for (int begin = pass_begin; begin < pass_end; begin += kStage) {
        const int end = min(begin + kStage, pass_end);
        // steps are walked cyclically from a block-dependent start (see PERMUTO_STAGGER)
        const int nsteps = (end - begin + LPS - 1) / LPS;
        int step = (TABLE && kStagger) ? (int)(blockIdx.x % (unsigned)nsteps) : 0;
        // the next step's 32 bytes of the gradient row are requested before this step is worked on
        float g_next[F * LPS];
        load_row_segment<F, LPS>(p, a.grad_features, n, begin + step * LPS, g_next);
        if (begin != pass_begin) __syncthreads();
        stage_levels(p, begin, end, levels);
        __syncthreads();
#pragma unroll 1
        for (int it = 0; it < nsteps; ++it) {
            const int l0 = begin + step * LPS;
            step = (step + 1 == nsteps) ? 0 : step + 1;
            if (TABLE && l0 == begin) sc.probe = a.aggregate != 0;
            float g[F * LPS];
#pragma unroll
            for (int i = 0; i < F * LPS; ++i) g[i] = g_next[i];
            if (it + 1 < nsteps) load_row_segment<F, LPS>(p, a.grad_features, n, begin + step * LPS, g_next);
#pragma unroll
            for (int k = 0; k < LPS; ++k) {
                const int l = l0 + k;
                if (l >= end) continue;  // uniform
                LevelConst<D> lc;
                load_level(levels, l - begin, lc);
                if (lc.weight == 0.0f) continue;  // every addend of this level is an exact zero
                Simplex<D> s;
                locate_simplex<D>(pos, largest, lc, s);
                uint32_t slot[D + 1];
                to_slots(p, s, slot);

                if (POS) {
                    // EncodingGPU.cuh:671-749
                    float gs[F];  // upstream gradient with the level weight and 1/(d+1) folded in
#pragma unroll
                    for (int f = 0; f < F; ++f) gs[f] = g[F * k + f] * lc.weight * kInv;
                    float dBs[D + 2];
#pragma unroll
                    for (int q = 0; q <= D; ++q) {
                        float v[F];
                        gather<F, HALF>(p.table, l, p.capacity, slot[q], v);
                        float t = v[0] * gs[0];
#pragma unroll
                        for (int f = 1; f < F; ++f) t = fmaf(v[f], gs[f], t);
                        dBs[q] = t;
                    }
                    dBs[D + 1] = dBs[0];
                    float dE[D + 1];  // of the coordinate whose rank is k, then by coordinate
#pragma unroll
                    for (int kk = 0; kk <= D; ++kk) dE[kk] = dBs[D - kk] - dBs[D + 1 - kk];
                    to_coordinates(s, dE);
                    float run = 0.f;
#pragma unroll
                    for (int i = 0; i < D; ++i) {
                        run += dE[i];
                        dpos[i] += lc.scale[i] * (run - (float)(i + 1) * dE[i + 1]);
                    }
                }

                if (TABLE) {
                    float* gbase = a.lattice_grad + (size_t)l * p.capacity * F;
                    float gk[F], w[D + 1];
#pragma unroll
                    for (int f = 0; f < F; ++f) gk[f] = g[F * k + f];
                    vertex_weights<D>(s, lc.weight * kInv, w);  // EncodingGPU.cuh:405-410
                    scatter_level<F>(sc, gbase, s.s, slot, w, gk);
                }
            }
        }
    }
    // Optional: the concatenated raw coordinates are outputs too, d out[F*L + i] / d pos[i] =
    // points_scaling.  The reference leaves this term out (its backward grids exclude the extra
    // levels, src/Encoding.cu:129-134,161), so it is added only on request.
    if (POS && a.concat_grad && p.extra_levels > 0 && blockIdx.y == 0 && p.level_begin == 0) {
        const float* g = a.grad_features + n * p.width + F * p.nr_levels;
#pragma unroll
        for (int i = 0; i < D; ++i) dpos[i] = fmaf(__ldg(g + i), p.points_scaling, dpos[i]);
    }
    if (POS && active) {
        float* dst = a.positions_grad + n * D;
#pragma unroll
        for (int i = 0; i < D; ++i) red_add1(dst + i, dpos[i]);  // accumulates across passes
    }
}

// ------------------------------------------------------------------------------------------
// table gradient of a batch in spatial order: one level per thread, points one after the other
// ------------------------------------------------------------------------------------------
// A strand is a run of consecutive points of the ordered batch.  The levels of a sweep are dealt to consecutive
// threads; each walks the strand for its own level and keeps the sums of the D+1 vertices it is at in
// registers (a vertex keeps its remainder from one simplex to the next, which is where its sum is looked for).
// A sum goes to the table when the walk has left its vertex.  A warp reads a gradient row as whole sectors, and
// no lane has to look at another: with two points per thread and the lanes of a warp merged by match and
// shuffles (the kernel before) 40 % of the instructions were merging, and coarse and fine levels
// took turns at the two limits.  Here every warp carries all levels at all times.
//
// What bounds it: the rate of L2 reductions (pos_dim 3, 24 levels, 2^20 points: 44 M, 199 us at 220 G/s of 244, and
// 250 with the clearing of the table) and the integer and select pipe (75 % with two vertices kept; 174 M
// instructions with one, 200 M with two, 212 M before).  Records wait in shared memory because a load takes its turn
// behind the reductions: with records and rows requested one point ahead from memory 280 us, through a
// per-thread ring of asynchronous copies 310 (the copies themselves).  Before -> now, first order / second
// order / both in one, us: pos_dim 3, 24 levels, 2^19 points 174 / 185 / 229 -> 138 / 150 / 164, 2^20 points 306 / 327 ->
// 250 / 269, 2^22 1080 -> 917; 2^20 points and 16 levels of pos_dim 4 328 / 358 / 448 -> 241 / 267 / 304, of pos_dim 6
// 482 / 521 / 622 -> 425 / 480 / 523; 11 levels of 4 features 224 -> 157, 6 of 8 features 210 -> 189.  A warp of 4 levels
// and 8 strands, which can drop the sums on levels that share nothing, takes 228 at pos_dim 4 and 854 for 2^22
// points, but 144 for 2^19, 459 at pos_dim 6 and 213 with 8 features.
//
// What the table receives: the addends of the first-order backward, of the double backward, or their sum.
enum class Order { First, Second, Both };

constexpr int kStrandLength = 16;  // points of a strand, at least: 8 / 16 / 32 points, 2^19 points 169 / 147 / 163 us
// a block's points: what its shared memory holds where a sweep has few levels
constexpr int kStrandPoints = D <= 3 ? 2048 : 1024;
// Sums kept per remainder.  With TWO the vertex before the last one is kept too, which catches walks that go to
// and fro between neighbouring simplices: 10 to 14 % fewer reductions for a quarter more instructions.
constexpr int strand_live(int feats, bool two) { return (D + 1) * (feats + 1) * (two ? 2 : 1); }
constexpr int strand_left(int feats) { return (D + 1) * (feats + 1); }  // words a thread leaves at its strand's end
constexpr int strand_threads(int feats) { return strand_left(feats) * 4 * 256 <= 48 * 1024 ? 256 : 128; }  // of a block, at most
// warps per SM that the registers have to allow: the sums and their slots stay live over the walk
constexpr int strand_warps(int feats, bool two) {
    return strand_live(feats, two) <= 24 ? 32 : (strand_live(feats, two) <= 30 ? 24 : (strand_live(feats, two) <= 60 ? 16 : 12));
}
constexpr int kRecordVec = D <= 3 ? 1 : 2;  // float4s of a record

// With a position gradient in the same pass (F = 2): the entry of a vertex is gathered when the walk arrives at it, a
// thread leaves its level's part of a point's gradient in shared memory, and every kPosBatch points the block sums
// the parts over the levels.  The geometry of a point is worked out once for both gradients, and entries are
// gathered through the same walk (one_walk has the figures).  Bound like the table gradient alone, with the
// gathers in the queue of the reductions.
constexpr int kPosBatch = D <= 3 ? 8 : 4;
constexpr int pos_stage_words(int threads) { return kPosBatch * D * (threads + 1); }  // rows shifted by a bank

enum class Extra { None, Positions, PositionsHalf };  // Half: of an fp16 table
constexpr int strand_blocks(int feats, bool two, Extra extra) {
    return (extra == Extra::None ? strand_warps(feats, two) : (D <= 4 ? 24 : 16)) * 32 / strand_threads(feats);
}

template <int F, Order ORDER, bool TWO, Extra EXTRA>
__global__ void __launch_bounds__(strand_threads(F), strand_blocks(F, TWO, EXTRA))
scatter_strands_kernel(const CombinedArgs a) {
    constexpr bool kPos = EXTRA != Extra::None;
    constexpr bool kSecond = ORDER != Order::First;
    constexpr bool kBoth = ORDER == Order::Both;
    constexpr float kInv = 1.0f / (D + 1);
    constexpr uint32_t kNone = 0xffffffffu;  // no slot: capacities are below 2^31
    const Problem& p = a.p;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int pass_begin = p.level_begin + (int)blockIdx.y * p.levels_per_pass;
    const int levels = min(p.levels_per_pass, p.level_end - pass_begin);
    const int strands = (int)blockDim.x / levels;
    const int strand = (int)threadIdx.x / levels;
    const int l = pass_begin + (int)threadIdx.x - strand * levels;
    const int64_t block_first = (int64_t)blockIdx.x * a.points_per_block;
    const int block_points = (int)min((int64_t)a.points_per_block, p.n_points - block_first);
    const int each = (a.points_per_block + strands - 1) / strands;
    const int first = strand * each, last = min(first + each, block_points);
    const bool merge = a.aggregate != 0;
    float* gbase = a.lattice_grad + (size_t)l * p.capacity * F;

    // the block's records, and what else it needs of each point
    float4* record = reinterpret_cast<float4*>(smem_raw);
    float* dpgs = reinterpret_cast<float*>(record + kRecordVec * a.points_per_block);
    for (int i = threadIdx.x; i < block_points; i += blockDim.x) {
        float x[D];
        const int64_t n = load_point(p, block_first + i, x);
        float r[4 * kRecordVec];
#pragma unroll
        for (int j = 0; j < 4 * kRecordVec; ++j) r[j] = j < D ? x[j < D ? j : 0] : 0.f;
        r[4 * kRecordVec - 1] = __uint_as_float((uint32_t)n);
#pragma unroll
        for (int v = 0; v < kRecordVec; ++v) record[i * kRecordVec + v] = make_float4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
        if constexpr (kSecond) {
#pragma unroll
            for (int j = 0; j < D; ++j) dpgs[i * D + j] = __ldg(a.double_positions_grad + n * D + j);
        }
    }
    __syncthreads();

    uint32_t cur[D + 1];
    float acc[D + 1][F];
    float entry[kPos ? D + 1 : 1][F];
#pragma unroll
    for (int r = 0; r <= D; ++r) {
        cur[r] = kNone;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            acc[r][f] = 0.f;
            if (kPos) entry[kPos ? r : 0][f] = 0.f;
        }
    }
    // a closed level's addends are exact zeros
    const bool works = strand < strands && first < last && __ldg(p.anneal + l) != 0.0f;
    float* stage = reinterpret_cast<float*>(smem_raw) + kRecordVec * 4 * a.points_per_block;  // kPos
    const int pitch = (int)blockDim.x + 1;
    int batch = 0;
    if constexpr (kPos) {
        if (!works) {
            for (int k = 0; k < kPosBatch * D; ++k) stage[k * pitch + threadIdx.x] = 0.f;
        }
    }
    // the block's position gradients of points batch .. batch + kPosBatch of every strand
    auto sum_positions = [&]() {
        __syncthreads();
        for (int u = threadIdx.x; u < strands * kPosBatch * D; u += blockDim.x) {
            const int of = u % strands, k = u / strands;  // k = point of the batch * D + coordinate
            const int i = batch + k / D, at = of * each + i;
            if (i < each && at < block_points) {
                const float* src = stage + k * pitch + of * levels;
                float sum = 0.f;
                for (int j = 0; j < levels; ++j) sum += src[j];
                const int64_t n = (int64_t)__float_as_uint(record[at * kRecordVec + kRecordVec - 1].w);
                if (a.concat_grad && p.extra_levels > 0 && blockIdx.y == 0 && p.level_begin == 0)  // as in backward_kernel
                    sum = fmaf(__ldg(a.grad_features + n * p.width + F * p.nr_levels + k % D), p.points_scaling, sum);
                red_add1(a.positions_grad + n * D + k % D, sum);
            }
        }
        __syncthreads();
    };
    if (kPos || works) {
        const float* rows1 = (ORDER == Order::Second ? a.second_grad_features : a.grad_features) + F * l;
        const float* rows2 = a.second_grad_features + F * l;  // Both
        float next1[F], next2[kBoth ? F : 1];
        auto request = [&](int i) {  // the rows of a point, while the point before it is worked on
            const int64_t n = (int64_t)__float_as_uint(record[min(i, last - 1) * kRecordVec + kRecordVec - 1].w);
            load_feats<F>(rows1 + n * p.width, next1);
            if constexpr (kBoth) load_feats<F>(rows2 + n * p.width, next2);
        };
        LevelConst<D> lc;
        if (works) {
            request(first);
            lc.weight = __ldg(p.anneal + l);
#pragma unroll
            for (int i = 0; i < D; ++i) {
                lc.shift[i] = __ldg(p.shift + l * D + i);
                lc.scale[i] = __ldg(p.scale + l * D + i);
            }
            lc.reach = exact_reach<D>(p.shift + l * D, p.scale + l * D);
        }
        uint32_t old[TWO ? D + 1 : 1];
        float old_sum[TWO ? D + 1 : 1][F];
        if constexpr (TWO) {
#pragma unroll
            for (int r = 0; r <= D; ++r) {
                old[r] = kNone;
#pragma unroll
                for (int f = 0; f < F; ++f) old_sum[r][f] = 0.f;
            }
        }
        int i = first;
        do {
        const int end = !works ? first : (kPos ? min(first + batch + kPosBatch, last) : last);
#pragma unroll 1
        for (; i < end; ++i) {
            float g1[F], g2[kBoth ? F : 1];
#pragma unroll
            for (int f = 0; f < F; ++f) {
                g1[f] = next1[f];
                if (kBoth) g2[kBoth ? f : 0] = next2[kBoth ? f : 0];
            }
            request(i + 1);
            float v[4 * kRecordVec], x[D];
#pragma unroll
            for (int q = 0; q < kRecordVec; ++q) {
                const float4 t = record[i * kRecordVec + q];
                v[4 * q] = t.x;
                v[4 * q + 1] = t.y;
                v[4 * q + 2] = t.z;
                v[4 * q + 3] = t.w;
            }
#pragma unroll
            for (int j = 0; j < D; ++j) x[j] = v[j];
            Simplex<D> s;
            locate_simplex<D>(x, largest_coordinate<D>(x), lc, s);
            uint32_t slot[D + 1];
            to_slots(p, s, slot);
            to_remainders(s.s, slot);
            if constexpr (kPos) {
                // as in backward_kernel (EncodingGPU.cuh:671-749)
                float dB[D + 1];
#pragma unroll
                for (int r = 0; r <= D; ++r) {
                    if (slot[r] != cur[r]) gather<F, EXTRA == Extra::PositionsHalf>(p.table, l, p.capacity, slot[r], entry[kPos ? r : 0]);
                    float t = entry[kPos ? r : 0][0] * (g1[0] * lc.weight * kInv);
#pragma unroll
                    for (int f = 1; f < F; ++f) t = fmaf(entry[kPos ? r : 0][f], g1[f] * lc.weight * kInv, t);
                    dB[r] = t;
                }
                from_remainders(s.s, dB);
                float dE[D + 1];
#pragma unroll
                for (int k = 0; k <= D; ++k) dE[k] = dB[D - k] - dB[k == 0 ? 0 : D + 1 - k];
                to_coordinates(s, dE);
                float* dst = stage + (i - first - batch) * D * pitch + threadIdx.x;
                float run = 0.f;
#pragma unroll
                for (int j = 0; j < D; ++j) {
                    run += dE[j];
                    dst[j * pitch] = lc.scale[j] * (run - (float)(j + 1) * dE[j + 1]);
                }
            }
            float w1[D + 1], w2[kBoth ? D + 1 : 1], dpg[kSecond ? D : 1];
            if constexpr (kSecond) {
#pragma unroll
                for (int j = 0; j < D; ++j) dpg[j] = dpgs[i * D + j];
            }
            if constexpr (ORDER != Order::Second)
                vertex_weights<D>(s, lc.weight * kInv, w1);
            else
                second_order_weights(s, lc, dpg, w1);
            to_remainders(s.s, w1);
            if constexpr (kBoth) {
                second_order_weights(s, lc, dpg, w2);
                to_remainders(s.s, w2);
            }
#pragma unroll
            for (int r = 0; r <= D; ++r) {
                const bool same = merge && slot[r] == cur[r];
                float sum[F];
                if constexpr (TWO) {
                    const bool back = merge && slot[r] == old[r];
                    if (!same && !back && old[r] != kNone) red_add<F>(gbase, old[r], old_sum[r]);
#pragma unroll
                    for (int f = 0; f < F; ++f) {
                        sum[f] = same ? acc[r][f] : (back ? old_sum[r][f] : 0.f);
                        old_sum[r][f] = same ? old_sum[r][f] : acc[r][f];
                    }
                    old[r] = same ? old[r] : cur[r];
                } else {
                    if (!same && i > first) red_add<F>(gbase, cur[r], acc[r]);
#pragma unroll
                    for (int f = 0; f < F; ++f) sum[f] = same ? acc[r][f] : 0.f;
                }
                cur[r] = slot[r];
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    acc[r][f] = fmaf(w1[r], g1[f], sum[f]);
                    if constexpr (kBoth) acc[r][f] = fmaf(w2[r], g2[f], acc[r][f]);
                }
            }
        }
        if constexpr (kPos) {
            sum_positions();
            batch += kPosBatch;
        }
        } while (kPos && batch < each);
        if constexpr (TWO) {
#pragma unroll
            for (int r = 0; r <= D; ++r)
                if (old[r] != kNone) red_add<F>(gbase, old[r], old_sum[r]);
        }
    }

    // Neighbouring strands end at the same vertices on coarse levels, whose few slots take one reduction per
    // 4 ns each: what the strands are left with is summed along the block first.
    uint32_t* left_slot = reinterpret_cast<uint32_t*>(smem_raw);                   // [vertex][thread]
    float* left_sum = reinterpret_cast<float*>(left_slot + (D + 1) * blockDim.x);  // [vertex][feature][thread]
    __syncthreads();  // the records are done with
#pragma unroll
    for (int r = 0; r <= D; ++r) {
        left_slot[r * blockDim.x + threadIdx.x] = cur[r];
#pragma unroll
        for (int f = 0; f < F; ++f) left_sum[(r * F + f) * blockDim.x + threadIdx.x] = acc[r][f];
    }
    __syncthreads();
    if (strand >= strands) return;
    for (int r = strand; r <= D; r += strands) {
        uint32_t at = kNone;
        float sum[F];
        for (int j = (int)threadIdx.x - strand * levels; j < strands * levels; j += levels) {
            const uint32_t slot = left_slot[r * blockDim.x + j];
            if (slot == kNone) continue;
            const bool same = merge && slot == at;
            if (!same && at != kNone) red_add<F>(gbase, at, sum);
            at = slot;
#pragma unroll
            for (int f = 0; f < F; ++f) sum[f] = left_sum[(r * F + f) * blockDim.x + j] + (same ? sum[f] : 0.f);
        }
        if (at != kNone) red_add<F>(gbase, at, sum);
    }
}

// ------------------------------------------------------------------------------------------
// double backward of the position gradient
// ------------------------------------------------------------------------------------------
template <int F, int LPS, bool TABLE, bool GGF, bool HALF, bool SHIFTED>
__global__ void __launch_bounds__(kThreads, min_blocks(F, false)) double_backward_kernel(const DoubleBackwardArgs a) {
    const Problem& p = a.p;
    __shared__ __align__(16) float levels[kStage * kRecord];
    const int64_t i_raw = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool active = i_raw < p.n_points;
    const int pass_begin = p.level_begin + (int)blockIdx.y * p.levels_per_pass;
    const int pass_end = min(pass_begin + p.levels_per_pass, p.level_end);
    const unsigned lane = threadIdx.x & 31u;

    float pos[D], dpg[D];
    const int64_t n = load_point(p, active ? i_raw : p.n_points - 1, pos);
    const float largest = largest_coordinate<D>(pos);
#pragma unroll
    for (int i = 0; i < D; ++i) dpg[i] = __ldg(a.double_positions_grad + n * D + i);
    Scatter sc{lane, active, a.aggregate != 0};  // as in backward_kernel
    ShiftedRow row(a.grad_grad_features + n * p.width + F * pass_begin);  // used by SHIFTED only, as in forward_kernel

#pragma unroll 1
    for (int begin = pass_begin; begin < pass_end; begin += kStage) {
        const int end = min(begin + kStage, pass_end);
        const int nsteps = (end - begin + LPS - 1) / LPS;
        int step = (TABLE && kStagger) ? (int)(blockIdx.x % (unsigned)nsteps) : 0;
        float g_next[F * LPS];  // as in backward_kernel: the next step's gradient segment is requested early
        if (TABLE) load_row_segment<F, LPS>(p, a.grad_features, n, begin + step * LPS, g_next);
        if (begin != pass_begin) __syncthreads();
        stage_levels(p, begin, end, levels);
        __syncthreads();
#pragma unroll 1
        for (int it = 0; it < nsteps; ++it) {
            const int l0 = begin + step * LPS;
            step = (step + 1 == nsteps) ? 0 : step + 1;
            if (TABLE && l0 == begin) sc.probe = a.aggregate != 0;
            float g[F * LPS];
            if (TABLE) {
#pragma unroll
                for (int i = 0; i < F * LPS; ++i) g[i] = g_next[i];
                if (it + 1 < nsteps) load_row_segment<F, LPS>(p, a.grad_features, n, begin + step * LPS, g_next);
            }
            float out[F * LPS];
#pragma unroll
            for (int k = 0; k < LPS; ++k) {
                const int l = l0 + k;
                float o[F];
#pragma unroll
                for (int f = 0; f < F; ++f) o[f] = 0.f;
                if (l < end) {
                    LevelConst<D> lc;
                    load_level(levels, l - begin, lc);
                    if (lc.weight != 0.0f) {
                        Simplex<D> s;
                        locate_simplex<D>(pos, largest, lc, s);
                        uint32_t slot[D + 1];
                        to_slots(p, s, slot);

                        float dBw[D + 1];
                        second_order_weights(s, lc, dpg, dBw);

                        if (GGF) {
#pragma unroll
                            for (int q = 0; q <= D; ++q) {
                                float v[F];
                                gather<F, HALF>(p.table, l, p.capacity, slot[q], v);  // EncodingGPU.cuh:1484-1485
#pragma unroll
                                for (int f = 0; f < F; ++f) o[f] = fmaf(dBw[q], v[f], o[f]);
                            }
                        }
                        if (TABLE) {  // EncodingGPU.cuh:1244-1245
                            float* gbase = a.lattice_grad + (size_t)l * p.capacity * F;
                            float gk[F];
#pragma unroll
                            for (int f = 0; f < F; ++f) gk[f] = g[F * k + f];
                            scatter_level<F>(sc, gbase, s.s, slot, dBw, gk);
                        }
                    }
                }
#pragma unroll
                for (int f = 0; f < F; ++f) out[F * k + f] = o[f];
            }
            if (SHIFTED) {
                if (active) row.push(reinterpret_cast<const float(&)[8]>(out), F * min(LPS, end - l0));
            } else if (GGF && active) {
                store_row_segment<F, LPS>(p, a.grad_grad_features, n, l0, out);
            }
        }
    }
    if (SHIFTED && active) row.finish();
    if (GGF && active && p.extra_levels > 0 && blockIdx.y == 0 && p.level_begin == 0) {  // EncodingGPU.cuh:1290-1295
        float* dst = a.grad_grad_features + n * p.width + F * p.nr_levels;
        for (int c = 0; c < F * p.extra_levels; ++c) dst[c] = 0.f;
    }
}

// ------------------------------------------------------------------------------------------
// debug view: one thread per (point, level)
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) debug_kernel(const DebugArgs a) {
    const Problem& p = a.p;
    const int64_t n = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (n >= p.n_points) return;
    const int l = blockIdx.y;
    float pos[D];
    load_pos(p, n, pos);
    LevelConst<D> lc;
    lc.weight = 1.0f;
    lc.reach = exact_reach<D>(p.shift + l * D, p.scale + l * D);
    const float largest = largest_coordinate<D>(pos);
#pragma unroll
    for (int i = 0; i < D; ++i) {
        lc.shift[i] = __ldg(p.shift + l * D + i);
        lc.scale[i] = __ldg(p.scale + l * D + i);
    }
    Simplex<D> s;
    locate_simplex<D>(pos, largest, lc, s);
    uint32_t slot[D + 1];
    to_slots(p, s, slot);
    float w[D + 1];
    vertex_weights<D>(s, 1.0f / (D + 1), w);
    to_remainders(s.s, slot);
    to_remainders(s.s, w);
    int k[D + 1];  // rank of every coordinate before the wrap
#pragma unroll
    for (int i = 0; i <= D; ++i) k[i] = i;
    to_coordinates(s, k);
    const int64_t base = (n * p.nr_levels + l) * (D + 1);
    int q = s.s < 0 ? s.s + D + 1 : s.s;  // vertex of remainder 0
#pragma unroll
    for (int r = 0; r <= D; ++r) {
        if (a.keys) {
#pragma unroll
            for (int i = 0; i < D; ++i) a.keys[(base + r) * D + i] = s.lift[i] + q - (k[i] > D - q ? D + 1 : 0);
        }
        if (a.slots) a.slots[base + r] = (int32_t)slot[r];
        if (a.bary) a.bary[base + r] = w[r];
        if (a.rank) {
            const int wrapped = k[r] + s.s;
            a.rank[base + r] = wrapped < 0 ? wrapped + D + 1 : (wrapped > D ? wrapped - (D + 1) : wrapped);
        }
        q = q == D ? 0 : q + 1;
    }
}

// Levels handled by one thread in one sweep over the points.  A multiple of the levels per step
// (one 32-byte row segment per step).  More levels per pass means fewer sweeps -- each sweep
// re-reads the positions and touches only its own 32-byte pieces of every 128-byte line of the
// feature rows, which costs a 4x DRAM over-fetch on the gradient reads with one step per sweep
// -- but a larger set of table slices is live in L2 at once: capacity * 4F bytes per level for
// the values and as much again for their gradient.  Measured on B200 (pos_dim 3, 4 and 6,
// capacities 2^18..2^20, F = 2): scatter-only kernels are fastest with every level in one sweep
// up to a gradient table of about 100 MB; gather kernels, and scatter kernels beyond that, with
// two sweeps, the finest third of the levels in the second; gather+scatter kernels with about
// 64 MB live.
enum class Traffic { Gather, Scatter, Both };

inline int pick_levels_per_pass(const Problem& p, int requested, Traffic t, int lps) {
    const int levels = p.level_end - p.level_begin;
    int lpp = requested;
    if (lpp <= 0 && p.order != nullptr) {
        lpp = levels;  // neighbouring points share their lines: nothing to split (pos_dim 3, 2^20 points: 201 us, two sweeps 224)
    } else if (lpp <= 0) {
        const double slice = (p.table_half ? 2.0 : 4.0) * p.nr_feat * p.capacity;
        const double mb = 1024.0 * 1024.0;
        if (t == Traffic::Scatter) {
            // one sweep while the fp32 gradient table is within reach of L2 (measured up to the
            // 100.7 MB of capacity 2^19 x 24 levels); beyond that the same two sweeps as the gather
            // kernels (capacity 2^20 x 24 levels, 201 MB: 1.05 ms against 1.84 in one sweep)
            const double gslice = 4.0 * p.nr_feat * p.capacity;
            if (gslice * levels <= 128.0 * mb) {
                lpp = levels;
            } else {
                lpp = ((2 * levels + 2) / 3 + lps - 1) / lps * lps;
                const int cap = (int)(128.0 * mb / gslice);
                if (lpp > cap) lpp = cap;
            }
        }
        else if (t == Traffic::Gather) {
            // Coarse levels touch few slots whatever the capacity; what must fit in L2 together
            // is the saturated, fine levels of a pass.  Two passes with the finest third of the
            // levels in the second one measured best from capacity 2^18 to 2^20 (forward at 2^20 and
            // 24 levels: 0.70 ms against 0.91 with two equal passes and 0.93 with one); tables of a
            // few MB stay in one pass, very large slices are capped at 128 MB per pass.
            if (slice * levels <= 32.0 * mb) {
                lpp = levels;
            } else {
                lpp = ((2 * levels + 2) / 3 + lps - 1) / lps * lps;
                const int cap = (int)(128.0 * mb / slice);
                if (lpp > cap) lpp = cap;
            }
        }
        else
            lpp = (int)(64.0 * mb / (slice + 4.0 * p.nr_feat * p.capacity));  // values + their fp32 gradient
    }
    lpp = (lpp / lps) * lps;
    if (lpp < lps) lpp = lps;
    if (lpp > levels) lpp = ((levels + lps - 1) / lps) * lps;
    return lpp;
}

inline dim3 grid_for(const Problem& p) {
    const unsigned gx = (unsigned)((p.n_points + kThreads - 1) / kThreads);
    const unsigned gy = (unsigned)((p.level_end - p.level_begin + p.levels_per_pass - 1) / p.levels_per_pass);
    return dim3(gx, gy, 1);
}

// small problems get one level per thread and pass so that the grid still covers the machine
inline bool use_single_level(const Problem& p) {
    const int lps = 8 / p.nr_feat;
    const int64_t steps = (p.level_end - p.level_begin + lps - 1) / lps;
    const int64_t blocks = ((p.n_points + kThreads - 1) / kThreads) * steps;
    const int sms = sm_count();
    return lps > 1 && blocks < 2 * (sms > 0 ? sms : 148);
}


// A batch with fewer than two blocks of 256 points per multiprocessor has its levels split over more
// blocks, as far as whole steps go (2^14 points: table gradient 31 -> 25 us, forward 12.7 -> 10.7).
// Aiming for a full wave instead makes 2^15 and 2^16 points slower (position gradient 16.7 -> 20.8 us).
inline int spread_levels(const Problem& p, int lpp, int lps) {
    const int levels = p.level_end - p.level_begin;
    const int64_t points = (p.n_points + kThreads - 1) / kThreads;
    const int64_t passes = 2 * sm_count() / points;
    const int steps = (levels + lps - 1) / lps;
    if (passes <= 1) return lpp;
    const int each = (int)((steps + passes - 1) / passes) * lps;
    return each < lpp ? each : lpp;
}

template <class Args>
inline Args with_schedule(const Args& in, bool single, Traffic t) {
    Args a = in;
    const int lps = 8 / a.p.nr_feat;
    if (single) {
        a.p.levels_per_pass = 1;
    } else {
        const int requested = a.p.levels_per_pass;
        a.p.levels_per_pass = pick_levels_per_pass(a.p, requested, t, lps);
        if (requested <= 0) a.p.levels_per_pass = spread_levels(a.p, a.p.levels_per_pass, lps);
    }
    return a;
}

template <int F, int LPS, bool SHIFTED>
cudaError_t launch_forward_rows(const ForwardArgs& a, cudaStream_t st) {
    if (a.p.table_half)
        forward_kernel<F, LPS, true, SHIFTED><<<grid_for(a.p), kThreads, 0, st>>>(a);
    else
        forward_kernel<F, LPS, false, SHIFTED><<<grid_for(a.p), kThreads, 0, st>>>(a);
    return cudaGetLastError();
}
template <int F, int LPS>
cudaError_t launch_forward(const ForwardArgs& a, cudaStream_t st) {
    if constexpr (F * LPS == 8 && F < 8)
        if (!a.p.rows_vec8_ok) return launch_forward_rows<F, LPS, true>(a, st);
    return launch_forward_rows<F, LPS, false>(a, st);
}

template <int F, int LPS>
cudaError_t launch_forward_linear(const ForwardLinearArgs& in, cudaStream_t st) {
    ForwardLinearArgs a = in;
    size_t smem = (size_t)kRing * kSliceBytes + (size_t)a.layer[0].out_features * a.k_pad * sizeof(float);
    int hmax = 0;  // widest hidden layer
    for (int i = 1; i < a.nr_layers; ++i) {
        if (a.layer[i].in_features > hmax) hmax = a.layer[i].in_features;
        if (a.layer[i].out_features % 16 == 0) smem += (size_t)a.layer[i].out_features * a.layer[i].in_features * sizeof(float);
    }
    a.levels_offset = (int32_t)smem;
    smem += (size_t)a.p.nr_levels * kRecord * sizeof(float);
    for (int i = 0; i < a.nr_layers; ++i) smem += (size_t)(a.layer[i].out_features + 3) / 4 * 4 * sizeof(float);
    const MlpLayer& tail = a.layer[a.nr_layers - 1];
    if (tail.out_features % 16 != 0) smem += (size_t)tail.out_features * tail.in_features * sizeof(float);
    // as many blocks as an SM holds (launch bounds, shared and tensor memory), each walking over several tiles
    const int64_t tiles = (a.p.n_points + kTileRows - 1) / kTileRows;
    const int fits = (int)((size_t)(227 * 1024) / (smem + 2048));
    const int resident = min(min(fused_blocks(F, hmax), 512 / a.tmem_cols), fits > 0 ? fits : 1);
    const int64_t blocks = min(tiles, (int64_t)max(sm_count(), 1) * resident);
    const dim3 g((unsigned)blocks);
    auto launch = [&](auto kernel) -> cudaError_t {
        if (smem + 1024 > 48 * 1024) {  // the kernel's few static shared words count against the default limit
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
        kernel<<<g, kTileRows, smem, st>>>(a);
        return cudaGetLastError();
    };
    const bool h = a.p.table_half != 0;
    if (a.nr_layers == 1) return h ? launch(forward_mlp_kernel<F, LPS, true, 0>) : launch(forward_mlp_kernel<F, LPS, false, 0>);
    if (hmax <= 32) return h ? launch(forward_mlp_kernel<F, LPS, true, 32>) : launch(forward_mlp_kernel<F, LPS, false, 32>);
    return h ? launch(forward_mlp_kernel<F, LPS, true, 64>) : launch(forward_mlp_kernel<F, LPS, false, 64>);
}

// The table is only read where something is gathered (position gradient, grad-grad features):
// the scatter-only kernels have no fp16 variant.
template <int F, int LPS>
cudaError_t launch_backward(const BackwardArgs& a, cudaStream_t st) {
    const dim3 g = grid_for(a.p);
    const bool h = a.p.table_half != 0;
    if (a.lattice_grad && a.positions_grad) {
        if (h) backward_kernel<F, LPS, true, true, true><<<g, kThreads, 0, st>>>(a);
        else backward_kernel<F, LPS, true, true, false><<<g, kThreads, 0, st>>>(a);
    } else if (a.lattice_grad) {
        backward_kernel<F, LPS, true, false, false><<<g, kThreads, 0, st>>>(a);
    } else if (a.positions_grad) {
        if (h) backward_kernel<F, LPS, false, true, true><<<g, kThreads, 0, st>>>(a);
        else backward_kernel<F, LPS, false, true, false><<<g, kThreads, 0, st>>>(a);
    }
    return cudaGetLastError();
}

template <int F, int LPS>
cudaError_t launch_double(const DoubleBackwardArgs& a, cudaStream_t st) {
    const dim3 g = grid_for(a.p);
    const bool h = a.p.table_half != 0;
    if (a.lattice_grad && a.grad_grad_features) {
        if (h) double_backward_kernel<F, LPS, true, true, true, false><<<g, kThreads, 0, st>>>(a);
        else double_backward_kernel<F, LPS, true, true, false, false><<<g, kThreads, 0, st>>>(a);
    } else if (a.lattice_grad) {
        double_backward_kernel<F, LPS, true, false, false, false><<<g, kThreads, 0, st>>>(a);
    } else if (a.grad_grad_features) {
        if constexpr (F * LPS == 8 && F < 8) {
            if (!a.p.rows_vec8_ok) {
                if (h) double_backward_kernel<F, LPS, false, true, true, true><<<g, kThreads, 0, st>>>(a);
                else double_backward_kernel<F, LPS, false, true, false, true><<<g, kThreads, 0, st>>>(a);
                return cudaGetLastError();
            }
        }
        if (h) double_backward_kernel<F, LPS, false, true, true, false><<<g, kThreads, 0, st>>>(a);
        else double_backward_kernel<F, LPS, false, true, false, false><<<g, kThreads, 0, st>>>(a);
    }
    return cudaGetLastError();
}

// Two vertices per remainder (F = 2) where reductions are what there is too much of: the more dimensions, the
// more vertices a walk comes back to, and the more points, the fewer it leaves.  us, one -> two, at 2^18 / 2^19 / 2^20
// / 2^21 points: pos_dim 2 64 -> 69 / 102 -> 112 / 188 -> 206 / 351 -> 388; 3 95 -> 87 / 146 -> 138 / 261 -> 249 / 479 -> 472; 4 120 -> 99 /
// 161 -> 148 / 241 -> 254 / 417 -> 462; 5 165 -> 130 / 221 -> 200 / 363 -> 344 / 612 -> 628; 6 202 -> 163 / 294 -> 254 / 480 -> 425 /
// 863 -> 767; 7 242 -> 186 / 348 -> 299 / 609 -> 512 / 1079 -> 917.  Second order: 3 97 -> 89 / 150 -> 151 / 269 -> 288; 5 166 -> 139 / 231 ->
// 220 / 380 -> 394; others as first order.
template <Order ORDER>
bool keep_two_vertices(int64_t points) {
    constexpr bool kFirst = ORDER == Order::First;
    switch (D) {
        case 2: return false;
        case 3: return kFirst || points < 3 << 17;
        case 4: return points < 3 << 18;
        case 5: return points < (kFirst ? 3 << 19 : 3 << 18);
        default: return true;
    }
}

template <int F, Order ORDER, bool TWO, Extra EXTRA = Extra::None>
cudaError_t launch_strands(const CombinedArgs& in, cudaStream_t st) {
    CombinedArgs a = in;
    const int levels = a.p.level_end - a.p.level_begin;
    // One sweep, but two, the finest third of the levels in the second, of tables beyond 144 MB at pos_dim 5 and more,
    // where most levels fill their slices: pos_dim 5, 24 levels of 2^20 entries, 2^19 points 763 -> 395 us, pos_dim 6, 20
    // levels, 2^20 points 788 -> 595; pos_dim 6 with 134 MB 476 -> 489, and pos_dim 2 to 4 with 201 MB and coarser levels
    // 218 -> 256 and 263 -> 294 (filled ones 576 -> 421).
    const bool two_sweeps = D >= 5 && F == 2 && (double)levels * a.p.capacity * 4 * F > 144.0 * 1024 * 1024;
    const int whole = two_sweeps ? (2 * levels + 2) / 3 : levels;
    const int lpp = min(a.p.levels_per_pass > 0 ? min(a.p.levels_per_pass, levels) : whole, strand_threads(F));
    a.p.levels_per_pass = lpp;
    // the levels of a sweep are dealt to threads: the largest block among those that leave the fewest idle
    int threads = (lpp + 31) / 32 * 32;
    for (int t = threads; t <= strand_threads(F); t += 32)
        if (t / lpp * threads >= threads / lpp * t) threads = t;
    const int strands = threads / lpp;
    // whole waves of resident blocks, as many as strands of the least length allow
    const int64_t resident = (int64_t)max(sm_count(), 1) * max(strand_blocks(F, TWO, EXTRA) * strand_threads(F) / threads, 1);
    const int64_t waves = max((int64_t)1, a.p.n_points / (resident * strands * kStrandLength));
    a.points_per_block = (int32_t)min((int64_t)kStrandPoints, (a.p.n_points + resident * waves - 1) / (resident * waves));
    const dim3 g((unsigned)((a.p.n_points + a.points_per_block - 1) / a.points_per_block), (unsigned)((levels + lpp - 1) / lpp));
    const int point_words = 4 * kRecordVec + (ORDER != Order::First ? D : 0);
    const int stage_words = EXTRA == Extra::None ? 0 : pos_stage_words(threads);
    const int smem = max(strand_left(F) * threads, point_words * a.points_per_block + stage_words) * (int)sizeof(float);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(scatter_strands_kernel<F, ORDER, TWO, EXTRA>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    scatter_strands_kernel<F, ORDER, TWO, EXTRA><<<g, threads, smem, st>>>(a);
    return cudaGetLastError();
}
template <Order ORDER>
cudaError_t launch_strands_by_width(const CombinedArgs& a, cudaStream_t st) {
    switch (a.p.nr_feat) {
        case 2: return keep_two_vertices<ORDER>(a.p.n_points) ? launch_strands<2, ORDER, true>(a, st) : launch_strands<2, ORDER, false>(a, st);
        case 4: return launch_strands<4, ORDER, false>(a, st);
        case 8: return launch_strands<8, ORDER, false>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

// feature width and step size are compile-time: pick the instantiation
#define PERMUTO_BY_WIDTH(fn, a, single, st)                                              \
    switch ((a).p.nr_feat) {                                                             \
        case 2: return (single) ? fn<2, 1>(a, st) : fn<2, 4>(a, st);                     \
        case 4: return (single) ? fn<4, 1>(a, st) : fn<4, 2>(a, st);                     \
        case 8: return fn<8, 1>(a, st);                                                  \
        default: return cudaErrorInvalidValue;                                           \
    }

}  // namespace

#define PERMUTO_CAT_(a, b) a##b
#define PERMUTO_CAT(a, b) PERMUTO_CAT_(a, b)

cudaError_t PERMUTO_CAT(launch_forward_dim, PERMUTO_DIM)(const ForwardArgs& a0, cudaStream_t st) {
    const bool single = use_single_level(a0.p);
    const ForwardArgs a = with_schedule(a0, single, Traffic::Gather);
    PERMUTO_BY_WIDTH(launch_forward, a, single, st)
}

cudaError_t PERMUTO_CAT(launch_forward_linear_dim, PERMUTO_DIM)(const ForwardLinearArgs& a, cudaStream_t st) {
    switch (a.p.nr_feat) {  // always whole 8-float steps: the tile is padded, not the level loop
        case 2: return launch_forward_linear<2, 4>(a, st);
        case 4: return launch_forward_linear<4, 2>(a, st);
        case 8: return launch_forward_linear<8, 1>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

// Both gradients in one walk: two features, pos_dim 2 and 3 (with more dimensions a thread's registers hold too
// little), and values and gradient of a sweep within reach of L2 together -- a gather that misses waits behind
// the reductions.  us, two launches -> one, at 2^18 / 2^19 / 2^20 / 2^21 points: pos_dim 2 123 -> 99 / 193 -> 167 / 338 -> 310 /
// 635 -> 585; 3 167 -> 142 / 267 -> 245 / 471 -> 443 / 887 -> 826; 4 145 -> 138 / 242 -> 245 / 420 -> 456 / 773 -> 869; 6 219 -> 217 / 390 ->
// 399 / 732 -> 777; pos_dim 3 with tables of 201 MB 320 -> 427 / 504 -> 718 / 876 -> 1248.
inline bool one_walk(const Problem& p) {
    const double slice = ((p.table_half ? 2.0 : 4.0) + 4.0) * p.nr_feat * p.capacity;
    return D <= 3 && p.nr_feat == 2 && slice * (p.level_end - p.level_begin) <= 112.0 * 1024 * 1024;
}

// Else a batch in spatial order takes its table gradient and what it gathers in two launches: the scatter has
// a kernel of its own, and the gather alone runs with more warps per SM.
cudaError_t PERMUTO_CAT(launch_backward_dim, PERMUTO_DIM)(const BackwardArgs& a0, cudaStream_t st) {
    BackwardArgs in = a0;
    if constexpr (D <= 3) {
        if (in.p.order && in.lattice_grad && in.positions_grad && one_walk(in.p)) {
            CombinedArgs r{in.p, in.grad_features, nullptr, nullptr, in.lattice_grad, in.aggregate};
            r.positions_grad = in.positions_grad;
            r.concat_grad = in.concat_grad;
            return in.p.table_half ? launch_strands<2, Order::First, false, Extra::PositionsHalf>(r, st)
                                   : launch_strands<2, Order::First, false, Extra::Positions>(r, st);
        }
    }
    if (in.p.order && in.lattice_grad) {
        const CombinedArgs r{in.p, in.grad_features, nullptr, nullptr, in.lattice_grad, in.aggregate};
        const cudaError_t e = launch_strands_by_width<Order::First>(r, st);
        if (e != cudaSuccess || !in.positions_grad) return e;
        in.lattice_grad = nullptr;
    }
    const bool single = use_single_level(in.p);
    const Traffic t = (in.lattice_grad && in.positions_grad) ? Traffic::Both
                                                             : (in.lattice_grad ? Traffic::Scatter : Traffic::Gather);
    const BackwardArgs a = with_schedule(in, single, t);
    PERMUTO_BY_WIDTH(launch_backward, a, single, st)
}

cudaError_t PERMUTO_CAT(launch_double_backward_dim, PERMUTO_DIM)(const DoubleBackwardArgs& a0, cudaStream_t st) {
    DoubleBackwardArgs in = a0;
    if (in.p.order && in.lattice_grad) {
        const CombinedArgs r{in.p, nullptr, in.double_positions_grad, in.grad_features, in.lattice_grad, in.aggregate};
        const cudaError_t e = launch_strands_by_width<Order::Second>(r, st);
        if (e != cudaSuccess || !in.grad_grad_features) return e;
        in.lattice_grad = nullptr;
    }
    const bool single = use_single_level(in.p);
    const Traffic t = (in.lattice_grad && in.grad_grad_features)
                          ? Traffic::Both
                          : (in.lattice_grad ? Traffic::Scatter : Traffic::Gather);
    const DoubleBackwardArgs a = with_schedule(in, single, t);
    PERMUTO_BY_WIDTH(launch_double, a, single, st)
}

cudaError_t PERMUTO_CAT(launch_combined_dim, PERMUTO_DIM)(const CombinedArgs& a, cudaStream_t st) {
    if (a.p.order) return launch_strands_by_width<Order::Both>(a, st);
    // small batches: two launches onto the same table
    const BackwardArgs first{a.p, a.grad_features, a.lattice_grad, nullptr, a.aggregate, 0};
    const cudaError_t e = PERMUTO_CAT(launch_backward_dim, PERMUTO_DIM)(first, st);
    if (e != cudaSuccess) return e;
    const DoubleBackwardArgs second{a.p, a.double_positions_grad, a.second_grad_features, a.lattice_grad, nullptr, a.aggregate};
    return PERMUTO_CAT(launch_double_backward_dim, PERMUTO_DIM)(second, st);
}

cudaError_t PERMUTO_CAT(launch_debug_dim, PERMUTO_DIM)(const DebugArgs& a, cudaStream_t st) {
    const dim3 g((unsigned)((a.p.n_points + kThreads - 1) / kThreads), (unsigned)a.p.nr_levels, 1);
    debug_kernel<<<g, kThreads, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace permuto
