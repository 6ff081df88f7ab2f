// Per-(point, level) geometry of the permutohedral lattice: elevate, find the enclosing
// simplex, barycentric weights, hash the d+1 vertex keys.
//
// Behaviour follows kernels/permutohedral_encoding/EncodingGPU.cuh:130-223 and :22-45 of the
// reference (paths relative to its project root): the integer results (remainder-0 point,
// ranks, keys, slots) are bit-identical to it; the barycentric weights agree to fp32 rounding
// (about 1e-7 absolute) but not bit for bit.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace permuto {

constexpr uint32_t kHashMul = 2531011u;  // EncodingGPU.cuh:29

// M^e mod 2^32
__host__ __device__ constexpr uint32_t hash_pow(int e) {
    uint32_t r = 1u;
    for (int i = 0; i < e; ++i) r *= kHashMul;
    return r;
}

// sum of the hash powers of the d key coordinates: what adding 1 to every coordinate adds to the hash
template <int D>
__host__ __device__ constexpr uint32_t hash_all() {
    uint32_t r = 0u;
    for (int i = 0; i < D; ++i) r += hash_pow(D - i);
    return r;
}

// Hash step of coordinate i: walking from vertex q-1 to vertex q of the simplex adds 1 to every
// coordinate and takes D+1 off one of them, and the hash is linear over Z/2^32.
template <int D>
__host__ __device__ constexpr uint32_t hash_step(int i) {
    return hash_all<D>() - (i < D ? (uint32_t)(D + 1) * hash_pow(D - i) : 0u);
}

// One level's constants.
template <int D>
struct LevelConst {
    float weight;
    float shift[D];
    float scale[D];
    float reach;  // points with every |coordinate| below it elevate to less than 2^22 (exact_reach)
};

// Largest coordinate for which every elevated coordinate of the level stays below 2^22:
// |e_i| <= sum_j j * scale_j * (|pos_j| + |shift_j|), j = 1..D, with a margin for the roundings.
// Testing a point's largest coordinate once against this replaces D+1 maxima per level.
template <int D>
__device__ __forceinline__ float exact_reach(const float* __restrict__ shift, const float* __restrict__ scale) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int j = 1; j <= D; ++j) {
        const float s = (float)j * fabsf(__ldg(scale + j - 1));
        a += s;
        b = fmaf(s, fabsf(__ldg(shift + j - 1)), b);
    }
    return (4194304.0f * 0.9999f - b) / a;  // negative or NaN: no point qualifies
}

template <int D>
__device__ __forceinline__ float largest_coordinate(const float (&pos)[D]) {
    float r = 0.f;
#pragma unroll
    for (int i = 0; i < D; ++i) r = fmaxf(r, fabsf(pos[i]));
    return r;
}

// The simplex around a point, its vertices numbered q = 0..D along the walk that leaves the
// *unwrapped* nearest remainder-0 point:
//     key_q[i] = R_i - s + q - (D+1) * [k_i > D - q],   s = sum(R) / (D+1)
// with k_i the descending rank of coordinate i's residual.  The reference first shifts the ranks by
// s, wraps them back into 0..D and corrects R accordingly (.cuh:177-186); that only renumbers the
// same D+1 vertices cyclically (its remainder r is q - s modulo D+1), so nothing that sums over the
// vertices needs the wrap, and the weight of vertex q is the gap between neighbouring residuals
// whichever way they are numbered.
template <int D>
struct Simplex {
    float x[D + 1];     // residuals e - R in descending order (units of the elevated space)
    uint32_t step[D + 1];  // hash steps in the same order
    uint32_t hash0;     // hash of vertex 0, before the modulo
    int s;              // sum(R) / (D+1); only computed where it is used
    int lift[D + 1];    // R_i - s (debug view)
    bool swapped[(D + 1) * D / 2];  // outcome of every comparator of the sorting network
};

// Adjacent comparators of an odd-even transposition network (D+1 stages, (D+1)D/2 comparators).
// Only neighbours are exchanged and only on strict inequality, so equal residuals keep their order:
// a tie raises the later index's rank, as .cuh:166-173 has it.
template <int D, class F>
__device__ __forceinline__ void for_each_comparator(F&& f) {
    int c = 0;
#pragma unroll
    for (int stage = 0; stage <= D; ++stage) {
#pragma unroll
        for (int i = stage & 1; i < D; i += 2) f(c++, i);
    }
}
template <int D, class F>
__device__ __forceinline__ void for_each_comparator_reversed(F&& f) {
    int c = (D + 1) * D / 2;
#pragma unroll
    for (int stage = D; stage >= 0; --stage) {
#pragma unroll
        for (int i = D - 1; i >= 0; --i)
            if ((i & 1) == (stage & 1)) f(--c, i);
    }
}

// order by rank -> order by coordinate (runs the network backwards)
template <int D, class T>
__device__ __forceinline__ void to_coordinates(const Simplex<D>& s, T (&v)[D + 1]) {
    for_each_comparator_reversed<D>([&](int c, int i) {
        const T a = v[i], b = v[i + 1];
        v[i] = s.swapped[c] ? b : a;
        v[i + 1] = s.swapped[c] ? a : b;
    });
}
// order by coordinate -> order by rank
template <int D, class T>
__device__ __forceinline__ void to_ranks(const Simplex<D>& s, T (&v)[D + 1]) {
    for_each_comparator<D>([&](int c, int i) {
        const T a = v[i], b = v[i + 1];
        v[i] = s.swapped[c] ? b : a;
        v[i + 1] = s.swapped[c] ? a : b;
    });
}

// Rounding of every operation of the elevate step is explicit, because simplex selection at fine
// levels hinges on single ulps of the elevated coordinates (they reach 1e5..1e6).  The sequence
// below is what nvcc's default -fmad=true makes of the reference source (.cuh:130-138), established
// by comparing against the reference's own outputs for every pos_dim (cf_i = t_i*scale_i,
// t_i = pos_i + shift_i):
//   i = D      : e[D] = -(D*cf_D), sm = cf_D
//   2 <= i < D : e[i] = fma(-i, cf_i, sm), sm = sm + cf_i       (cf_i rounded, it feeds i*cf_i)
//   i = 1      : e[1] = fma(-t_1, scale_1, sm), e[0] = fma(t_1, scale_1, sm)
//
// Nearest remainder-0 point.  The reference takes the closer of floor(e/(D+1))*(D+1) and
// ceil(e/(D+1))*(D+1), the lower one on a tie (.cuh:150-161): r = ceil((e - (D+1)/2) / (D+1)).
// Below 2^22 this comes out of the float adder without a conversion instruction (conversions and
// floor run at a quarter of the rate of an add or less): adding 1.5*2^23 leaves the integer in the
// low mantissa bits, read as an integer for the hash and, after subtracting it again, as a float.
//  * D+1 a power of two: both additions round upwards, so rounding never crosses a multiple of D+1
//    from above (the multiple itself is representable) and the ceiling is exact.
//  * otherwise the reciprocal is inexact: round to nearest, then move by ceil((residual - (D+1)/2) /
//    (D+1)), which is not zero where the residual is outside (-(D+1)/2, (D+1)/2].  The fp32 reciprocals
//    of 3, 5, 6 and 7 are rounded upwards by 0.25 to 0.75 * 2^-24 of their value: a residual of
//    -(D+1)/2 gives -1, and the next one above it, rounded upwards by the subtraction to a multiple of
//    2^-22 or 2^-21, already 0.
// The residual e - (D+1)*r is exact in both cases (r*(D+1) <= 2|e| or r = 0), which is the
// reference's -(up - e) or e - down.  Where 2^22 may be exceeded (`largest`, the point's largest
// coordinate, against the level's reach) the reference's own expressions are used.
//
// Instructions per point and level, pos_dim 3: about 110 against 245 for a version with floor,
// rank counting, rank wrap and select-by-rank.
template <int D>
__device__ __forceinline__ void locate_simplex(const float (&pos)[D], float largest, const LevelConst<D>& lc, Simplex<D>& s) {
    constexpr float kInv = 1.0f / (D + 1);
    constexpr float kDp1 = (float)(D + 1);
    constexpr float kHalf = 0.5f * (D + 1);
    constexpr bool kPow2 = ((D + 1) & D) == 0;
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    constexpr int kMagicBits = 0x4B400000;

    float e[D + 1];
    float sm = 0.0f;
#pragma unroll
    for (int i = D; i > 0; --i) {
        const float t = __fadd_rn(pos[i - 1], lc.shift[i - 1]);
        const float sc = lc.scale[i - 1];
        if (i == 1) {
            e[1] = __fmaf_rn(-t, sc, sm);
            sm = __fmaf_rn(t, sc, sm);
        } else {
            const float cf = __fmul_rn(t, sc);
            if (i == D) {
                e[i] = -__fmul_rn((float)i, cf);
                sm = cf;
            } else {
                e[i] = __fmaf_rn(-(float)i, cf, sm);
                sm = __fadd_rn(sm, cf);
            }
        }
    }
    e[0] = sm;

    float res[D + 1];
    int rint[D + 1];  // R_i / (D+1)
    if (largest < lc.reach) {
        uint32_t h = 0u;
        int sum = 0;
#pragma unroll
        for (int i = 0; i <= D; ++i) {
            float w, r;
            if (kPow2) {
                w = __fmaf_ru(__fadd_ru(e[i], -kHalf), kInv, kMagic);
                r = __fsub_rn(w, kMagic);
                res[i] = __fmaf_rn(-kDp1, r, e[i]);
            } else {
                w = __fmaf_rn(e[i], kInv, kMagic);
                r = __fsub_rn(w, kMagic);
                res[i] = __fmaf_rn(-kDp1, r, e[i]);
                const float fix = __fsub_rn(__fmaf_ru(__fadd_ru(res[i], -kHalf), kInv, kMagic), kMagic);
                w = __fadd_rn(w, fix);
                res[i] = __fmaf_rn(-kDp1, fix, res[i]);
            }
            const int bits = __float_as_int(w);
            rint[i] = bits - kMagicBits;
            sum += rint[i];
            // hash of the vertex-0 key R_i - s over the D hashed coordinates, with R_i = (D+1)*rint_i
            // and s = sum(rint); the D+1 steps add up to zero, so the bias of `bits` drops out
            h -= (uint32_t)bits * hash_step<D>(i);
        }
        s.hash0 = h;
        s.s = sum;
#pragma unroll
        for (int i = 0; i <= D; ++i) s.lift[i] = (D + 1) * rint[i] - sum;
    } else {
        // coordinates beyond the exact range of the adder trick: the reference's expressions (.cuh:150-161, :176)
        float rem0f[D + 1], sumf = 0.0f;
#pragma unroll
        for (int i = 0; i <= D; ++i) {
            const float v = __fmul_rn(e[i], kInv);
            const float down = __fmul_rn(floorf(v), kDp1), up = __fmul_rn(ceilf(v), kDp1);
            const float du = __fsub_rn(up, e[i]), dd = __fsub_rn(e[i], down);
            rem0f[i] = du < dd ? up : down;
            res[i] = du < dd ? -du : dd;
            sumf = __fadd_rn(sumf, rem0f[i]);
        }
        s.s = __float2int_rn(__fmul_rn(sumf, kInv));
        uint32_t h = 0u;
#pragma unroll
        for (int i = 0; i <= D; ++i) {
            s.lift[i] = (int)rem0f[i] - s.s;
            if (i < D) h += (uint32_t)s.lift[i] * hash_pow(D - i);
        }
        s.hash0 = h;
    }

#pragma unroll
    for (int i = 0; i <= D; ++i) {
        s.x[i] = res[i];
        s.step[i] = hash_step<D>(i);
    }
    for_each_comparator<D>([&](int c, int i) {
        const float a = s.x[i], b = s.x[i + 1];
        const bool sw = a < b;
        s.x[i] = sw ? b : a;
        s.x[i + 1] = sw ? a : b;
        const uint32_t p = s.step[i], q = s.step[i + 1];
        s.step[i] = sw ? q : p;
        s.step[i + 1] = sw ? p : q;
        s.swapped[c] = sw;
    });
}

// hash of vertex q = 0..D, before the modulo
template <int D>
__device__ __forceinline__ void vertex_hashes(const Simplex<D>& s, uint32_t (&h)[D + 1]) {
    h[0] = s.hash0;
#pragma unroll
    for (int q = 1; q <= D; ++q) h[q] = h[q - 1] + s.step[D + 1 - q];
}

// barycentric weight of vertex q = 0..D times `factor` * (D+1)
template <int D>
__device__ __forceinline__ void vertex_weights(const Simplex<D>& s, float factor, float (&w)[D + 1]) {
    w[0] = __fadd_rn(__fsub_rn(s.x[D], s.x[0]), (float)(D + 1)) * factor;
#pragma unroll
    for (int q = 1; q <= D; ++q) w[q] = __fsub_rn(s.x[D - q], s.x[D + 1 - q]) * factor;
}

__device__ __forceinline__ void red_add1(float* p, float x) {
    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p), "f"(x) : "memory");
}

}  // namespace permuto
