// Walsh-Hadamard building blocks for many rows (prompts): 32 values per thread, exchanges through shared memory.
//
// A segment is 4096 columns for a CTA of 128 threads (blocks of more than 256, up to 4096); it
// may hold several blocks.  Element e of a segment is at e + 8 (e >> 8) in the exchange buffer, which keeps all accesses
// below free of bank conflicts.  The layouts of a thread's 32 values, by the bits of e that vary inside the thread:
//   pieces   bits 0-2, 10 and 11: four pieces of eight consecutive elements, loaded and stored as 16 bytes of fp16 each
//   columns  bits 3-7
//   far      bits 0 and 8-11: sixteen pairs, 256 elements apart
// A transform does the stages of bits 0-2 in pieces, 3-7 in columns, 8-11 in far: in ascending order, the order of the
// kernels with eight values per thread, so that the results of both are the same bits.  Stages at or above the block size
// are skipped.  A thread that has read its values in one layout may write them in the same layout without a barrier.
// Against eight values per thread with shuffles (five stages x eight values through the same pipe as shared memory):
// 2048 x 4096 in 13.4 us instead of 19.3.
#pragma once
#include "common.cuh"
#include "fwht.cuh"

namespace rptc {

constexpr int kCtaSegFloats = 4096 + 128;

// One butterfly stage over bit `H` of the index of v.
template <int H>
__device__ __forceinline__ void stage(float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if ((i & H) == 0) {
            const float a = v[i], b = v[i + H];
            v[i] = a + b;
            v[i + H] = a - b;
        }
}

// v[8 j + i] is element i of piece j.
__device__ __forceinline__ void piece_stages(float (&v)[32]) {
    stage<1>(v);                       // blocks have at least eight elements
    stage<2>(v);
    stage<4>(v);
}
// v[k] is element bits 3-7 = k.
__device__ __forceinline__ void column_stages(float (&v)[32], int block_bits) {
    if (block_bits > 3) stage<1>(v);
    if (block_bits > 4) stage<2>(v);
    if (block_bits > 5) stage<4>(v);
    if (block_bits > 6) stage<8>(v);
    if (block_bits > 7) stage<16>(v);
}
// v[2 k + e] is element e of pair k.
__device__ __forceinline__ void far_stages(float (&v)[32], int block_bits) {
    if (block_bits > 8) stage<2>(v);
    if (block_bits > 9) stage<4>(v);
    if (block_bits > 10) stage<8>(v);
    if (block_bits > 11) stage<16>(v);
}

// Where a thread's values are; t of 128 threads in a CTA segment.
struct SegThread {
    int lane, warp, t;
    __device__ __forceinline__ SegThread() : lane(threadIdx.x & 31), warp((threadIdx.x >> 5) & 3), t(threadIdx.x & 127) {}
    __device__ __forceinline__ int piece(int j) const { return 8 * t + 1024 * j; }
    __device__ __forceinline__ int pair(int k) const { return 2 * t + 256 * k; }
    __device__ __forceinline__ int column() const {      // element of k = 0: bits 0-2 from the lane, bits 8 up from the rest
        return (lane & 7) + 256 * ((lane >> 3) + 4 * warp);
    }
    static __device__ __forceinline__ int at(int e) { return e + 8 * (e >> 8); }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
    // The two halves of a piece as 16-byte accesses; lanes with bit 2 set take the upper half first, so that eight lanes
    // with a stride of 32 bytes meet all banks once.
    __device__ __forceinline__ void put_pieces(float *buf, const float (&v)[32]) const {
        const bool swap = lane & 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 *p = reinterpret_cast<float4 *>(buf + at(piece(j)));
            const float4 a = make_float4(v[8 * j], v[8 * j + 1], v[8 * j + 2], v[8 * j + 3]);
            const float4 b = make_float4(v[8 * j + 4], v[8 * j + 5], v[8 * j + 6], v[8 * j + 7]);
            p[swap ? 1 : 0] = swap ? b : a;
            p[swap ? 0 : 1] = swap ? a : b;
        }
    }
    __device__ __forceinline__ void get_pieces(const float *buf, float (&v)[32]) const {
        const bool swap = lane & 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 *p = reinterpret_cast<const float4 *>(buf + at(piece(j)));
            const float4 x = p[swap ? 1 : 0], y = p[swap ? 0 : 1];
            const float4 a = swap ? y : x, b = swap ? x : y;
            v[8 * j] = a.x, v[8 * j + 1] = a.y, v[8 * j + 2] = a.z, v[8 * j + 3] = a.w;
            v[8 * j + 4] = b.x, v[8 * j + 5] = b.y, v[8 * j + 6] = b.z, v[8 * j + 7] = b.w;
        }
    }
    __device__ __forceinline__ void put_pairs(float *buf, const float (&v)[32]) const {
#pragma unroll
        for (int k = 0; k < 16; ++k) *reinterpret_cast<float2 *>(buf + at(pair(k))) = make_float2(v[2 * k], v[2 * k + 1]);
    }
    __device__ __forceinline__ void get_pairs(const float *buf, float (&v)[32]) const {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 p = *reinterpret_cast<const float2 *>(buf + at(pair(k)));
            v[2 * k] = p.x, v[2 * k + 1] = p.y;
        }
    }
    __device__ __forceinline__ void put_columns(float *buf, const float (&v)[32]) const {
        float *p = buf + at(column());
#pragma unroll
        for (int k = 0; k < 32; ++k) p[8 * k] = v[k];
    }
    __device__ __forceinline__ void get_columns(const float *buf, float (&v)[32]) const {
        const float *p = buf + at(column());
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = p[8 * k];
    }
};

__device__ __forceinline__ void unpack8_at(const uint4 &a, float *v) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(u32_as_half2(w[i]));
        v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
}

}  // namespace rptc
