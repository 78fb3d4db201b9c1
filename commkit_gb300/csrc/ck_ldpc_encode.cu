// The accumulator encoder in one kernel: s = H_info u over GF(2), the
// accumulation p_j = s_j + p_{j - g}, and the codeword bytes [u | p]
// (commkit/coding/ldpc.py:445-536).
//
// Bytes bound the byte-wise form: one thread per check XORed single bytes
// (2432 blocks, 86 us for 1000 frames of code C), another pass accumulated
// them with a byte in 32-byte sectors of g-strided chains (44 us), a third
// copied the information (20 us).  Here up to 32 frames share a word: a block
// packs its frames' information bits into words of one bit per frame (bytes
// to bits by a multiply, then a 32 x 32 bit transpose of shuffles), so a
// check's XOR and the accumulation serve 32 frames at once from shared
// memory, and nothing is kept between kernels.
//
// A block takes a group of frames and a tile of the accumulator's g
// residues: the chains of different residues are independent, so wide
// accumulators (lifted codes, g = Z) split over blocks, each packing the
// group's information anew (from L2).  The rows of a tile go in chunks of
// four rows per thread, whose column loads are in flight together, each chunk
// scanned over its chains in shared memory.  Measured (encode_blocks, calls
// back to back; the figures above are of each kernel alone, cold): 1000 frames
// of code C 130 to 31 us, 4096 frames of code A 31 to 14 us (the launch), 128
// frames of DVB-S2 normal 97 to 64 us.  A few frames of one long chain
// keep the byte-wise kernels (few_long_frames, ck_sim.cu).
#include <stdint.h>

#include <algorithm>
#include <numeric>

#include "ck_ldpc_encode.h"
#include "ck_ldpc_internal.h"

namespace {

constexpr int kLoadLanes = 32 * 16;                    // columns per warp step: 16 bytes per lane
constexpr uint32_t kTileWords = 32 * 17;               // per warp: 32 frames x 32 lanes x 16 bits, rows padded
constexpr int kRows = 4;                               // rows of a chunk per thread

struct EncodeArgs {
    const int8_t* info;
    int8_t* words;
    const int32_t* row_ptr;
    const int32_t* cols;
    int32_t* bad;  // or null: set when an information byte is not 0 or 1
    int64_t B;
    int32_t k, m, n, g;
    int32_t frames;      // per group, up to 32
    int32_t tile, tiles; // residues per tile, tiles
    int32_t copy;        // bytes per access of the information's copy
};

// 16 bytes at p, of which the first `left` (a multiple of V, 0 for none)
// exist, in loads of V bytes; the others read as 0.
template <int V>
__device__ __forceinline__ uint4 load16(const int8_t* p, int left) {
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if constexpr (V == 16) {
        if (left > 0) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
            return v;
        }
    } else if constexpr (V >= 4) {
#pragma unroll
        for (int i = 0; i < 16 / V; ++i) {
            if (V * i < left) {
                if constexpr (V == 8) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p) + i);
                    w[2 * i] = v.x;
                    w[2 * i + 1] = v.y;
                } else {
                    w[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < left) w[i / 4] |= static_cast<uint32_t>(static_cast<uint8_t>(__ldg(p + i))) << (8 * (i % 4));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Bit 0 of each of a word's four bytes, as bits 0..3: the products of the
// multiply land on distinct bits, byte i's on bit 24 + i.
__device__ __forceinline__ uint32_t low_bits(uint32_t w) { return ((w & 0x01010101u) * 0x01020408u) >> 24 & 0xfu; }

// The warp's 32 x 32 bit transpose: lane r holds row r; on return lane c
// holds column c (bit r = row r's bit c).  Swaps off-diagonal blocks of
// 16, 8, .. 1.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
    for (int j = 16; j >= 1; j >>= 1) {
        const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        const bool up = lane & j;
        const uint32_t keep = up ? ~m : m;
        x = (x & keep) | (__funnelshift_l(y, y, up ? 32 - j : j) & ~keep);
    }
    return x;
}

// Copies columns [0, k) of F frames, `first`, `first + step`, ... in accesses
// of the size of U.
template <class U>
__device__ __forceinline__ void copy_info(const int8_t* info, int8_t* words, int32_t k, int32_t n, int32_t F,
                                          uint32_t first, uint32_t step) {
    const uint32_t units = static_cast<uint32_t>(k) / sizeof(U);
    for (uint32_t i = first; i < units * F; i += step) {
        const uint32_t f = i / units, c = (i - f * units) * sizeof(U);
        *reinterpret_cast<U*>(words + static_cast<int64_t>(f) * n + c) =
            __ldg(reinterpret_cast<const U*>(info + static_cast<int64_t>(f) * k + c));
    }
}

// V: bytes per load of the information; R: parity bytes per store.
template <int T, int V, int R>
__global__ void __launch_bounds__(T) encode_kernel(const EncodeArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    const int32_t kw = (a.k + 31) / 32 * 32;
    uint32_t* u = smem;               // a word per information bit
    uint32_t* carry = u + kw;         // the chains' last parity, per residue
    uint32_t* x = carry + (a.tile + 3) / 4 * 4;  // a chunk of rows; before that the packing's tiles
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t* bits = x + warp * kTileWords;

    const int64_t group = blockIdx.x / static_cast<uint32_t>(a.tiles);
    const int32_t tile = static_cast<int32_t>(blockIdx.x - group * a.tiles);
    const int64_t f0 = group * a.frames;
    const int32_t F = static_cast<int32_t>(min(static_cast<int64_t>(a.frames), a.B - f0));
    const int8_t* info = a.info + f0 * a.k;
    int8_t* words = a.words + f0 * a.n;

    // Pack: 512 columns of the group's frames per warp step.
    uint32_t bad = 0u;
    for (int32_t c0 = warp * kLoadLanes; c0 < a.k; c0 += T / 32 * kLoadLanes) {
        const int32_t left = max(0, min(16, a.k - c0 - 16 * lane));
        const int8_t* src = info + c0 + 16 * lane;
#pragma unroll 8
        for (int32_t f = 0; f < F; ++f) {
            const uint4 v = load16<V>(src + static_cast<int64_t>(f) * a.k, left);
            bad |= (v.x | v.y | v.z | v.w) & 0xfefefefeu;
            reinterpret_cast<uint16_t*>(bits + 17 * f)[lane] = static_cast<uint16_t>(
                low_bits(v.x) | low_bits(v.y) << 4 | low_bits(v.z) << 8 | low_bits(v.w) << 12);
        }
        __syncwarp();
        for (int32_t c = c0; c < min(c0 + kLoadLanes, a.k); c += 32)
            u[c + lane] = transpose32(lane < F ? bits[17 * lane + (c - c0) / 32] : 0u, lane);
        __syncwarp();
    }
    if (a.bad && bad) atomicOr(a.bad, 1);

    // The information part of the codewords, shared out over the tiles.
    {
        const uint32_t first = tid + T * tile, step = T * a.tiles;
        switch (a.copy) {
            case 16: copy_info<uint4>(info, words, a.k, a.n, F, first, step); break;
            case 8: copy_info<uint2>(info, words, a.k, a.n, F, first, step); break;
            case 4: copy_info<uint32_t>(info, words, a.k, a.n, F, first, step); break;
            default: copy_info<signed char>(reinterpret_cast<const int8_t*>(info), words, a.k, a.n, F, first, step);
        }
    }

    const int32_t r0 = tile * a.tile, tw = min(a.tile, a.g - r0);
    const int32_t total = (a.m - r0 + a.g - 1) / a.g * tw;  // the tile's rows, chain step by chain step
    const int32_t C = T / tw * tw;                          // rows per step of a chunk, kRows steps
    for (int i = tid; i < tw; i += T) carry[i] = 0u;
    const int32_t res = tid % tw;
    // Store work: a thread takes R rows of a chunk and every S-th frame.
    const int32_t nq = kRows * C / R;
    const int32_t S = nq < T ? T / nq : 1;
    __syncthreads();
    for (int32_t base = 0; base < total; base += kRows * C) {
        // The thread's rows base + q C + tid, their loads in flight together.
        int32_t e[kRows], e1[kRows];
        uint32_t v[kRows];
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
            const int32_t i = base + q * C + tid;
            const int32_t j = i / tw * a.g + r0 + res;
            const bool row = tid < C && i < total && j < a.m;
            e[q] = row ? __ldg(a.row_ptr + j) : 0;
            e1[q] = row ? __ldg(a.row_ptr + j + 1) : 0;
            v[q] = 0u;
        }
        for (bool more = true; more;) {
            int32_t c[kRows][4];
#pragma unroll
            for (int q = 0; q < kRows; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) c[q][i] = e[q] + i < e1[q] ? __ldg(a.cols + e[q] + i) : -1;
            more = false;
#pragma unroll
            for (int q = 0; q < kRows; ++q) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (c[q][i] >= 0) v[q] ^= u[c[q][i]];
                e[q] += 4;
                more |= e[q] < e1[q];
            }
        }
        // XOR scan along the chains (rows tw apart), each step of C rows by
        // itself, then over the steps.
        const uint32_t last = tid < C ? carry[res] : 0u;
        uint32_t before[kRows];  // parity of the chain before the step
        if (tw == 1) {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
#pragma unroll
                for (int q = 0; q < kRows; ++q) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, v[q], d);
                    if (lane >= d) v[q] ^= o;
                }
#pragma unroll
            for (int q = 0; q < kRows; ++q)
                if (lane == 31) x[q * (T / 32) + warp] = v[q];
            __syncthreads();
            if (warp < kRows) {
                uint32_t t = lane < T / 32 ? x[warp * (T / 32) + lane] : 0u;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, t, d);
                    if (lane >= d) t ^= o;
                }
                if (lane < T / 32) x[warp * (T / 32) + lane] = t;
            }
            __syncthreads();
            uint32_t t = last;
#pragma unroll
            for (int q = 0; q < kRows; ++q) {
                before[q] = t ^ (warp > 0 ? x[q * (T / 32) + warp - 1] : 0u);
                t ^= x[q * (T / 32) + T / 32 - 1];
            }
        } else {
            for (int32_t d = tw; d < C; d <<= 1) {
#pragma unroll
                for (int q = 0; q < kRows; ++q) x[q * T + tid] = v[q];
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kRows; ++q)
                    if (tid < C && tid >= d) v[q] ^= x[q * T + tid - d];
                __syncthreads();
            }
            if (tid < C && tid >= C - tw)
#pragma unroll
                for (int q = 0; q < kRows; ++q) x[q * T + res] = v[q];
            __syncthreads();
            uint32_t t = last;
#pragma unroll
            for (int q = 0; q < kRows; ++q) {
                before[q] = t;
                t ^= tid < C ? x[q * T + res] : 0u;
            }
        }
        __syncthreads();
        if (tid < C) {
#pragma unroll
            for (int q = 0; q < kRows; ++q) x[q * C + tid] = v[q] ^ before[q];
            if (tid >= C - tw) carry[res] = v[kRows - 1] ^ before[kRows - 1];
        }
        __syncthreads();
        // The chunk's parity bytes.
        for (int32_t i = tid; i < nq * S; i += T) {
            const int32_t fs = i / nq, at = (i - fs * nq) * R;
            if (base + at >= total) continue;
            const int32_t q = (base + at) / tw;
            const int32_t j = q * a.g + r0 + (base + at - q * tw);
            int8_t* d = words + a.k + j;
            if constexpr (R == 4) {
                const uint4 w = *reinterpret_cast<const uint4*>(x + at);
                if (j + 3 < a.m && a.k + j + 3 < a.n) {
#pragma unroll 4
                    for (int32_t f = fs; f < F; f += S)
                        *reinterpret_cast<uint32_t*>(d + static_cast<int64_t>(f) * a.n) =
                            (w.x >> f & 1u) | (w.y >> f & 1u) << 8 | (w.z >> f & 1u) << 16 | (w.w >> f & 1u) << 24;
                } else {
                    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
                    for (int32_t f = fs; f < F; f += S)
#pragma unroll
                        for (int i4 = 0; i4 < 4; ++i4)
                            if (j + i4 < a.m && a.k + j + i4 < a.n)
                                d[static_cast<int64_t>(f) * a.n + i4] = static_cast<int8_t>(ws[i4] >> f & 1u);
                }
            } else {
                const uint32_t w = x[at];
                if (j < a.m && a.k + j < a.n)
#pragma unroll 4
                    for (int32_t f = fs; f < F; f += S) d[static_cast<int64_t>(f) * a.n] = static_cast<int8_t>(w >> f & 1u);
            }
        }
        __syncthreads();
    }
}

template <int T, int R>
const void* pick(int v) {
    switch (v) {
        case 16: return reinterpret_cast<const void*>(encode_kernel<T, 16, R>);
        case 8: return reinterpret_cast<const void*>(encode_kernel<T, 8, R>);
        case 4: return reinterpret_cast<const void*>(encode_kernel<T, 4, R>);
        default: return reinterpret_cast<const void*>(encode_kernel<T, 1, R>);
    }
}

// The largest power of two up to 16 that divides every given value.
int common_vector(std::initializer_list<uint64_t> values) {
    int v = 16;
    for (uint64_t x : values)
        while (x % v) v /= 2;
    return v == 2 ? 1 : v;
}

}  // namespace

int ck::encode_accumulate(const int8_t* info, int64_t B, int32_t k, int32_t m, int32_t n,
                          const int32_t* row_ptr, const int32_t* cols, int32_t g, int8_t* words, int32_t* bad,
                          cudaStream_t stream, bool* done) {
    *done = false;
    int dev = 0, sms = 0, optin = 0;
    CK_CUDA(cudaGetDevice(&dev));
    CK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    EncodeArgs a{info, words, row_ptr, cols, bad, B, k, m, n, g, 32, 0, 0, 1};
    a.g = std::min(g, m);  // a chain of one step either way
    // Long chains take larger blocks where the information leaves room.  Tiles of at least 32 residues (one
    // store segment), as many as fill the GPU with groups of 32 frames; then
    // fewer frames per group (short batches) until it is filled.
    const auto bytes_of = [&](int T, int32_t tile) {
        return 4 * (static_cast<size_t>((k + 31) / 32 * 32) + (tile + 3) / 4 * 4 + static_cast<size_t>(T / 32) * kTileWords);
    };
    static_assert(32 * kRows <= kTileWords, "a chunk fits the packing's tiles");
    const int T = a.g < 32 && bytes_of(1024, a.g) <= static_cast<size_t>(optin) ? 1024 : 512;
    const int32_t most = std::max(1, a.g / 32);
    const int64_t groups = (B + 31) / 32;
    const int64_t want = std::min<int64_t>(most, std::max<int64_t>((a.g + T - 1) / T, (sms + groups - 1) / groups));
    a.tile = static_cast<int32_t>((a.g + want - 1) / want);
    if (want > 1) a.tile = (a.tile + 15) / 16 * 16;
    a.tiles = (a.g + a.tile - 1) / a.tile;
    while (a.frames > 1 && (B + a.frames - 1) / a.frames * a.tiles * 2 <= sms) a.frames /= 2;
    const int64_t blocks = (B + a.frames - 1) / a.frames * a.tiles;
    const size_t smem = bytes_of(T, a.tile);
    if (smem > static_cast<size_t>(optin) || blocks >= (int64_t(1) << 31) || a.tile > T) return CK_OK;
    const uint64_t at = reinterpret_cast<uintptr_t>(info), to = reinterpret_cast<uintptr_t>(words);
    const int v = common_vector({static_cast<uint64_t>(k), at});
    a.copy = common_vector({static_cast<uint64_t>(k), static_cast<uint64_t>(n), at, to});
    // Four parity bytes per store where every residue run is of fours.
    const bool four = a.copy >= 4 && a.g % 4 == 0 && a.tile % 4 == 0;
    const void* kernel = T == 1024 ? (four ? pick<1024, 4>(v) : pick<1024, 1>(v)) : (four ? pick<512, 4>(v) : pick<512, 1>(v));
    CK_TRY(ck::allow_max_smem(kernel, dev, optin));
    void* args[] = {&a};
    CK_TRY(ck::cuda_check(cudaLaunchKernel(kernel, dim3(static_cast<unsigned>(blocks)), dim3(T), args, smem, stream),
                          "encoder launch"));
    *done = true;
    return CK_OK;
}
