// The labelling of Gray cross QAM at compile time (5, 7 and 9 bits per
// symbol), for the max-log demapper over every point (ck_llr_points.cuh).
//
// The cross is the Gray rectangle of ceil(K/2) x floor(K/2) bits with its
// outer columns folded onto the top and bottom of the central square
// (commkit/mapping/gray.py:301-425).  Its points lie on N x N coordinate
// values (N = 6, 12, 24), and the points whose bit b is v form a few
// rectangles of them: 26 for the 14 halves of 128 points.
#pragma once

#include <stdint.h>

namespace ck {
namespace llr {
namespace points {

template <int K>
struct Cross {
    static constexpr bool kIs = K >= 5 && K <= 9 && K % 2 == 1;
    static constexpr int NI = (K + 1) / 2, NQ = K / 2;
    static constexpr int W = 1 << NI, H = 1 << NQ, kWing = kIs ? 1 << (NI - 3) : 0;
    static constexpr int N = kIs ? W - 2 * kWing : 1;  // coordinate values per axis (H + 2 wing as well)

    static __host__ __device__ constexpr int rank(int g) {
        for (int s = 1; s < 16; s <<= 1) g ^= g >> s;
        return g;
    }
    // Coordinate indices (from the lowest value) of a label's point.
    static __host__ __device__ constexpr int re(int label) {
        const int gi = rank(label >> NQ), gq = rank(label & (H - 1));
        return (gi < kWing || gi >= W - kWing ? gq + (W - H) / 2 : gi) - kWing;
    }
    static __host__ __device__ constexpr int im(int label) {
        const int gi = rank(label >> NQ), gq = rank(label & (H - 1));
        return (gi < kWing ? H + kWing - 1 - gi : gi >= W - kWing ? -1 - (gi - (W - kWing)) : gq) + kWing;
    }

    // Per bit b (MSB first) and half v: the rectangles cols[b][v][j] x
    // rows[b][v][j] (sets of coordinate indices), one for each row j that is
    // the first with its columns; rows is 0 for the other rows.
    struct Sets {
        uint32_t cols[K][2][N], rows[K][2][N];
    };
    static constexpr Sets make() {
        Sets s{};
        for (int l = 0; kIs && l < (1 << K); ++l)
            for (int b = 0; b < K; ++b) s.cols[b][(l >> (K - 1 - b)) & 1][im(l)] |= 1u << re(l);
        for (int b = 0; b < K; ++b)
            for (int v = 0; v < 2; ++v)
                for (int j = N - 1; j >= 0; --j) {
                    const uint32_t c = s.cols[b][v][j];
                    if (!c) continue;
                    for (int i = j; i < N; ++i)
                        if (s.cols[b][v][i] == c) {
                            s.rows[b][v][j] |= 1u << i;
                            if (i > j) s.rows[b][v][i] = 0u;
                        }
                }
        return s;
    }
    static constexpr Sets kSets = make();
};

// Minimum of a[i] over the set M, by aligned ranges [LO, LO + SIZE) so that
// the sets' common parts are common subexpressions.
template <uint32_t M, int LO, int SIZE, int N>
__device__ __forceinline__ float min_over(const float (&a)[N]) {
    constexpr uint32_t range = (SIZE >= 32 ? 0xffffffffu : (1u << SIZE) - 1u) << LO;
    static_assert((M & range) != 0u, "an empty set");
    if constexpr (SIZE == 1) {
        return a[LO];
    } else {
        constexpr int half = SIZE / 2;
        constexpr uint32_t low = ((1u << half) - 1u) << LO, high = low << half;
        if constexpr (!(M & low)) {
            return min_over<M, LO + half, half>(a);
        } else if constexpr (!(M & high)) {
            return min_over<M, LO, half>(a);
        } else {
            return fminf(min_over<M, LO, half>(a), min_over<M, LO + half, half>(a));
        }
    }
}

// Smallest squared distance to the points whose bit B is V: the minimum over
// their rectangles of (smallest column distance) + (smallest row distance),
// dr and di the squared coordinate distances.  Rounded addition keeps order,
// so this is the minimum of the points' own rounded sums.
template <int K, int B, int V, int J = 0, int N>
__device__ __forceinline__ float cross_nearest(const float (&dr)[N], const float (&di)[N], float p) {
    if constexpr (J < N) {
        constexpr uint32_t rows = Cross<K>::kSets.rows[B][V][J];
        if constexpr (rows != 0u) {
            constexpr uint32_t cols = Cross<K>::kSets.cols[B][V][J];
            p = fminf(p, __fadd_rn(min_over<cols, 0, 32>(dr), min_over<rows, 0, 32>(di)));
        }
        return cross_nearest<K, B, V, J + 1>(dr, di, p);
    } else {
        return p;
    }
}
template <int K, int B = 0, int N>
__device__ __forceinline__ void cross_halves(const float (&dr)[N], const float (&di)[N], float (&p)[2][K]) {
    if constexpr (B < K) {
        p[0][B] = cross_nearest<K, B, 0>(dr, di, __int_as_float(0x7f800000));
        p[1][B] = cross_nearest<K, B, 1>(dr, di, __int_as_float(0x7f800000));
        cross_halves<K, B + 1>(dr, di, p);
    }
}

}  // namespace points
}  // namespace llr
}  // namespace ck
