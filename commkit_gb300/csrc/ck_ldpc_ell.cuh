// The min-sum decoder of codes without circulant structure: rows in 32-row groups
// with 16-bit columns, one persistent frame group per frame
// (ck_ldpc_kernel.cuh has the frame loop of the circulant codes and Params).
#pragma once

#include "ck_ldpc_kernel.cuh"

namespace ck {
namespace ldpc {

// What bounds such a code: its rows gather and scatter scattered posteriors.
// In device memory every lane of an access costs a line of its own (DVB-S2
// normal 1/2, N = 64800: about 21 lines per warp access, an L1 cycle each,
// which the two dependent loads of a row's pointers and columns add to), so
// the frame's posterior lives in shared memory, where a warp access costs
// its bank conflicts only:
//  * variables [0, ns) in shared memory, the rest (12 % of that code, the
//    last parity bits, which few rows touch) in the slot's device memory;
//    one block per SM then holds a frame of N = 64800 (228 KB).  The word
//    after variable ns - 1 holds +inf, the column of edges that a row does
//    not have: such a message changes no minimum and no sign;
//  * a row's columns are 16-bit places (v, or v + 1 from ns on), 8 to a
//    16-byte load, and, like its message state, loaded one row ahead: neither
//    depends on another thread, so the loads cross the layer barrier;
//  * every layer's rows start at a multiple of 32 and are ordered by the
//    plan (rows of a layer share no variable, so any order gives the same
//    bits): rows that touch device memory first, so that other rows cover
//    their loads, then the others by degree, in an order that spreads the
//    lanes of each access over the banks (2.3 cycles per access on that code
//    against 3.5 in schedule order).  A group of 32 rows runs the unrolled
//    row body of the circulant codes for its largest degree; only groups
//    marked special test their columns.
// Measured on that code against the posterior and 32-bit CSR columns in
// device memory: 64 frames, 11 iterations on average, 2.13 ms (a cluster of
// four blocks per frame) to 0.90 ms; 152 / 400 frames of 8 iterations (IRA
// rows of 7) 2.69 / 7.98 to 0.44 / 1.28 ms; one frame 496 to 432 us; N =
// 16200 in shared memory either way, rows of 6 / 14, 152 frames: 230 / 617 to
// 145 / 157 us.

// Threads per block the kernels are built for: registers scale inversely
// (rows of 7, 64 frames, 14 iterations: 1290 us with 1024 threads at 64
// registers, which spill, 1023 us with 768 at 80).
__host__ __device__ constexpr int ell_max_threads(int dmax) { return dmax > 16 ? 384 : (dmax > 8 ? 512 : 768); }

// Posterior access by place: shared memory up to the +inf word at ns, else
// the slot's device memory.
template <int W>
struct EllPost {
    const uint32_t (&w)[4 * W];
    uint32_t a_addr;  // shared address of variable 0
    uint32_t ns;
    float* g;  // variable ns, at place ns + 1
    __device__ __forceinline__ uint32_t col(int e) const { return (e & 1) ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu; }
    __device__ __forceinline__ float ld(uint32_t c) const {
        return c <= ns ? ld_shared_f32(a_addr + 4u * c) : __ldcg(g + (c - ns - 1u));
    }
    __device__ __forceinline__ void st(uint32_t c, float v) const {
        if (c < ns)
            st_shared_f32(a_addr + 4u * c, v);
        else if (c > ns)
            __stcg(g + (c - ns - 1u), v);
    }
};

// A row's columns and message state, loaded ahead of its update.
template <int W>
struct EllRow {
    uint32_t w[4 * W];
    uint4 state;
    uint32_t info;
};

template <int W>
__device__ __forceinline__ void ell_load_columns(const Params& p, uint32_t info, uint32_t row, EllRow<W>& r) {
    r.info = info;
    const uint4* cols = p.ell + row;
#pragma unroll
    for (int c = 0; c < W; ++c) {
        if (c == 0 || ell_degree(info) > 8u * c) {
            const uint4 v = __ldg(cols + static_cast<uint32_t>(c) * p.ell_rows);
            r.w[4 * c] = v.x;
            r.w[4 * c + 1] = v.y;
            r.w[4 * c + 2] = v.z;
            r.w[4 * c + 3] = v.w;
        }
    }
}

// XOR of the sign words of a row's posteriors (bit 31: its parity).
template <int DMAX, int W>
__device__ __forceinline__ uint32_t ell_parity(const EllRow<W>& r, const EllPost<W>& post) {
    const int d = static_cast<int>(ell_degree(r.info));
    uint32_t x = 0u;
    if (r.info & (kEllGeneral | kEllSpecial)) {
#pragma unroll
        for (int e = 0; e < DMAX; ++e)
            if (e < d) x ^= __float_as_uint(post.ld(post.col(e)));
    } else {
#pragma unroll
        for (int e = 0; e < DMAX; ++e)
            if (e < d) x ^= __float_as_uint(ld_shared_f32(post.a_addr + 4u * post.col(e)));
    }
    return x;
}

// State: the packed min-sum state (MinSumState), beside decode_kernel's
// interface with
//   uint4 load(row) const           the row's state
//   template <int DMAX, int W> void ell_row(p, r, post, row) const
//                                   one row with its columns and state in r
// Sum-product keeps the CSR kernels: phi bounds its rows, and this form's
// registers cost it more (rows of 6, 400 frames of N = 16200: 921 us against
// 852) than its loads gain.
template <template <bool> class State, int DMAX, bool R_SMEM>
__global__ void __launch_bounds__(ell_max_threads(DMAX)) decode_ell_kernel(const __grid_constant__ Params p) {
    extern __shared__ __align__(128) unsigned char smem[];
    using ck::group_any;
    using ck::group_sync;
    constexpr int W = (DMAX + 7) / 8;
    const uint32_t rows_all = p.ell_rows;
    int2* s_layer = reinterpret_cast<int2*>(smem);  // first row and end of each layer, then an empty one
    uint32_t* s_info = reinterpret_cast<uint32_t*>(smem) + 2 * (p.L + 1);
    for (int i = threadIdx.x; i <= p.L; i += blockDim.x) s_layer[i] = reinterpret_cast<const int2*>(p.layer)[i];
    for (uint32_t i = threadIdx.x; i < rows_all / 32; i += blockDim.x) s_info[i] = p.ell_info[i];

    const int g = threadIdx.x / p.T;
    const int tid = threadIdx.x - g * p.T;
    const int bar = g + 1;
    const uint32_t slot = blockIdx.x * static_cast<uint32_t>(p.G) + static_cast<uint32_t>(g);
    unsigned char* gbase = smem + p.tables_bytes + static_cast<uint32_t>(g) * p.group_bytes;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(gbase);
    volatile uint32_t* s_frame = reinterpret_cast<volatile uint32_t*>(gbase + 8);
    float* a = reinterpret_cast<float*>(gbase + p.app_off);
    const uint32_t a_addr = ck::smem_addr(a);
    float* tail = p.g_app + static_cast<size_t>(slot) * p.app_stride;  // variables ns .. N
    const State<R_SMEM> st(p, gbase, slot);
    if (tid == 0) {
        ck::mbar_init(mbar, 1);
        ck::fence_mbar_init();
        a[p.ell_ns] = ck::inf_f();
    }
    __syncthreads();

    const int32_t ns = p.ell_ns;
    const int32_t n_s = min(p.n_in, ns);  // sent variables in shared memory
    const uint32_t T = static_cast<uint32_t>(p.T);
    EllRow<W> next;
    auto prefetch = [&](uint32_t row) {
        ell_load_columns<W>(p, s_info[row >> 5], row, next);
        next.state = st.load(row);
    };
    auto post_of = [&](const EllRow<W>& r) {
        return EllPost<W>{r.w, a_addr, static_cast<uint32_t>(ns), tail};
    };
    // True in every thread of the group when every check holds: T rows
    // first (an unconverged frame usually fails there), then kRows times as
    // many per barrier, their columns in flight together.  The rows that fill a layer up to a multiple of 32
    // have no edges.
    auto satisfied = [&]() -> bool {
        constexpr uint32_t kRows = 4 / W;
        uint32_t per = 1;
        for (uint32_t base = 0; base < rows_all; base += per * T, per = kRows) {
            uint32_t bad = 0u;
            EllRow<W> r[kRows];
#pragma unroll
            for (uint32_t k = 0; k < kRows; ++k) {
                const uint32_t row = base + k * T + static_cast<uint32_t>(tid);
                r[k].info = 0u;
                if (k < per && row < rows_all) ell_load_columns<W>(p, s_info[row >> 5], row, r[k]);
            }
#pragma unroll
            for (uint32_t k = 0; k < kRows; ++k) bad |= ell_parity<DMAX, W>(r[k], post_of(r[k]));
            if (group_any(static_cast<int>(bad >> 31), bar, p.T)) return false;
        }
        return true;
    };

    uint32_t phase = 0;
    for (;;) {
        if (tid == 0) *s_frame = atomicAdd(p.counter, 1u);
        group_sync(bar, p.T);
        const uint32_t f = *s_frame;
        if (f >= p.B) break;
        const float* src = p.llr_in + static_cast<size_t>(f) * p.n_in;

        // The channel LLRs; punctured variables start at 0.  x + 0 turns -0
        // into +0 and keeps every other value (the row updates rely on it).
        bool loaded = true;
        if (p.bulk_load) {
            if (tid == 0) {
                ck::fence_proxy_async_smem();
                ck::mbar_arrive_expect_tx(mbar, static_cast<uint32_t>(n_s) * 4u);
                ck::bulk_g2s(a, src, static_cast<uint32_t>(n_s) * 4u, mbar);
            }
        } else {
            for (int i = tid; i < n_s; i += p.T) a[i] = __fadd_rn(__ldcs(src + i), 0.0f);
        }
        for (int i = n_s + tid; i < ns; i += p.T) a[i] = 0.0f;
        for (int i = ns + tid; i < p.N; i += p.T)
            __stcg(tail + (i - ns), i < p.n_in ? __fadd_rn(__ldcs(src + i), 0.0f) : 0.0f);
        st.zero(p, tid, p.T);
        if (p.bulk_load) {
            loaded = ck::mbar_wait(mbar, phase);
            phase ^= 1u;
            if (loaded)
                for (int i = tid; i < n_s; i += p.T) a[i] = __fadd_rn(a[i], 0.0f);
        }
        if (group_any(loaded ? 0 : 1, bar, p.T)) {
            // A bulk copy did not complete in time: report and stop this
            // group after a last bounded wait for the copy in flight.
            if (tid == 0) {
                atomicOr(p.status, ck::kStatusTimeout);
                p.iters[f] = -1;
                p.valid[f] = 0;
            }
            (void)ck::mbar_wait(mbar, phase ^ 1u);
            return;
        }

        int32_t it = 0;
        bool ok = false;
        for (;;) {
            if (p.early_stop || it == p.max_iterations) ok = satisfied();
            if (ok || it >= p.max_iterations) break;
            // The thread's rows of layer l are its first + tid, + T, ...; the
            // row after the current one, in this layer or the next, is
            // loaded before the current one is updated.
            int2 rows = s_layer[0];
            uint32_t row = static_cast<uint32_t>(rows.x + tid);
            bool have = row < static_cast<uint32_t>(rows.y);
            if (have) prefetch(row);
            for (int32_t l = 0; l < p.L; ++l) {
                const uint32_t end = static_cast<uint32_t>(rows.y);
                rows = s_layer[l + 1];
                const uint32_t first2 = static_cast<uint32_t>(rows.x + tid);
                const bool more = first2 < static_cast<uint32_t>(rows.y);
                if (!have && more) prefetch(first2);
                while (have) {
                    const EllRow<W> cur = next;
                    const uint32_t at = row;
                    row += T;
                    have = row < end;
                    if (have)
                        prefetch(row);
                    else if (more)
                        prefetch(first2);
                    st.template ell_row<DMAX, W>(p, cur, post_of(cur), at);
                }
                row = first2;
                have = more;
                group_sync(bar, p.T);
            }
            ++it;
        }

        float* dst = p.llr_out + static_cast<size_t>(f) * p.n_in;
        for (int i = tid; i < n_s; i += p.T) __stcs(dst + i, a[i]);
        for (int i = ns + tid; i < p.n_in; i += p.T) __stcs(dst + i, __ldcg(tail + (i - ns)));
        if (p.bits) {
            int8_t* bdst = p.bits + static_cast<size_t>(f) * p.k_bits;
            for (int i = tid; i < p.k_bits; i += p.T)
                bdst[i] = (i < ns ? a[i] : __ldcg(tail + (i - ns))) < 0.0f ? 1 : 0;
        }
        if (tid == 0) {
            p.iters[f] = it;
            p.valid[f] = ok ? 1 : 0;
        }
        // Everyone has read the posterior before the next frame overwrites it.
        group_sync(bar, p.T);
    }
}

#ifndef __CUDACC_RTC__
// The kernel for codes whose longest row has max_deg (up to kPackedDegree)
// edges.
KernelFn min_sum_ell_kernel(int max_deg, bool r_smem);
#endif

}  // namespace ldpc
}  // namespace ck
