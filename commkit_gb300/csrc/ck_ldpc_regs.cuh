// The latency form of the code-specialised decoder: a frame's check messages
// and columns in registers (min-sum as described here; sum-product below).  An NVRTC source (ck_ldpc_jit.cu).
#pragma once

#include "ck_ldpc_minsum.cuh"

namespace ck {
namespace ldpc {

// What bounds a batch that does not fill the GPU is the time of one frame's
// iteration: with one thread per row, a scheduler holds one or two warps and
// waits on every instruction of a row (code A: about 480 cycles a layer, of
// which a row's loads, minima and stores are a third).  So here
//  * two lanes share a row (lanes l and l + 16 of a warp, half of its edges
//    each, their minima and signs joined by three shuffles);
//  * a lane's messages and its columns' shared addresses stay in registers
//    over the whole decode (the program's edge slots are constants), so an
//    edge is one shared load and one store, of its posterior;
//  * the base rows of a layer go together: all loads, then all minima, then
//    all stores.
// An edge that a lane does not have (rows of odd degree, rows past the
// lifting) is a slot whose column is the lane's own word after the posterior,
// +inf at the frame's start: its message changes no minimum and no sign.
// Same float operations on the same values as the other forms (min1 and min2
// of the row are those of its edges in any grouping): the same bits.
// Measured on code A (Z = 54, 124 registers, 4 frames per SM): 50 iterations
// of 16 frames 113 to 64 us; with one message per edge in shared memory (10
// frames per SM) 1024 frames at 2.5 dB 122 us against 88, 4096 183 against
// 158, 8192 at 1.6 dB 447 against 483: batches of more waves
// than reg_waves (ck_ldpc.cu) keep the shared form.
//
// Prog (generated): kSlots edge slots per lane;
//   columns(a, a_addr, r, h, own)  the shared addresses of row r, half h;
//   clear(m)  zero messages;
//   iteration(m, a, scale, offset, T)  every layer, each with the barrier;
//   syndrome(a, T)  the early-stop test.

// One row's share of a lane: its D slots' messages and posteriors to Q, and
// the row's two smallest magnitudes and sign parity.
struct RegRow {
    float min1, min2;
    uint32_t par;
};
template <int D>
__device__ __forceinline__ RegRow reg_row_minima(const float (&q)[D]) {
    float min1 = fabsf(q[0]), min2 = ck::inf_f();
    uint32_t par = __float_as_uint(q[0]);
    // A NaN magnitude counts as absent, as in qc_row_edges.
    min1 = fminf(min1, ck::inf_f());
#pragma unroll
    for (int e = 1; e < D; ++e) {
        const float mag = fabsf(q[e]);
        min2 = fminf(min2, fmax_nan(min1, mag));
        min1 = fminf(min1, mag);
        par ^= __float_as_uint(q[e]);
    }
    const float o1 = __shfl_xor_sync(0xffffffffu, min1, 16), o2 = __shfl_xor_sync(0xffffffffu, min2, 16);
    par ^= __shfl_xor_sync(0xffffffffu, par, 16);
    RegRow r;
    r.min2 = fminf(fminf(min2, o2), fmaxf(min1, o1));
    r.min1 = fminf(min1, o1);
    r.par = par & 0x80000000u;
    return r;
}
// The row's new message magnitudes with its parity sign (p2 for every edge at
// the minimum, as in qc_row_edges), and one edge's new message and posterior.
struct RegOut {
    float min1;
    uint32_t p1, p2;
};
__device__ __forceinline__ RegOut reg_row_out(const RegRow& r, const float scale, const float offset) {
    const float n1 = fmaxf(__fsub_rn(__fmul_rn(scale, r.min1), offset), 0.0f);
    const float n2 = fmaxf(__fsub_rn(__fmul_rn(scale, r.min2), offset), 0.0f);
    return RegOut{r.min1, __float_as_uint(n1) ^ r.par, __float_as_uint(n2) ^ r.par};
}
__device__ __forceinline__ void reg_edge(const RegOut& o, const float q, const uint32_t a, float& m) {
    const uint32_t pm = fabsf(q) == o.min1 ? o.p2 : o.p1;
    m = __uint_as_float(pm ^ (__float_as_uint(q) & 0x80000000u));
    st_shared_f32(a, __fadd_rn(q, m));
}

// Sum-product (a generated iteration of its own): phi as ck_ldpc_sp.cu has it,
// and the row's total of phi values edge by edge in column order, the lower
// lane's edges first: the upper lane goes on from the lower one's sum.  A
// missing edge's +inf adds phi(30) = -0 to it.  The phi calls bound it, two
// per edge and iteration of some 40 instructions each: with one thread per
// row a frame's iteration is the chain of a row's calls, layer after layer;
// here it is half of that, all base rows of a layer run theirs together, and
// degrees are constants (the table-driven kernel steps through its degree
// bound).  Every size gains, so there is no limit of waves, and every code
// measured: 8 iterations of 1 / 608 / 6000 frames, Z = 8 (69 slots) 366 / 370 /
// 1050 to 90 / 91 / 483 us, Z = 256 (43 slots) 296 / 638 / 6223 to 82 / 314 / 3055,
// also where the slots exceed the registers and spill, Z = 256 (65 slots) 447 /
// 986 us to 149 / 540 for 1 / 608 frames, Z = 240 (72 slots) 496 / 1046 to 163 /
// 605.  50 iterations, table-driven kernel against this one: code B (Z = 96) at 3.2 dB 1 frame 75
// to 20 us, 256 frames 1159 to 255, 2048 1266 to 423, at 2.4 dB 2048 frames
// 2417 to 1474; code A at 1.6 dB 16 frames 733 to 103 us, 1024 1581 to 478,
// 4096 2289 to 1187.
__device__ __forceinline__ float reg_phi(float x) {
    x = fminf(fmaxf(x, 1e-7f), 30.0f);
    return -logf(tanhf(__fmul_rn(0.5f, x)));
}
struct RegSum {
    float total;
    bool neg;  // the row's parity of Q < 0
};
template <int D>
__device__ __forceinline__ RegSum reg_row_total(const float (&q)[D], const float (&ph)[D], const bool upper) {
    bool neg = false;
    float lower = 0.0f;
#pragma unroll
    for (int e = 0; e < D; ++e) {
        neg ^= q[e] < 0.0f;
        lower = __fadd_rn(lower, ph[e]);
    }
    float total = __shfl_xor_sync(0xffffffffu, lower, 16);
#pragma unroll
    for (int e = 0; e < D; ++e) total = __fadd_rn(total, ph[e]);
    const float other = __shfl_xor_sync(0xffffffffu, total, 16);
    neg ^= __shfl_xor_sync(0xffffffffu, static_cast<int>(neg), 16) != 0;
    return RegSum{upper ? total : other, neg};
}
__device__ __forceinline__ void reg_sp_edge(const RegSum& s, const float q, const float ph, const uint32_t a,
                                            float& m) {
    const float mag = reg_phi(__fsub_rn(s.total, ph));
    m = s.neg != (q < 0.0f) ? -mag : mag;
    st_shared_f32(a, __fadd_rn(q, m));
}

// One frame per block of p.T threads.
template <class Prog>
__device__ __forceinline__ void decode_regs_body(const Params& p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem);
    volatile uint32_t* s_frame = reinterpret_cast<volatile uint32_t*>(smem + 8);
    float* a = reinterpret_cast<float*>(smem + p.app_off);
    const uint32_t a_addr = ck::smem_addr(a);
    const uint32_t own = a_addr + 4u * static_cast<uint32_t>(p.N + tid);
    uint32_t cols[Prog::kSlots];
    float m[Prog::kSlots];
    Prog::columns(cols, a_addr, static_cast<uint32_t>(tid >> 5) * 16u + (lane & 15), lane >> 4, own);
    if (tid == 0) {
        ck::mbar_init(mbar, 1);
        ck::fence_mbar_init();
    }
    // All blocks of a direct launch are resident at once, so this store is far
    // ahead of a wait that runs out (2^24 polls) in any of them.
    if (p.direct && blockIdx.x == 0 && tid == 0) *p.status = 0u;
    __syncthreads();
    uint32_t phase = 0;
    for (;;) {
        uint32_t f;
        if (p.direct) {
            f = blockIdx.x;
        } else {
            if (tid == 0) *s_frame = atomicAdd(p.counter, 1u);
            __syncthreads();
            f = *s_frame;
            if (f >= p.B) break;
        }
        const float* src = p.llr_in + static_cast<size_t>(f) * p.n_in;
        bool loaded = true;
        if (p.bulk_load && tid == 0) {
            ck::fence_proxy_async_smem();
            ck::mbar_arrive_expect_tx(mbar, static_cast<uint32_t>(p.n_in) * 4u);
            ck::bulk_g2s(a, src, static_cast<uint32_t>(p.n_in) * 4u, mbar);
        }
        for (int i = p.n_in + tid; i < p.N; i += p.T) a[i] = 0.0f;
        st_shared_f32(own, ck::inf_f());
        Prog::clear(m);
        if (p.bulk_load) {
            loaded = ck::mbar_wait(mbar, phase);
            phase ^= 1u;
            // x + 0 turns -0 into +0 (see qc_row_cols).
            if (loaded)
                for (int i = tid; i < p.n_in; i += p.T) a[i] = __fadd_rn(a[i], 0.0f);
        } else {
            for (int i = tid; i < p.n_in; i += p.T) a[i] = __fadd_rn(__ldcs(src + i), 0.0f);
        }
        if (__syncthreads_or(loaded ? 0 : 1)) {
            // A bulk copy did not complete in time: report and stop after a
            // last bounded wait for the copy in flight.
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
            if (p.early_stop || it == p.max_iterations) ok = Prog::syndrome(cols, p.T);
            if (ok || it >= p.max_iterations) break;
            Prog::iteration(m, cols, p.scale, p.offset, p.T);
            ++it;
        }
        float* dst = p.llr_out + static_cast<size_t>(f) * p.n_in;
        for (int i = tid; i < p.n_in; i += p.T) __stcs(dst + i, a[i]);
        if (p.bits) {
            int8_t* bdst = p.bits + static_cast<size_t>(f) * p.k_bits;
            for (int i = tid; i < p.k_bits; i += p.T) bdst[i] = a[i] < 0.0f ? 1 : 0;
        }
        if (tid == 0) {
            p.iters[f] = it;
            p.valid[f] = ok ? 1 : 0;
        }
        if (p.direct) break;
        // Everyone has read `a` before the next frame overwrites it.
        __syncthreads();
    }
}

}  // namespace ldpc
}  // namespace ck
