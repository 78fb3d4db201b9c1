// Host side of the layered LDPC decoder: the first-fit layer schedule and
// the decoding plan (schedule validation, recovery of the circulant
// structure of quasi-cyclic codes, device tables).
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <numeric>
#include <vector>

#include "ck_ldpc_internal.h"

// ---------------------------------------------------------------------------
// First-fit schedule: restates LDPCCode._schedule and _first_fit
// (commkit/coding/ldpc.py:283-296, 422-442).
// ---------------------------------------------------------------------------

extern "C" int ck_ldpc_schedule(const int32_t* checks, const int32_t* variables, int64_t E,
                                int32_t m, int32_t N, int32_t* row_ptr, int32_t* cols,
                                int32_t* layer_ptr, int32_t* num_layers) {
    ck::clear_error();
    if (!checks || !variables || !row_ptr || !cols || !layer_ptr || !num_layers)
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL argument");
    if (m < 1 || N < 1 || E < 1 || E >= (int64_t(1) << 31))
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "bad sizes m=%d N=%d E=%lld", m, N,
                        static_cast<long long>(E));
    // Rows in natural order: the edges are sorted by (row, column).
    std::vector<int64_t> ptr(static_cast<size_t>(m) + 1, 0);
    for (int64_t e = 0; e < E; ++e) {
        const int32_t r = checks[e];
        const int32_t c = variables[e];
        if (r < 0 || r >= m || c < 0 || c >= N)
            return ck::fail(CK_ERR_INVALID_ARGUMENT, "edge %lld out of range", static_cast<long long>(e));
        if (e > 0 && (checks[e - 1] > r || (checks[e - 1] == r && variables[e - 1] >= c)))
            return ck::fail(CK_ERR_INVALID_ARGUMENT,
                            "edges must be sorted by (row, column) without duplicates");
        ++ptr[static_cast<size_t>(r) + 1];
    }
    for (int32_t r = 0; r < m; ++r) ptr[r + 1] += ptr[r];

    // Layers used by each variable, as a bit set of `words` 64-bit words.
    size_t words = 1;
    std::vector<uint64_t> masks(static_cast<size_t>(N) * words, 0);
    std::vector<int32_t> color(static_cast<size_t>(m));
    std::vector<uint64_t> used;
    int32_t layers = 0;
    for (int32_t r = 0; r < m; ++r) {
        used.assign(words, 0);
        for (int64_t e = ptr[r]; e < ptr[r + 1]; ++e) {
            const uint64_t* mv = &masks[static_cast<size_t>(variables[e]) * words];
            for (size_t w = 0; w < words; ++w) used[w] |= mv[w];
        }
        // Lowest layer not in `used`.
        int32_t c = -1;
        for (size_t w = 0; w < words && c < 0; ++w) {
            if (~used[w]) c = static_cast<int32_t>(w * 64 + __builtin_ctzll(~used[w]));
        }
        if (c < 0) c = static_cast<int32_t>(words * 64);
        if (static_cast<size_t>(c) >= words * 64) {
            // Grow every mask by one word.
            const size_t nw = words + 1;
            std::vector<uint64_t> grown(static_cast<size_t>(N) * nw, 0);
            for (int32_t v = 0; v < N; ++v)
                memcpy(&grown[static_cast<size_t>(v) * nw], &masks[static_cast<size_t>(v) * words],
                       words * sizeof(uint64_t));
            masks.swap(grown);
            words = nw;
        }
        for (int64_t e = ptr[r]; e < ptr[r + 1]; ++e)
            masks[static_cast<size_t>(variables[e]) * words + static_cast<size_t>(c / 64)] |=
                uint64_t(1) << (c % 64);
        color[r] = c;
        layers = std::max(layers, c + 1);
    }
    // Stable grouping of the rows by layer.
    std::vector<int32_t> count(static_cast<size_t>(layers) + 1, 0);
    for (int32_t r = 0; r < m; ++r) ++count[color[r] + 1];
    for (int32_t l = 0; l < layers; ++l) count[l + 1] += count[l];
    std::vector<int32_t> order(static_cast<size_t>(m));
    {
        std::vector<int32_t> next(count.begin(), count.end() - 1);
        for (int32_t r = 0; r < m; ++r) order[next[color[r]]++] = r;
    }
    row_ptr[0] = 0;
    int64_t out = 0;
    for (int32_t i = 0; i < m; ++i) {
        const int32_t r = order[i];
        for (int64_t e = ptr[r]; e < ptr[r + 1]; ++e) cols[out++] = variables[e];
        row_ptr[i + 1] = static_cast<int32_t>(out);
    }
    for (int32_t l = 0; l <= layers; ++l) layer_ptr[l] = count[l];
    *num_layers = layers;
    return CK_OK;
}

// ---------------------------------------------------------------------------
// Plan
// ---------------------------------------------------------------------------

namespace {

// The circulant structure of a schedule for lifting Z, if it has one: every
// layer is a run of whole base rows (Z consecutive schedule rows whose row
// r has, at edge e, the column j_e Z + (o_e + r) mod Z for one j_e and
// shift o_e), with the block columns j_e strictly increasing along a row.
bool try_qc(const int32_t* row_ptr, const int32_t* cols, const int32_t* layer_ptr, int32_t m,
            int32_t N, int32_t L, int32_t Z, ck_ldpc_plan* plan) {
    if (Z < 2 || m % Z || N % Z) return false;
    for (int32_t l = 0; l < L; ++l)
        if ((layer_ptr[l + 1] - layer_ptr[l]) % Z) return false;
    const int32_t mb = m / Z;
    std::vector<int32_t> eptr(1, 0);
    std::vector<int32_t> blk_col, blk_shift;
    for (int32_t b = 0; b < mb; ++b) {
        const int32_t r0 = b * Z;
        const int32_t e0 = row_ptr[r0];
        const int32_t deg = row_ptr[r0 + 1] - e0;
        for (int32_t e = 0; e < deg; ++e) {
            const int32_t c = cols[e0 + e];
            const int32_t j = c / Z;
            if (e > 0 && j <= blk_col.back() / Z) return false;
            blk_col.push_back(j * Z);
            blk_shift.push_back(c % Z);
        }
        for (int32_t r = 1; r < Z; ++r) {
            const int32_t er = row_ptr[r0 + r];
            if (row_ptr[r0 + r + 1] - er != deg) return false;
            for (int32_t e = 0; e < deg; ++e) {
                const int32_t c = cols[er + e];
                const int32_t want_o = (blk_shift[eptr.back() + e] + r) % Z;
                if (c != blk_col[eptr.back() + e] + want_o) return false;
            }
        }
        eptr.push_back(static_cast<int32_t>(blk_col.size()));
    }
    plan->qc = true;
    plan->Z = Z;
    plan->mb = mb;
    plan->nb = N / Z;
    plan->nnzb = static_cast<int32_t>(blk_col.size());
    plan->h_layer.assign(static_cast<size_t>(L) + 1, 0);
    for (int32_t l = 0; l <= L; ++l) plan->h_layer[l] = layer_ptr[l] / Z;
    plan->h_eptr = eptr;
    plan->h_blk.resize(blk_col.size() * 2);
    // Per circulant: (j Z + shift, (j + 1) Z), so that row r's column is
    // r + first, wrapped back by Z once it reaches the block's end.
    for (size_t i = 0; i < blk_col.size(); ++i) {
        plan->h_blk[2 * i] = blk_col[i] + blk_shift[i];
        plan->h_blk[2 * i + 1] = blk_col[i] + Z;
    }
    return true;
}

// Rows of one layer and degree in an order that spreads the lanes of each
// shared-memory access over the banks: groups of 32 are filled row by row,
// each time with the row of the next kWindow that raises the groups' largest
// bank counts least (then the one meeting the fewest taken banks), the first
// among equals.  cols(r)[e] is edge e's variable.  Each row of the window
// keeps its cost, and a taken row changes that of the few that share one of
// its banks (DVB-S2 normal: 7 ms on the GB300 host, 22 to reckon
// every cost of the window anew).
template <class Cols>
void spread_banks(std::vector<int32_t>& rows, int32_t deg, const Cols& cols) {
    constexpr int kWindow = 128, kIndexBits = 15;
    if (rows.size() > (1u << kIndexBits)) return;  // rows of a layer share no variable: N / 2 at most
    struct Banks {
        uint64_t places[32][kWindow / 64];  // of the window whose row has this bank
        uint32_t count[32], top;
    };
    std::vector<Banks> banks(static_cast<size_t>(deg), Banks{});
    uint32_t key[kWindow];  // cost and index in `rows`: the least is the row to take
    uint8_t place[1u << kIndexBits];  // of a row in the window
    const auto term = [](uint32_t n, uint32_t top) { return n + (n >= top ? 1024u : 0u); };
    const auto bank = [&](uint32_t index, int32_t e) { return static_cast<uint32_t>(cols(rows[index])[e]) & 31u; };
    uint32_t next = 0;
    const auto enter = [&](int i) {
        uint32_t cost = 0;
        for (int32_t e = 0; e < deg; ++e) {
            Banks& s = banks[e];
            const uint32_t b = bank(next, e);
            s.places[b][i / 64] |= uint64_t(1) << i % 64;
            cost += term(s.count[b], s.top);
        }
        key[i] = cost << kIndexBits | next;
        place[next++] = static_cast<uint8_t>(i);
    };
    const auto add = [&](const uint64_t (&places)[kWindow / 64], uint32_t cost) {
        for (int w = 0; w < kWindow / 64; ++w)
            for (uint64_t m = places[w]; m; m &= m - 1) key[64 * w + __builtin_ctzll(m)] += cost << kIndexBits;
    };
    std::vector<int32_t> out;
    out.reserve(rows.size());
    int size = static_cast<int>(std::min<size_t>(kWindow, rows.size()));
    for (int i = 0; i < kWindow; ++i) key[i] = UINT32_MAX;
    for (int i = 0; i < size; ++i) enter(i);
    while (out.size() < rows.size()) {
        if (out.size() % 32 == 0) {
            for (Banks& s : banks) {
                std::fill(s.count, s.count + 32, 0u);
                s.top = 0;
            }
            for (int i = 0; i < size; ++i)
                if (key[i] != UINT32_MAX)
                    key[i] = static_cast<uint32_t>(deg) * term(0, 0) << kIndexBits | (key[i] & ((1u << kIndexBits) - 1));
        }
        uint32_t least = UINT32_MAX;
        for (int i = 0; i < kWindow; ++i) least = std::min(least, key[i]);
        const uint32_t taken = least & ((1u << kIndexBits) - 1);
        const int at = place[taken];
        out.push_back(rows[taken]);
        for (int32_t e = 0; e < deg; ++e) {
            Banks& s = banks[e];
            const uint32_t c = bank(taken, e), was = s.count[c];
            s.places[c][at / 64] &= ~(uint64_t(1) << at % 64);
            if (was < s.top) {
                add(s.places[c], term(was + 1, s.top) - term(was, s.top));
            } else {  // the largest count rises: the other banks that hold it no longer do
                add(s.places[c], 1u);
                for (uint32_t b = 0; b < 32; ++b)
                    if (b != c && s.count[b] == s.top) add(s.places[b], 0u - 1024u);
                ++s.top;
            }
            ++s.count[c];
        }
        key[at] = UINT32_MAX;
        if (next < rows.size()) enter(at);
    }
    rows.swap(out);
}

// The ELL form of a code without circulants (ck_ldpc_ell.cuh), when it has
// one: `smem` bytes of shared memory per block.
void make_ell(const int32_t* row_ptr, const int32_t* cols, const int32_t* layer_ptr, int32_t smem,
              ck_ldpc_plan* plan) {
    const int32_t L = plan->L, N = plan->N;
    if (plan->max_deg > ck::ldpc::kPackedDegree || N > 65535) return;  // places up to N in 16 bits
    // Short codes with rows of up to 8 edges: the CSR rows, of 32 frames per block, are as fast or faster in batches
    // (4 iterations, CSR rows against this form, 1 / 1000 / 5000 frames: N = 130 25 / 27 / 52 against 30 / 53 / 65
    // us, N = 2000 35 / 70 / 233 against 32 / 83 / 242, N = 4000 38 / 102 / 403 against 37 / 114 / 454, N = 5000
    // 52 / 151 / 577 against 37 / 134 / 551).  Longer rows gain at every length (N = 1000, rows of 13: 84 / 93 / 184
    // against 42 / 50 / 135).
    if (plan->max_deg <= 8 && N < 5000) return;
    // Layers are filled up to 32 rows, in the message state and the syndrome test as well: above twice the rows the
    // state outgrows the gain (N = 16200, 400 frames, 4 iterations, layers of 16 / 8 / 4 rows: 78 / 156 / 312 MB of
    // state against 39, and 1.28 / 4.9 / 10.1 ms against the CSR rows' 1.80 / 3.5 / 6.5).
    int64_t filled = 0;
    for (int32_t l = 0; l < L; ++l) filled += (layer_ptr[l + 1] - layer_ptr[l] + 31) / 32 * 32;
    if (filled > 2 * static_cast<int64_t>(plan->m)) return;
    // First row and end of each layer, then an empty one.
    std::vector<int32_t>& range = plan->ell_layer;
    range.clear();
    int32_t rows = 0;
    for (int32_t l = 0; l < L; ++l) {
        const int32_t count = layer_ptr[l + 1] - layer_ptr[l];
        range.push_back(rows);
        range.push_back(rows + count);
        rows += (count + 31) / 32 * 32;
    }
    range.push_back(0);
    range.push_back(0);
    plan->ell_rows = rows;
    // Variables in shared memory: what the tables, a control block and the
    // +inf word leave.
    const int64_t room =
        static_cast<int64_t>(smem) - (static_cast<int64_t>(2 * (L + 1) + rows / 32) * 4 + 127) / 128 * 128 - 128;
    const int64_t fit = room / 128 * 32 - 32;
    if (fit < N / 2) return;
    const int32_t ns = plan->ell_ns = static_cast<int32_t>(std::min<int64_t>(N, fit));
    plan->ell = true;
    const int32_t chunks = (plan->max_deg + 7) / 8;
    std::vector<uint16_t> c16(static_cast<size_t>(chunks) * rows * 8, static_cast<uint16_t>(ns));
    plan->ell_info.assign(static_cast<size_t>(rows) / 32, 0);
    const auto deg_of = [&](int32_t r) { return row_ptr[r + 1] - row_ptr[r]; };
    const auto cols_of = [&](int32_t r) { return cols + row_ptr[r]; };
    std::vector<int32_t> order;
    std::vector<std::vector<int32_t>> by_deg, tail_by_deg;
    for (int32_t l = 0; l < L; ++l) {
        order.clear();
        by_deg.assign(static_cast<size_t>(plan->max_deg) + 1, {});
        tail_by_deg = by_deg;
        for (int32_t r = layer_ptr[l]; r < layer_ptr[l + 1]; ++r)  // columns increase along a row: the last one decides
            (cols[row_ptr[r + 1] - 1] >= ns ? tail_by_deg : by_deg)[deg_of(r)].push_back(r);
        for (int32_t d = plan->max_deg; d >= 2; --d)
            order.insert(order.end(), tail_by_deg[d].begin(), tail_by_deg[d].end());
        for (int32_t d = plan->max_deg; d >= 2; --d) {
            spread_banks(by_deg[d], d, cols_of);
            order.insert(order.end(), by_deg[d].begin(), by_deg[d].end());
        }
        for (size_t g = 0; g < order.size(); g += 32) {
            const size_t at0 = static_cast<size_t>(range[2 * l]) + g;
            const size_t count = std::min<size_t>(32, order.size() - g);
            int32_t top = 0;
            for (size_t i = 0; i < count; ++i) top = std::max(top, deg_of(order[g + i]));
            bool general = false, special = count < 32;
            for (size_t i = 0; i < count; ++i) {
                const int32_t r = order[g + i], d = deg_of(r);
                special |= d != top || cols_of(r)[d - 1] >= ns;
                for (int32_t e = 0; e < d; ++e) {
                    const int32_t c = cols_of(r)[e];
                    general |= c >= ns && e < top - ck::ldpc::kEllTailEdges;
                    c16[(static_cast<size_t>(e / 8) * rows + at0 + i) * 8 + e % 8] =
                        static_cast<uint16_t>(c >= ns ? c + 1 : c);
                }
            }
            plan->ell_info[at0 / 32] =
                static_cast<int32_t>(static_cast<uint32_t>(top) | (general ? ck::ldpc::kEllGeneral : 0u) |
                                     (special ? ck::ldpc::kEllSpecial : 0u));
        }
    }
    plan->ell_cols.resize(c16.size() / 2);
    memcpy(plan->ell_cols.data(), c16.data(), c16.size() * 2);
}

int upload(const std::vector<int32_t>& h, int32_t** d) {
    *d = nullptr;
    if (h.empty()) return CK_OK;
    CK_CUDA(cudaMalloc(d, h.size() * sizeof(int32_t)));
    CK_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    return CK_OK;
}

}  // namespace

namespace {

// Checks a schedule and fills the host side of `plan` (sizes, degree bound,
// circulant structure); touches no device.
int plan_host(const int32_t* row_ptr, const int32_t* cols, const int32_t* layer_ptr, int32_t m, int32_t N,
              int32_t L, ck_ldpc_plan* plan) {
    if (!row_ptr || !cols || !layer_ptr)
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "row_ptr, cols and layer_ptr are required");
    if (m < 1 || N < 1 || L < 1)
        return ck::fail(CK_ERR_INVALID_ARGUMENT,
                        "row_ptr and layer_ptr need at least 2 entries (m=%d, L=%d)", m, L);
    if (row_ptr[0] != 0) return ck::fail(CK_ERR_INVALID_ARGUMENT, "row_ptr[0] must be 0");
    int32_t max_deg = 0;
    for (int32_t r = 0; r < m; ++r) {
        const int32_t d = row_ptr[r + 1] - row_ptr[r];
        if (d < 2)
            return ck::fail(CK_ERR_INVALID_ARGUMENT, "row %d has %d edges; every check needs >= 2",
                            r, d);
        max_deg = std::max(max_deg, d);
    }
    const int32_t E = row_ptr[m];
    for (int32_t e = 0; e < E; ++e)
        if (cols[e] < 0 || cols[e] >= N)
            return ck::fail(CK_ERR_INVALID_ARGUMENT, "cols[%d] = %d out of [0, %d)", e, cols[e], N);
    if (layer_ptr[0] != 0 || layer_ptr[L] != m)
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "layer_ptr must run from 0 to m");
    for (int32_t l = 0; l < L; ++l)
        if (layer_ptr[l + 1] <= layer_ptr[l])
            return ck::fail(CK_ERR_INVALID_ARGUMENT, "layer %d is empty or decreasing", l);
    // Rows of a layer must share no variable: the decoder updates them at once.
    {
        std::vector<int32_t> owner(static_cast<size_t>(N), -1);
        for (int32_t l = 0; l < L; ++l)
            for (int32_t r = layer_ptr[l]; r < layer_ptr[l + 1]; ++r)
                for (int32_t e = row_ptr[r]; e < row_ptr[r + 1]; ++e) {
                    if (owner[cols[e]] == l)
                        return ck::fail(CK_ERR_INVALID_ARGUMENT,
                                        "rows of layer %d share variable %d", l, cols[e]);
                    owner[cols[e]] = l;
                }
    }
    // Edges of a row in increasing column order (as LDPCCode stores them).
    for (int32_t r = 0; r < m; ++r)
        for (int32_t e = row_ptr[r] + 1; e < row_ptr[r + 1]; ++e)
            if (cols[e] <= cols[e - 1])
                return ck::fail(CK_ERR_INVALID_ARGUMENT,
                                "the columns of row %d must be increasing", r);
    plan->m = m;
    plan->N = N;
    plan->E = E;
    plan->L = L;
    plan->max_deg = max_deg;
    int32_t max_layer_rows = 0;
    for (int32_t l = 0; l < L; ++l)
        max_layer_rows = std::max(max_layer_rows, layer_ptr[l + 1] - layer_ptr[l]);
    plan->max_layer_rows = max_layer_rows;

    // Lifting: the largest Z dividing N and every layer's row count for
    // which the circulant pattern holds.
    int32_t g = N;
    for (int32_t l = 0; l < L; ++l) g = std::gcd(g, layer_ptr[l + 1] - layer_ptr[l]);
    for (int32_t Z = g; Z >= 2 && !plan->qc; --Z) {
        if (g % Z) continue;
        if (m / Z > ck::kMaxBaseRows) break;
        try_qc(row_ptr, cols, layer_ptr, m, N, L, Z, plan);
    }
    if (plan->qc && plan->nnzb > ck::kMaxBlocks) plan->qc = false;
    return CK_OK;
}

}  // namespace

extern "C" int ck_ldpc_plan_create(const int32_t* row_ptr, const int32_t* cols,
                                   const int32_t* layer_ptr, int32_t m, int32_t N, int32_t L,
                                   ck_ldpc_plan** out) {
    ck::clear_error();
    if (!out) return ck::fail(CK_ERR_INVALID_ARGUMENT, "plan is NULL");
    *out = nullptr;
    static std::atomic<uint64_t> next_id{1};
    ck_ldpc_plan* plan = new ck_ldpc_plan();
    plan->id = next_id.fetch_add(1);
    int status = plan_host(row_ptr, cols, layer_ptr, m, N, L, plan);
    if (status == CK_OK) status = ck::cuda_check(cudaGetDevice(&plan->device), "cudaGetDevice");
    if (status != CK_OK) {
        delete plan;
        return status;
    }
    if (plan->qc) {
        status = upload(plan->h_layer, &plan->d_layer);
        if (status == CK_OK) status = upload(plan->h_eptr, &plan->d_eptr);
        if (status == CK_OK) status = upload(plan->h_blk, &plan->d_blk);
    } else {
        int smem = 0;
        status = ck::cuda_check(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, plan->device),
                                "cudaDeviceGetAttribute");
        if (status == CK_OK) make_ell(row_ptr, cols, layer_ptr, smem, plan);
        plan->h_layer.assign(layer_ptr, layer_ptr + L + 1);
        if (status == CK_OK && plan->ell) {
            status = upload(plan->ell_layer, &plan->d_ell_layer);
            if (status == CK_OK) status = upload(plan->ell_cols, &plan->d_ell_cols);
            if (status == CK_OK) status = upload(plan->ell_info, &plan->d_ell_info);
        }
        std::vector<int32_t> rp(row_ptr, row_ptr + m + 1), cc(cols, cols + plan->E);
        if (status == CK_OK) status = upload(plan->h_layer, &plan->d_layer);
        if (status == CK_OK) status = upload(rp, &plan->d_eptr);
        if (status == CK_OK) status = upload(cc, &plan->d_cols);
    }
    if (status != CK_OK) {
        ck_ldpc_plan_destroy(plan);
        return status;
    }
    plan->divZ = ck::FastDiv::make(static_cast<uint32_t>(plan->qc ? plan->Z : 1));
    *out = plan;
    return CK_OK;
}

extern "C" int ck_ldpc_specialised_source(const int32_t* row_ptr, const int32_t* cols,
                                          const int32_t* layer_ptr, int32_t m, int32_t N, int32_t L,
                                          int32_t form, char* out, size_t capacity, size_t* length) {
    ck::clear_error();
    if (!length) return ck::fail(CK_ERR_INVALID_ARGUMENT, "length is NULL");
    if (form < 0 || form > 3) return ck::fail(CK_ERR_INVALID_ARGUMENT, "form must be 0, 1, 2 or 3");
    ck_ldpc_plan plan;
    CK_TRY(plan_host(row_ptr, cols, layer_ptr, m, N, L, &plan));
    if (!plan.qc) return ck::fail(CK_ERR_UNSUPPORTED, "the schedule has no circulant structure");
    if (plan.max_deg > ck::ldpc::kPackedDegree)
        return ck::fail(CK_ERR_UNSUPPORTED,
                        "rows of %d edges: codes with rows above %d edges run the any-degree kernels, "
                        "which have no code-specialised form", plan.max_deg, ck::ldpc::kPackedDegree);
    const int dmax = ck::ldpc::kernel_dmax(true, plan.max_deg);
    const ck_ldpc_plan* plans[1] = {&plan};
    const int parts[1] = {form == 2 ? 2 : 1};  // form 2: two threads per row slot, else one
    const int edges[1] = {form == 3 ? 1 : 0};  // form 3: one message per edge in shared memory
    const std::string src = form == 0 ? ck::ldpc::specialised_source(plan, dmax)
                                      : ck::ldpc::mixed_source(plans, parts, edges, 1, dmax);
    *length = src.size();
    if (out && capacity > 0) {
        const size_t n = std::min(capacity - 1, src.size());
        memcpy(out, src.data(), n);
        out[n] = '\0';
    }
    return CK_OK;
}

extern "C" int ck_ldpc_plan_destroy(ck_ldpc_plan* plan) {
    if (!plan) return CK_OK;
    int dev = -1;
    (void)cudaGetDevice(&dev);
    if (dev != plan->device) (void)cudaSetDevice(plan->device);
    if (plan->d_layer) (void)cudaFree(plan->d_layer);
    if (plan->d_eptr) (void)cudaFree(plan->d_eptr);
    if (plan->d_blk) (void)cudaFree(plan->d_blk);
    if (plan->d_cols) (void)cudaFree(plan->d_cols);
    if (plan->d_ell_layer) (void)cudaFree(plan->d_ell_layer);
    if (plan->d_ell_cols) (void)cudaFree(plan->d_ell_cols);
    if (plan->d_ell_info) (void)cudaFree(plan->d_ell_info);
    ck::ldpc::forget_plan_kernels(plan);
    if (dev >= 0 && dev != plan->device) (void)cudaSetDevice(dev);
    delete plan;
    return CK_OK;
}

extern "C" int ck_ldpc_plan_get_info(const ck_ldpc_plan* plan, ck_ldpc_plan_info* info) {
    if (!plan || !info) return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL argument");
    info->quasi_cyclic = plan->qc ? 1 : 0;
    info->lifting = plan->qc ? plan->Z : 0;
    info->base_rows = plan->qc ? plan->mb : 0;
    info->base_cols = plan->qc ? plan->nb : 0;
    info->blocks = plan->qc ? plan->nnzb : 0;
    info->num_checks = plan->m;
    info->num_variables = plan->N;
    info->num_edges = plan->E;
    info->num_layers = plan->L;
    info->max_row_degree = plan->max_deg;
    info->device = plan->device;
    return CK_OK;
}

extern "C" int ck_ldpc_plan_set_launch(ck_ldpc_plan* plan, const ck_ldpc_launch* launch) {
    ck::clear_error();
    if (!plan || !launch) return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL argument");
    const int32_t T = launch->threads_per_frame, G = launch->frames_per_block;
    if (T != 0 && (T < 32 || T > 1024 || T % 32))
        return ck::fail(CK_ERR_INVALID_ARGUMENT,
                        "threads_per_frame must be 0 or a multiple of 32 in [32, 1024], got %d", T);
    if (G < 0 || (T > 0 && G > 0 && T * G > 1024))
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "frames_per_block %d too large", G);
    if (T > 32 && G > ck::kMaxNamedGroups)
        return ck::fail(CK_ERR_INVALID_ARGUMENT,
                        "at most %d multi-warp frames per block (named barriers)",
                        ck::kMaxNamedGroups);
    if (launch->placement < CK_LDPC_PLACE_AUTO || launch->placement > CK_LDPC_PLACE_EDGES)
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "unknown placement %d", launch->placement);
    plan->launch = *launch;
    return CK_OK;
}

extern "C" int ck_ldpc_plan_set_specialise(ck_ldpc_plan* plan, int32_t mode) {
    ck::clear_error();
    if (!plan) return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL plan");
    if (mode != CK_LDPC_SPECIALISE_AUTO && mode != CK_LDPC_SPECIALISE_OFF && mode != CK_LDPC_SPECIALISE_ON)
        return ck::fail(CK_ERR_INVALID_ARGUMENT, "unknown specialisation mode %d", mode);
    plan->jit_mode = mode;
    return CK_OK;
}

extern "C" int ck_ldpc_plan_get_specialise(const ck_ldpc_plan* plan, int32_t* mode, int32_t* state) {
    ck::clear_error();
    if (!plan || !mode || !state) return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL argument");
    std::lock_guard<std::mutex> lock(plan->jit_mu);
    *mode = plan->jit_mode;
    *state = 0;
    for (const ck_ldpc_plan::Jit& j : plan->jit) {
        if (j.lib) *state = 1;
        if (*state == 1 || !j.tried) continue;
        *state = -1;
        (void)ck::fail(CK_ERR_UNSUPPORTED, "%s", j.why.c_str());
    }
    return CK_OK;
}

extern "C" int ck_ldpc_plan_get_launch(const ck_ldpc_plan* plan, ck_ldpc_launch* launch) {
    if (!plan || !launch) return ck::fail(CK_ERR_INVALID_ARGUMENT, "NULL argument");
    *launch = plan->launch;
    return CK_OK;
}
