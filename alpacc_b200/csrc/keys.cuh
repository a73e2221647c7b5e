// Pair ids and tile sums from terminals, for the grammars whose tables fit shared memory
// (build_key_tables says which; parse_pairs_kernel takes the others and the shards).
//
// A position's pair depends on the window of its q terminals before, itself and k - 1 after,
// cut at its document's ⊢ and ⊣.  The cut is in the tables: the window as it stands in memory
// is split into a left part (up to the position's own terminal) and a right part, each with a
// number for its class (left parts with the same pairs under every right part, and the other
// way round: json's 225 x 225 windows are 63 x 56 records, sexp's 49 are 16), and the record
// at (left class, right class) holds all that the pair adds up to, its id and whether the
// position is a ⊢.  So a position costs one or two 16-bit and one 8-byte load from shared memory, no
// comparison with the sentinels and no load from a key table in global memory.
//
// A warp takes a tile by itself, 8 positions a lane at a time, so there is no barrier: the
// terminals next to a lane's come from its neighbours by shuffles, and sums of up to 31 a
// position (the compact tables' limit) are added as bytes, four fields a word.  The eight
// positions with a ⊢ among them (rare but for batches of tiny documents) take the segmented
// sums.  Memory traffic is 4 B a position.
//
// At 256 MiB of json (37.5 M positions, 23 us of traffic at the measured copy rate) 230 -> 70
// us against parse_pairs_kernel, 38 -> 18 us at 32 MB, in batches of 13 KB documents 232 ->
// 72; up to 4 MB both are launch and latency, 12 us.
// The shared-memory pipe bounds it: two loads a position with a few lanes on one bank.
#pragma once

#include <map>
#include <string>

#include "parser.cuh"

namespace alp {

constexpr int KW_THREADS = 256;
constexpr int KW_ITEMS = 8;                   // positions of a lane at a time
constexpr int KW_STEP = 32 * KW_ITEMS;        // positions of a warp at a time
constexpr int KW_MAX_REC = 4096;              // records (32 KiB of shared memory)
constexpr int KW_MAX_PART = 8192;             // windows of a part (16 KiB)
constexpr long long KW_MAX_SPACE = 1 << 18;   // windows the tables are built from
constexpr uint32_t KW_BIAS = 15;              // depths are in [-15, 15]
constexpr uint32_t KW_HEAD = 1u << 8;

// rec.x: productions | terminal productions << 8 | rights << 16 | lefts << 24
// rec.y: depth change + KW_BIAS | ⊢ << 8 | pair id << 16
struct KeyTables {
    const uint16_t* row;  // [n_row] left part -> class * right classes
    const uint16_t* col;  // [n_col] right part -> class
    const uint2* rec;
    int n_row, n_col, n_rec;
};

struct KeyHost {
    std::vector<uint16_t> row, col;
    std::vector<uint32_t> rec;
};

// False: the general kernel (other lookarounds, a pair past the packed fields, tables past
// shared memory).
inline bool build_key_tables(const ParseHost& p, KeyHost& h) {
    const int q = p.q, k = p.k;
    if (!((q == 1 && k >= 1 && k <= 3) || (q == 2 && (k == 1 || k == 2)))) return false;
    const uint32_t T = p.T;
    if (p.key_space > KW_MAX_SPACE || p.pairs.size() >= 0xffffu) return false;
    size_t nl = 1, nr = 1;
    for (int i = 0; i <= q; ++i) nl *= T;
    for (int i = 1; i < k; ++i) nr *= T;
    if (nl > (size_t)KW_MAX_PART || nr > (size_t)KW_MAX_PART || (long long)(nl * nr) != p.key_space) return false;
    for (const PairInfo& x : p.pairs) {
        const uint32_t lefts = pair_lefts(x);
        if (x.n_prod > 31 || x.n_term > 31 || lefts > 15 || x.n_br - lefts > 15u) return false;
    }
    // the pair (and ⊢) of every window as it stands in memory
    std::vector<uint32_t> m(nl * nr);
    for (size_t l = 0; l < nl; ++l) {
        uint32_t t[8];
        size_t v = l;
        for (int j = q; j >= 0; --j) { t[j] = (uint32_t)(v % T); v /= T; }
        const uint32_t c = t[q];
        size_t xl = c, pw = T;
        bool ok = c != p.start;
        for (int j = q - 1; j >= 0; --j) {
            xl += pw * (ok ? t[j] : p.empty);
            pw *= T;
            ok = ok && t[j] != p.start;
        }
        for (size_t r = 0; r < nr; ++r) {
            uint32_t u[8];
            v = r;
            for (int j = k - 2; j >= 0; --j) { u[j] = (uint32_t)(v % T); v /= T; }
            size_t xr = 0;
            ok = c != p.end;
            for (int j = 0; j < k - 1; ++j) {
                xr = xr * T + (ok ? u[j] : p.empty);
                ok = ok && u[j] != p.end;
            }
            m[l * nr + r] = p.key_index[xl * nr + xr] | (c == p.start ? 0x10000u : 0u);
        }
    }
    std::map<std::string, uint32_t> seen;
    std::vector<size_t> first;  // a left part of each class
    std::vector<uint32_t> rc(nl);
    for (size_t l = 0; l < nl; ++l) {
        auto at = seen.emplace(std::string(reinterpret_cast<const char*>(&m[l * nr]), nr * 4), (uint32_t)seen.size());
        if (at.second) first.push_back(l);
        rc[l] = at.first->second;
    }
    seen.clear();
    std::vector<size_t> cfirst;
    h.col.resize(nr);
    std::string s(first.size() * 4, '\0');
    for (size_t r = 0; r < nr; ++r) {
        for (size_t i = 0; i < first.size(); ++i) memcpy(&s[4 * i], &m[first[i] * nr + r], 4);
        auto at = seen.emplace(s, (uint32_t)seen.size());
        if (at.second) cfirst.push_back(r);
        h.col[r] = (uint16_t)at.first->second;
    }
    const size_t nc = cfirst.size();
    if (first.size() * nc > (size_t)KW_MAX_REC) return false;
    h.row.resize(nl);
    for (size_t l = 0; l < nl; ++l) h.row[l] = (uint16_t)(rc[l] * nc);
    h.rec.resize(2 * first.size() * nc);
    for (size_t i = 0; i < first.size(); ++i)
        for (size_t c = 0; c < nc; ++c) {
            const uint32_t w = m[first[i] * nr + cfirst[c]], id = w & 0xffffu;
            uint32_t x = 0, y = KW_BIAS | ((w >> 16) ? KW_HEAD : 0u) | (id << 16);
            if (id != NO_PAIR) {
                const PairInfo& pi = p.pairs[id];
                const uint32_t lefts = pair_lefts(pi);
                x = pi.n_prod | ((uint32_t)pi.n_term << 8) | ((pi.n_br - lefts) << 16) | (lefts << 24);
                y += (uint32_t)(int32_t)pi.d_depth;
            }
            h.rec[2 * (i * nc + c)] = x;
            h.rec[2 * (i * nc + c) + 1] = y;
        }
    return true;
}

struct KeyArgs {
    KeyTables t;
    const uint16_t* P;
    uint16_t* pid;
    PosSums* tile_sums;
    long long L;
    const long long* dL;  // when set: the position count (L is then its capacity)
    uint32_t T, empty;
};

__host__ __device__ inline size_t keys_smem_bytes(int n_rec, int n_row, int n_col) {
    return (size_t)n_rec * 8 + (((size_t)n_row + n_col) * 2 + 7) / 8 * 8;
}

// Q and K as in parse_pairs_kernel, Q <= 2 and K <= 3.
template <int Q, int K>
__global__ void __launch_bounds__(KW_THREADS) parse_keys_kernel(KeyArgs a) {
    static_assert(Q >= 1 && Q <= 2 && K >= 1 && K <= 3, "a neighbour's word holds two terminals");
    static_assert(PP_TILE % KW_STEP == 0, "whole steps");
    extern __shared__ __align__(16) uint8_t smem[];
    uint2* s_rec = reinterpret_cast<uint2*>(smem);
    uint16_t* s_row = reinterpret_cast<uint16_t*>(s_rec + a.t.n_rec);
    uint16_t* s_col = s_row + a.t.n_row;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < a.t.n_rec; i += KW_THREADS) s_rec[i] = a.t.rec[i];
    for (int i = tid; i < a.t.n_row; i += KW_THREADS) s_row[i] = a.t.row[i];
    for (int i = tid; i < a.t.n_col; i += KW_THREADS) s_col[i] = a.t.col[i];
    after_prior_kernel();
    a.L = position_count(a.L, a.dL);
    __syncthreads();
    const long long L = a.L, n_tiles = (L + PP_TILE - 1) / PP_TILE;
    const uint32_t T = a.T, EE = a.empty | (a.empty << 16);
    auto two = [&](long long i) -> uint32_t {  // the terminals at i and i + 1
        return (i >= 0 && i < L ? (uint32_t)a.P[i] : a.empty) | ((i + 1 >= 0 && i + 1 < L ? (uint32_t)a.P[i + 1] : a.empty) << 16);
    };
    auto eight = [&](long long i) -> uint4 {
        if (i + KW_ITEMS <= L) return *reinterpret_cast<const uint4*>(a.P + i);
        if (i >= L) return make_uint4(EE, EE, EE, EE);
        return make_uint4(two(i), two(i + 2), two(i + 4), two(i + 6));
    };
    for (long long tile = (long long)warp * gridDim.x + blockIdx.x; tile < n_tiles;
         tile += (long long)gridDim.x * (KW_THREADS / 32)) {
        const long long base = tile * PP_TILE;
        uint4 w = eight(base + lane * KW_ITEMS), w1 = eight(base + KW_STEP + lane * KW_ITEMS);
        uint4 w2 = eight(base + 2 * KW_STEP + lane * KW_ITEMS);
        uint32_t carry = two(base - 2);                  // the terminals before the warp's
        const uint32_t after = two(base + PP_TILE);      // and those after the tile
        uint32_t lefts = 0;                              // of the position before the warp's
        if (base > 0) {
            uint32_t r = 0, c = 0;
#pragma unroll
            for (int j = Q; j >= 0; --j) r = r * T + (base - 1 - j >= 0 ? (uint32_t)a.P[base - 1 - j] : a.empty);
#pragma unroll
            for (int j = 0; j < K - 1; ++j) c = c * T + (base + j < L ? (uint32_t)a.P[base + j] : a.empty);
            lefts = s_rec[s_row[r] + (K > 1 ? s_col[c] : 0u)].x >> 24;
        }
        PosSums tot;
        possums_zero(tot);
        uint32_t nt = 0, brs = 0, cls = 0;  // this lane's: productions | terminals << 16, ...
        int32_t depth = 0;
        auto flush = [&]() {
            PosSums x;
            x.nodes = __reduce_add_sync(ALP_FULL_MASK, nt & 0xffffu);
            x.terms = __reduce_add_sync(ALP_FULL_MASK, nt >> 16);
            x.brs = __reduce_add_sync(ALP_FULL_MASK, brs);
            x.cls = __reduce_add_sync(ALP_FULL_MASK, cls);
            x.depth = __reduce_add_sync(ALP_FULL_MASK, depth);
            x.dnodes = x.nodes;
            x.v = 0;
            x.heads = 0;
            x.hpos = -1;
            tot = ps_combine(tot, x);
            nt = brs = cls = 0;
            depth = 0;
        };
#pragma unroll 1
        for (int step = 0; step < PP_TILE / KW_STEP; ++step) {
            const long long at = base + step * KW_STEP, i0 = at + lane * KW_ITEMS;
            if (at >= L) break;
            uint32_t up = __shfl_up_sync(ALP_FULL_MASK, w.w, 1);
            if (lane == 0) up = carry;
            carry = __shfl_sync(ALP_FULL_MASK, w.w, 31);
            uint32_t dn = 0;
            if (K > 1) {
                dn = __shfl_down_sync(ALP_FULL_MASK, w.x, 1);
                const uint32_t nx = __shfl_sync(ALP_FULL_MASK, w1.x, 0);
                if (lane == 31) dn = step == PP_TILE / KW_STEP - 1 ? after : nx;
            }
            // t[j + 2]: the terminal at i0 + j
            const uint32_t t[KW_ITEMS + 4] = {up & 0xffffu, up >> 16, w.x & 0xffffu, w.x >> 16, w.y & 0xffffu, w.y >> 16,
                                              w.z & 0xffffu, w.z >> 16, w.w & 0xffffu, w.w >> 16, dn & 0xffffu, dn >> 16};
            uint32_t two_at[KW_ITEMS + 2];  // number of the terminals at i0 + j - 1 and i0 + j
#pragma unroll
            for (int j = 0; j < KW_ITEMS + (K == 3 ? 2 : 0); ++j) two_at[j] = t[j + 1] * T + t[j + 2];
            uint2 r[KW_ITEMS];
#pragma unroll
            for (int j = 0; j < KW_ITEMS; ++j) {
                uint32_t x = s_row[Q == 2 ? t[j] * T * T + two_at[j] : two_at[j]];
                if (K == 2) x += s_col[t[j + 3]];
                if (K == 3) x += s_col[two_at[j + 2]];
                r[j] = s_rec[x];
            }
            if (at + KW_STEP > L) {
#pragma unroll
                for (int j = 0; j < KW_ITEMS; ++j)
                    if (i0 + j >= L) r[j] = make_uint2(0, KW_BIAS | ((uint32_t)NO_PAIR << 16));
            }
            if (i0 + KW_ITEMS <= L) {
                *reinterpret_cast<uint4*>(a.pid + i0) =
                    make_uint4(__byte_perm(r[0].y, r[1].y, 0x7632), __byte_perm(r[2].y, r[3].y, 0x7632),
                               __byte_perm(r[4].y, r[5].y, 0x7632), __byte_perm(r[6].y, r[7].y, 0x7632));
            } else {
#pragma unroll
                for (int j = 0; j < KW_ITEMS; ++j)
                    if (i0 + j < L) a.pid[i0 + j] = (uint16_t)(r[j].y >> 16);
            }
            uint32_t sx = 0, sy = 0, c = 0;
#pragma unroll
            for (int j = 0; j < KW_ITEMS; ++j) {
                sx += r[j].x;  // fields of at most 31, eight of them: no carry between bytes
                sy += r[j].y;
                if (j > 0) c += min(r[j - 1].x >> 24, (r[j].x >> 16) & 0xffu);
            }
            uint32_t lp = __shfl_up_sync(ALP_FULL_MASK, r[KW_ITEMS - 1].x >> 24, 1);
            if (lane == 0) lp = lefts;
            lefts = __shfl_sync(ALP_FULL_MASK, r[KW_ITEMS - 1].x >> 24, 31);
            if (!__any_sync(ALP_FULL_MASK, (sy >> 8) & 0xfu)) {
                cls += c + min(lp, (r[0].x >> 16) & 0xffu);
                nt += (sx & 0xffu) | ((sx & 0xff00u) << 8);
                brs += ((sx >> 16) & 0xffu) + (sx >> 24);
                depth += (int32_t)(sy & 0xffu) - (int32_t)(KW_ITEMS * KW_BIAS);
            } else {
                flush();
                PosSums acc;
                possums_zero(acc);
#pragma unroll
                for (int j = 0; j < KW_ITEMS; ++j) {
                    PosSums e;
                    possums_zero(e);
                    const uint32_t nr = (r[j].x >> 16) & 0xffu, nl = r[j].x >> 24;
                    e.nodes = e.dnodes = r[j].x & 0xffu;
                    e.terms = (r[j].x >> 8) & 0xffu;
                    e.brs = nr + nl;
                    e.depth = (int32_t)(r[j].y & 0xffu) - (int32_t)KW_BIAS;
                    if (r[j].y & KW_HEAD) {
                        e.heads = 1;
                        e.hpos = (int32_t)(i0 + j);
                    } else {
                        e.cls = min(lp, nr);
                    }
                    lp = nl;
                    acc = ps_combine(acc, e);
                }
                tot = ps_combine(tot, ps_shfl(ps_warp_scan(acc, lane), 31));
            }
            w = w1;
            w1 = w2;
            w2 = step + 3 < PP_TILE / KW_STEP ? eight(i0 + 3 * KW_STEP) : make_uint4(EE, EE, EE, EE);
        }
        flush();
        if (lane == 0) a.tile_sums[tile] = tot;
    }
}

inline const void* keys_kernel_for(int q, int k) {
    if (q == 1 && k == 1) return (const void*)parse_keys_kernel<1, 1>;
    if (q == 1 && k == 2) return (const void*)parse_keys_kernel<1, 2>;
    if (q == 1 && k == 3) return (const void*)parse_keys_kernel<1, 3>;
    if (q == 2 && k == 1) return (const void*)parse_keys_kernel<2, 1>;
    return (const void*)parse_keys_kernel<2, 2>;
}

}  // namespace alp
