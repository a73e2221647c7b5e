// The tree of a token sequence in one pass over its positions (sm_100a).
//
// parse_tree_kernel does for a tile of PP_TILE positions what the general form
// (parse_expand_kernel, two ple_tile_kernel passes) does in three: the segmented
// copies of productions and brackets (futhark/parser.fut:216-233), node tags and
// terminal spans (lines 305-329), the bracket check (lines 153-184) and the
// parents (lines 286-298), which are both "previous smaller-or-equal" searches
// (lines 72-108).
//
// One search serves both.  A position pops its rights from the parser's stack and pushes
// its lefts.  Every popped symbol becomes a node of the position (its production), and a
// pushed symbol is a child that a production of its own position still waits for.  So a
// node's parent is either in its own pair, a fixed distance away (a table entry), or the
// production whose left its right matches: the r-th right and the r-th node without a
// parent in the pair belong together (build_tree_tables checks that this holds for every
// pair of the grammar; the general kernels take the others).  The right that leaves depth
// d matches the left pushed onto depth d: at the last earlier position with lefts whose
// depth after its rights is D <= d, its left number d - D.  json: 1.06 searches a position
// where nodes and brackets apart need 1.93 and 1.06.
//
// The search is near first: a position against the thread's own earlier ones and the four
// of the thread before (90 % of json's), each lane for itself.  The rest, and the rights
// after a position's first, go through a queue of the warp, 32 at a time: the warp's
// earlier threads by runs of minima in registers, then earlier warps by a tree of minima
// in shared memory.  What the tile cannot answer goes to a list in the tile's own part of
// a global array (no global counter), and tree_escape_kernel answers it from earlier
// tiles' minima and staircases (the positions whose D is strictly below every later one
// of their tile).
//
// Nodes are then emitted as in parse_expand_kernel: the owners of a window of nodes in
// shared memory, one node per thread and step, coalesced stores; the parent is written
// with the other fields, so that no node value, bracket or staircase of nodes passes
// through memory.
#pragma once
#include "common.cuh"
#include "parser.cuh"

namespace alp {

// A pair: x = nodes | lefts << 8 | rights << 12 | terminal nodes << 16; y = first
// production record | first stack entry << 16.  Record n_pairs stands for "no pair".
// A production record: x = tag | kind << 16 (a terminal production's terminal and 1,
// else the production and 0; `plain`: always the production); y = terminal nodes before
// it in the pair | parent code << 24: the distance to the parent inside the pair, or
constexpr uint32_t TR_FIRST = 0xffu;  // the node of the pair's first right: parent kept per position
constexpr uint32_t TR_OTHER = 0xfeu;  // of a later right: stored by the search
// A stack entry: symbol | node << 16: of a right the node that its symbol becomes, of a
// left the node that waits for its symbol, TR_ROOT for the start symbol itself (pushed at
// ⊢; its node is the root) and TR_END for the end marker below it (popped at ⊣, no node).
constexpr uint32_t TR_ROOT = 0xffu;
constexpr uint32_t TR_END = 0xfeu;
constexpr uint32_t TR_NO_NODE = 0xffffu;  // a listed search: no node takes its answer
constexpr int TR_NONE = INT32_MAX;

// Whether a search that its tile cannot answer is listed for tree_escape_kernel: the right
// leaves depth d, `node` is the node that takes the answer, or TR_NO_NODE.  A tile's list has
// room for its nodes and one more.  Entries with a node pay for themselves.  Without one there
// is only the ⊣ that pops the end marker: from depth 0 or more its left lies in its own
// document, so only the document that the tile continues lists it, once; below depth 0 no left
// can match and the position has rejected its document already.  (A batch of documents such
// as json's `1 2`, no pair but ⊣'s, would list hundreds a tile where there are no nodes.)
__host__ __device__ inline bool tr_listed(int32_t d, uint32_t node) { return d >= 0 || node != TR_NO_NODE; }

struct TreeTables {
    const uint2* pairs;     // [n_pairs + 1]
    const uint2* rec;       // [n_pseq]
    const uint2* plain;     // [n_pseq]
    const uint32_t* stack;  // [n_stack]
    int n_pairs, n_pseq, n_stack;
};

struct TreeHost {
    std::vector<uint32_t> pairs, rec, plain, stack;
};
// The compact tables from the general ones; false when the grammar is outside their
// ranges (a tile's node count in 16 bits: at most 31 nodes a pair; lefts and rights in 4
// bits, record and stack indices and symbols in 16) or a pair's rights and lefts are not
// its nodes' open ends.  use[i]: 1 pair i stands at positions other than the first, 2 at a
// document's first, which pushes the end marker and the start symbol without a node.
inline bool build_tree_tables(const std::vector<PairInfo>& info, const std::vector<uint8_t>& use,
                              const std::vector<uint32_t>& stack, const std::vector<uint32_t>& pseq,
                              const std::vector<int32_t>& arity, const std::vector<int32_t>& pterm, TreeHost& h) {
    if (pseq.size() > 65535 || stack.size() > 65535 || stack.empty()) return false;
    h.stack.resize(stack.size());
    for (size_t i = 0; i < stack.size(); ++i) {
        if ((stack[i] & 0x7fffffffu) > 0xffffu) return false;
        h.stack[i] = stack[i] & 0xffffu;
    }
    h.rec.assign(2 * pseq.size(), 0);
    for (size_t j = 0; j < pseq.size(); ++j) {
        if (arity[pseq[j]] < 0) return false;
        h.rec[2 * j] = pterm[pseq[j]] >= 0 ? (uint32_t)pterm[pseq[j]] | (1u << 16) : pseq[j];
    }
    h.pairs.assign(2 * (info.size() + 1), 0);
    std::vector<uint8_t> seen(stack.size(), 0);
    uint32_t end_sym = 0x10000u;  // the first left of every ⊢ pair
    for (size_t i = 0; i < info.size(); ++i) {
        if (use[i] != 2) continue;
        if (info[i].n_br < 1) return false;
        const uint32_t e = h.stack[info[i].stack_begin];
        if (end_sym != 0x10000u && e != end_sym) return false;
        end_sym = e;
    }
    for (size_t i = 0; i < info.size(); ++i) {
        const PairInfo& p = info[i];
        int nl = 0, nr = 0;
        for (int j = 0; j < p.n_br; ++j) {
            const bool left = stack[p.stack_begin + j] >> 31;
            if (!left && nl) return false;  // a right after a left
            (left ? nl : nr) += 1;
        }
        if (p.n_prod > 31 || nl > 15 || nr > 15 || use[i] == 3) return false;
        const bool first = use[i] == 2;
        if (first && nr) return false;
        // the open ends of the pair's nodes, innermost last: the node that waits; the rights'
        // symbols below them, in order
        std::vector<uint32_t> open, right_node;
        if (first) open = {TR_END, TR_ROOT};
        int taken = 0, terms = 0;
        for (int k = 0; k < p.n_prod; ++k) {
            const size_t j = p.prod_begin + (size_t)k;
            uint32_t code;
            if (!open.empty()) {
                const uint32_t par = open.back();
                if (par == TR_END) return false;
                open.pop_back();
                code = par == TR_ROOT ? TR_FIRST : (uint32_t)k - par;  // (the root's parent is itself)
                if (par == TR_ROOT && k != 0) return false;
            } else {
                if (taken == nr) return false;  // a node that no right accounts for
                code = taken == 0 ? TR_FIRST : TR_OTHER;
                if (taken == 0 && k != 0) return false;
                ++taken;
                right_node.push_back((uint32_t)k);
            }
            // (past 15 lefts and a pop by each of 31 nodes the ends cannot become the lefts any more)
            for (int c = 0; c < arity[pseq[j]] && open.size() < 64; ++c) open.push_back((uint32_t)k);
            // pairs of different positions may share records: they must agree
            const uint32_t y = (uint32_t)terms | (code << 24);
            if (h.rec[2 * j + 1] && h.rec[2 * j + 1] != y) return false;
            h.rec[2 * j + 1] = y;
            if (pterm[pseq[j]] >= 0) ++terms;
        }
        if (taken == nr - 1 && (stack[p.stack_begin + nr - 1] & 0x7fffffffu) == end_sym) {
            right_node.push_back(TR_END);  // ⊣ pops the end marker
            ++taken;
        }
        if (taken != nr || (int)open.size() != nl) {
            if (use[i]) return false;
            continue;  // a pair that no key names
        }
        for (int j = 0; j < nr + nl; ++j) {
            const size_t e = p.stack_begin + (size_t)j;
            const uint32_t node = j < nr ? right_node[j] : open[j - nr];
            const uint32_t w = (h.stack[e] & 0xffffu) | (node << 16);
            if (seen[e] && h.stack[e] != w) return false;
            h.stack[e] = w;
            seen[e] = 1;
        }
        h.pairs[2 * i] = (uint32_t)p.n_prod | ((uint32_t)nl << 8) | ((uint32_t)nr << 12) | ((uint32_t)terms << 16);
        h.pairs[2 * i + 1] = p.prod_begin | (p.stack_begin << 16);
    }
    h.plain = h.rec;
    for (size_t j = 0; j < pseq.size(); ++j) h.plain[2 * j] = pseq[j];
    return true;
}

// What a tile leaves for tree_escape_kernel.
struct TreeTile {
    uint32_t node_base;  // its first node
    uint32_t esc;        // searches it could not answer
    uint32_t stair;      // entries of its staircase
    uint32_t pad;
};

struct TreeArgs {
    TreeTables t;
    uint32_t sent_l, sent_r;    // terminals ⊢ and ⊣
    const uint16_t* P;          // [L] terminals (several documents: document boundaries)
    const uint16_t* pid;        // [L] pair per position
    const uint32_t* pstart;     // [L] token spans
    const uint32_t* pend;
    long long L, n_docs;
    const long long* dL;        // when set: the position count (L is then its capacity)
    const PosSums* tile_sums;   // exclusive prefixes
    const long long* tok_off;   // several documents: tokens before each document
    uint32_t* tag;
    uint8_t* kind;
    int64_t* nstart;
    int64_t* nend;
    long long* parent;          // null: no parents (production sequence only)
    long long* node_off;        // [n_docs + 1]
    uint8_t* doc_valid;
    long long cap_nodes;
    int span_cap;
    // searches that leave a tile
    // depth; position in the tile | right << 11 | tile-local node << 16.  A tile's list has
    // room for its nodes and one more (tr_listed): it starts at its first node + its number
    uint2* esc;                 // [esc_cap], cap_nodes + tiles
    long long esc_cap;
    uint2* stair;               // [tiles * PP_TILE] D; position in the tile | first node (tile-local) << 16
    TreeTile* tiles;            // [tiles]
    int32_t* tile_min;          // [tiles] least D
    int32_t* m32;               // over 32 and 1024 tiles
    int32_t* m1024;
};

constexpr int TR_QUEUE = 64;                        // queued searches of a warp at a time
constexpr int TR_LEAVES = PP_THREADS;
constexpr size_t TR_POS_BYTES = 2 * (size_t)PP_TILE * 4;                     // sA, sTok
constexpr size_t TR_X_BYTES = 2 * (size_t)PP_TILE * 4                        // s_D, s_LN
                              + 2 * (size_t)TR_LEAVES * 4                    // tree
                              + (size_t)(PP_THREADS / 32) * TR_QUEUE * 4;    // queues
static_assert(TR_X_BYTES >= 2 * (size_t)EX_WIN + (size_t)PP_TILE * 4, "owners and parents fit the search arrays");
__host__ __device__ inline size_t tree_tables_bytes(int n_pairs, int n_pseq, int n_stack) {
    return (8 * ((size_t)n_pairs + 1) + 8 * (size_t)n_pseq + 4 * (size_t)n_stack + 15) & ~(size_t)15;
}
__host__ __device__ inline size_t tree_smem_bytes(int n_pairs, int n_pseq, int n_stack, bool one) {
    return tree_tables_bytes(n_pairs, n_pseq, n_stack) + TR_POS_BYTES + TR_X_BYTES + (one ? 0 : (size_t)PP_TILE * 4);
}

// fields of a pair's x
__device__ __forceinline__ uint32_t tr_np(uint32_t x) { return x & 31u; }
__device__ __forceinline__ uint32_t tr_nl(uint32_t x) { return (x >> 8) & 15u; }
__device__ __forceinline__ uint32_t tr_nr(uint32_t x) { return (x >> 12) & 15u; }
constexpr uint32_t TR_SUMS = 0x001f001fu;  // nodes | terminal nodes << 16

// last of the first `n` of four values that is <= x, or -1
__device__ __forceinline__ int tr_last4(const int4 v, int n, int32_t x) {
    int c = -1;
    if (n > 0 && v.x <= x) c = 0;
    if (n > 1 && v.y <= x) c = 1;
    if (n > 2 && v.z <= x) c = 2;
    if (n > 3 && v.w <= x) c = 3;
    return c;
}

// The document of a position (several documents: ⊢ tokens ⊣ each) is rejected.
__device__ __noinline__ void tr_reject(const long long* tok_off, long long n_docs, uint8_t* doc_valid, long long pos) {
    long long lo = 0, hi = n_docs - 1;
    while (lo < hi) {
        const long long mid = (lo + hi + 1) >> 1;
        if (tok_off[mid] + 2 * mid <= pos) lo = mid; else hi = mid - 1;
    }
    doc_valid[lo] = 0;
}

// ONE: the positions are one document (its ⊢ is position 0, its ⊣ position L - 1).
//
// Bound by its instruction stream (17 warp instructions a position, 62 % of issue slots);
// of 0.92 ms for 256 MiB of json (37 M positions, 72 M nodes, 2.46 GB) the node windows take
// 0.40, the searches 0.27, sums and records 0.20.  The general kernels take 1.34 ms there
// (0.79 expansion, then 0.37 and 0.21 for the two searches side by side).  2048 positions a
// tile: two CTAs of 512 threads an SM hold the tables twice and the searches stay inside the
// tile for all but 2 % of json's; four positions a thread make the vector loads and stores
// of the shared arrays 16 bytes.
template <bool ONE>
__global__ void __launch_bounds__(PP_THREADS, 2) parse_tree_kernel(TreeArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint2* s_pr = reinterpret_cast<uint2*>(smem);
    uint2* s_rec = s_pr + a.t.n_pairs + 1;
    uint32_t* s_se = reinterpret_cast<uint32_t*>(s_rec + a.t.n_pseq);
    uint8_t* base_pos = smem + tree_tables_bytes(a.t.n_pairs, a.t.n_pseq, a.t.n_stack);
    int32_t* sA = reinterpret_cast<int32_t*>(base_pos);           // first record - first (tile-local) node
    uint32_t* sTok = reinterpret_cast<uint32_t*>(sA + PP_TILE);   // token of the first terminal node
    uint8_t* X = base_pos + TR_POS_BYTES;
    // searching
    int32_t* s_D = reinterpret_cast<int32_t*>(X);                 // depth after the rights (with lefts)
    uint32_t* s_LN = reinterpret_cast<uint32_t*>(s_D + PP_TILE);  // first left's stack entry | first node << 16
    int32_t* tD = reinterpret_cast<int32_t*>(s_LN + PP_TILE);
    uint32_t* s_q = reinterpret_cast<uint32_t*>(tD + 2 * TR_LEAVES);
    // emitting (the same memory)
    uint16_t* s_own = reinterpret_cast<uint16_t*>(X);             // [EX_WIN] owner of each node
    uint32_t* sPar = reinterpret_cast<uint32_t*>(X + 2 * EX_WIN); // parent of a position's first node
    // several documents: first node of each position's document
    uint32_t* s_hd = reinterpret_cast<uint32_t*>(X + TR_X_BYTES);
    uint32_t* s_span = s_hd + (ONE ? 0 : PP_TILE);
    __shared__ uint4 s_w[PP_THREADS / 32];
    __shared__ uint32_t s_st[PP_THREADS / 32];
    __shared__ uint32_t s_en;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = PP_THREADS / 32;
    for (int i = tid; i <= a.t.n_pairs; i += PP_THREADS) s_pr[i] = a.t.pairs[i];
    for (int i = tid; i < a.t.n_pseq; i += PP_THREADS) s_rec[i] = a.t.rec[i];
    for (int i = tid; i < a.t.n_stack; i += PP_THREADS) s_se[i] = a.t.stack[i];
    after_prior_kernel();
    a.L = position_count(a.L, a.dL);
    if ((long long)blockIdx.x * PP_TILE >= a.L) return;  // with dL the grid covers the capacity
    const uint32_t NP = (uint32_t)a.t.n_pairs, last_se = (uint32_t)a.t.n_stack - 1u;
    const long long n_tiles = (a.L + PP_TILE - 1) / PP_TILE;
    // this thread's pair ids (and terminals), one tile ahead
    auto words = [&](long long i0, uint2& w, uint2& t) {
        if (i0 + PP_ITEMS <= a.L) {
            w = __ldg(reinterpret_cast<const uint2*>(a.pid + i0));
            if (!ONE) t = __ldg(reinterpret_cast<const uint2*>(a.P + i0));
        } else {
            uint32_t x[PP_ITEMS], y[PP_ITEMS];
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                x[j] = i0 + j < a.L ? a.pid[i0 + j] : NO_PAIR;
                y[j] = (!ONE && i0 + j < a.L) ? a.P[i0 + j] : 0xffffu;
            }
            w = make_uint2(x[0] | (x[1] << 16), x[2] | (x[3] << 16));
            t = make_uint2(y[0] | (y[1] << 16), y[2] | (y[3] << 16));
        }
    };
    uint2 nw = make_uint2(0, 0), nt = make_uint2(0, 0);
    words((long long)blockIdx.x * PP_TILE + tid * PP_ITEMS, nw, nt);
    for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const long long i0 = tile * PP_TILE + tid * PP_ITEMS;
        const PosSums tp = a.tile_sums[tile];
        uint32_t id[PP_ITEMS] = {nw.x & 0xffffu, nw.x >> 16, nw.y & 0xffffu, nw.y >> 16};
        uint32_t hm = 0, em = 0;  // ⊢ / ⊣ bits of this thread's positions
        if (ONE) {
            if (i0 == 0) hm = 1u;
            if (a.L - 1 >= i0 && a.L - 1 < i0 + PP_ITEMS) em = 1u << (uint32_t)(a.L - 1 - i0);
        } else {
            const uint32_t c[PP_ITEMS] = {nt.x & 0xffffu, nt.x >> 16, nt.y & 0xffffu, nt.y >> 16};
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                if (i0 + j < a.L) {
                    if (c[j] == a.sent_l) hm |= 1u << j;
                    if (c[j] == a.sent_r) em |= 1u << j;
                }
            }
        }
        if (tile + gridDim.x < n_tiles) words(i0 + (long long)gridDim.x * PP_TILE, nw, nt);
        __syncthreads();  // the tables are loaded; the tile before is done with the shared arrays
        uint32_t cnt[PP_ITEMS], beg[PP_ITEMS];
        uint32_t none = 0;  // positions without an admissible pair
#pragma unroll
        for (int j = 0; j < PP_ITEMS; ++j) {
            if (id[j] == NO_PAIR) {
                id[j] = NP;
                if (i0 + j < a.L) none |= 1u << j;
            }
            const uint2 r = s_pr[id[j]];
            cnt[j] = r.x;
            beg[j] = r.y;
        }
        // ---- sums before each thread's positions --------------------------------------
        uint32_t rN, rS, rB;        // ONE: rN = nodes | terminals << 16; else rN nodes, rS terminals |
                                    //   nodes since the last ⊢ << 16; rB depth
        uint32_t tn;                // nodes of the tile
        uint32_t hcount = 0;        // heads before this thread (in the tile)
        bool local = false;         // a head lies before this thread's positions in the tile
        uint32_t lasth = 0;         // its tile position + 1
        uint32_t fh = 0xffffffffu;  // first head of the tile: positions before it continue the
                                    //   document of the tile before (one document: all)
        uint32_t slo, shi;          // the tile's terminal nodes take the spans [slo, shi)
        if (ONE) {
            uint32_t A = 0, B = 0;
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                A += cnt[j] & TR_SUMS;
                B += tr_nl(cnt[j]) - tr_nr(cnt[j]);
            }
            uint32_t iA = A, iB = B;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t oA = __shfl_up_sync(ALP_FULL_MASK, iA, d), oB = __shfl_up_sync(ALP_FULL_MASK, iB, d);
                if (lane >= d) { iA += oA; iB += oB; }
            }
            if (lane == 31) s_w[warp] = make_uint4(iA, iB, 0, 0);
            if (tid == 0) s_en = 0;
            __syncthreads();
            uint4 v = make_uint4(0, 0, 0, 0);
            if (lane < NW) v = s_w[lane];
            const uint32_t pA = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? v.x : 0u);
            const uint32_t pB = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? v.y : 0u);
            const uint32_t tA = __reduce_add_sync(ALP_FULL_MASK, v.x);
            rN = pA + iA - A;
            rB = pB + iB - B;
            rS = 0;
            tn = tA & 0xffffu;
            slo = 1u + tp.terms;
            shi = slo + (tA >> 16);
        } else {
            uint32_t N = 0, S = 0, B = 0;
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                if ((hm >> j) & 1u) { S = 0; B = 0; }
                const uint32_t n = tr_np(cnt[j]);
                N += n;
                S += ((cnt[j] >> 16) & 31u) | (n << 16);
                B += tr_nl(cnt[j]) - tr_nr(cnt[j]);
            }
            const uint32_t any = __ballot_sync(ALP_FULL_MASK, hm != 0);
            const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
            const int seg = (any & le) ? 31 - __clz(any & le) : 0;
            uint32_t iN = N, iS = S, iB = B;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t oN = __shfl_up_sync(ALP_FULL_MASK, iN, d), oS = __shfl_up_sync(ALP_FULL_MASK, iS, d),
                               oB = __shfl_up_sync(ALP_FULL_MASK, iB, d);
                if (lane >= d) iN += oN;
                if (lane - d >= seg) { iS += oS; iB += oB; }
            }
            uint32_t eS = __shfl_up_sync(ALP_FULL_MASK, iS, 1), eB = __shfl_up_sync(ALP_FULL_MASK, iB, 1);
            if (lane == 0) { eS = 0; eB = 0; }
            uint32_t heads = 0, mine_before = 0, last = 0, first = 0;
            if (any) {
#pragma unroll
                for (int j = 0; j < PP_ITEMS; ++j) {
                    const uint32_t b = __ballot_sync(ALP_FULL_MASK, (hm >> j) & 1u);
                    heads += __popc(b);
                    mine_before += __popc(b & lt);
                }
                const int hl = 31 - __clz(any);
                const uint32_t hb = __shfl_sync(ALP_FULL_MASK, hm, hl);
                last = (uint32_t)((warp * 32 + hl) * PP_ITEMS + 31 - __clz(hb)) + 1u;
                const int fl = __ffs(any) - 1;
                first = (uint32_t)((warp * 32 + fl) * PP_ITEMS + __ffs(__shfl_sync(ALP_FULL_MASK, hm, fl)) - 1);
                const int pl = (any & lt) ? 31 - __clz(any & lt) : 0;
                const uint32_t pb = __shfl_sync(ALP_FULL_MASK, hm, pl);
                if (any & lt) lasth = (uint32_t)((warp * 32 + pl) * PP_ITEMS + 31 - __clz(pb)) + 1u;
            }
            if (lane == 31) s_w[warp] = make_uint4(iN, iS, iB, heads | (last << 8) | (first << 20));
            if (tid == 0) s_en = 0;
            __syncthreads();
            uint4 v = make_uint4(0, 0, 0, 0);
            if (lane < NW) v = s_w[lane];
            const uint32_t hw = __ballot_sync(ALP_FULL_MASK, (v.w & 0xffu) != 0);  // warps with heads
            const uint32_t hb4 = hw & ((1u << warp) - 1u);
            const int lw = hb4 ? 31 - __clz(hb4) : 0;
            const bool in = lane < warp && lane >= lw;
            const uint32_t pN = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? v.x : 0u);
            const uint32_t pS = __reduce_add_sync(ALP_FULL_MASK, in ? v.y : 0u);
            const uint32_t pB = __reduce_add_sync(ALP_FULL_MASK, in ? v.z : 0u);
            const uint32_t pH = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? (v.w & 0xffu) : 0u);
            const uint32_t plast = __shfl_sync(ALP_FULL_MASK, (v.w >> 8) & 0xfffu, lw);
            const uint32_t first_of = __shfl_sync(ALP_FULL_MASK, v.w >> 20, hw ? __ffs(hw) - 1 : 0);
            fh = hw ? first_of : (uint32_t)PP_TILE;
            tn = __reduce_add_sync(ALP_FULL_MASK, v.x);
            hcount = pH + mine_before;
            rN = pN + iN - N;
            if (lasth) {
                rS = eS;
                rB = eB;
            } else {
                rS = eS + pS;
                rB = eB + pB;
                if (hb4) lasth = plast;
            }
            local = lasth != 0;
            slo = (uint32_t)tp.hpos + 1u + tp.terms;
            const int tw = hw ? 31 - __clz(hw) : 0;
            const uint32_t tS = __reduce_add_sync(ALP_FULL_MASK, lane >= tw ? (v.y & 0xffffu) : 0u);
            const uint32_t tl = __shfl_sync(ALP_FULL_MASK, (v.w >> 8) & 0xfffu, tw);
            shi = hw ? (uint32_t)(tile * PP_TILE) + tl + tS : slo + tS;
        }
        // ---- the tile's token spans into shared memory while the searches run
        long long sp_lo = 0;
        uint32_t sp_n = 0;
        if (a.span_cap > 0 && ((reinterpret_cast<uintptr_t>(a.pstart) | reinterpret_cast<uintptr_t>(a.pend)) & 15) == 0) {
            const long long lo = (long long)(slo & ~3u), hi = min((long long)shi, a.L);
            if (hi > lo && ((hi - lo + 3) & ~3ll) <= (long long)a.span_cap) {  // the same in every thread
                sp_lo = lo;
                sp_n = (uint32_t)(hi - lo);
                const uint32_t chunks = (sp_n + 3) / 4;
                for (uint32_t c = tid; c < 2 * chunks; c += PP_THREADS) {
                    const bool e = c >= chunks;
                    const uint32_t cc = e ? c - chunks : c;
                    const long long idx = lo + 4 * (long long)cc;
                    ex_cp16(s_span + (e ? a.span_cap : 0) + 4 * cc, (e ? a.pend : a.pstart) + idx,
                            (uint32_t)min(16ll, 4 * (a.L - idx)));
                }
                ex_cp_commit();
            }
        }
        // ---- per position: depths and the rules that one position decides ------------------
        int32_t D[PP_ITEMS], dep[PP_ITEMS];
        uint32_t nof[PP_ITEMS], hd[PP_ITEMS];  // first node (tile-local); doc's first node (several documents)
        {
            int32_t bd = tp.depth;
            uint32_t bt = (ONE ? 0u : (uint32_t)tp.hpos) + 1u + tp.terms, bn = tp.dnodes;
            if (!ONE && local) {
                bd = 0;
                bt = (uint32_t)(tile * PP_TILE) + lasth;  // position of the head + 1
                bn = 0;
            }
            long long doc = ONE ? 0 : (long long)tp.heads + hcount - 1;
            uint32_t tk[PP_ITEMS];
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                const bool head = (hm >> j) & 1u;
                if (!ONE && head) {
                    rS = 0;
                    rB = 0;
                    bd = 0;
                    bt = (uint32_t)(i0 + j) + 1u;
                    bn = 0;
                    ++doc;
                }
                const bool dok = ONE || (doc >= 0 && doc < a.n_docs);
                nof[j] = ONE ? (rN & 0xffffu) : rN;
                tk[j] = bt + (ONE ? (rN >> 16) : (rS & 0xffffu));
                // the document's first node: this one less the nodes since its ⊢
                hd[j] = ONE ? 0u : tp.nodes + nof[j] - (bn + (rS >> 16));
                dep[j] = bd + (int32_t)rB;
                const int32_t nl = (int32_t)tr_nl(cnt[j]), nr = (int32_t)tr_nr(cnt[j]);
                D[j] = nl ? dep[j] - nr : TR_NONE;
                if (i0 + j < a.L) {
                    if (head && dok) a.node_off[doc] = (long long)tp.nodes + nof[j];
                    // no admissible pair; a depth below zero; unbalanced at the end
                    if ((((none >> j) & 1u) || dep[j] < nr || (((em >> j) & 1u) && dep[j] + nl != nr)) && dok)
                        a.doc_valid[doc] = 0;
                }
                if (ONE) {
                    rN += cnt[j] & TR_SUMS;
                } else {
                    const uint32_t n = tr_np(cnt[j]);
                    rN += n;
                    rS += ((cnt[j] >> 16) & 31u) | (n << 16);
                }
                rB += (uint32_t)(nl - nr);
            }
            reinterpret_cast<uint4*>(sTok)[tid] = make_uint4(tk[0], tk[1], tk[2], tk[3]);
        }
        reinterpret_cast<int4*>(sA)[tid] = make_int4((int)(beg[0] & 0xffffu) - (int)nof[0], (int)(beg[1] & 0xffffu) - (int)nof[1],
                                                     (int)(beg[2] & 0xffffu) - (int)nof[2], (int)(beg[3] & 0xffffu) - (int)nof[3]);
        reinterpret_cast<int4*>(s_D)[tid] = make_int4(D[0], D[1], D[2], D[3]);
        {
            uint32_t l[PP_ITEMS];
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) l[j] = ((beg[j] >> 16) + tr_nr(cnt[j])) | (nof[j] << 16);
            reinterpret_cast<uint4*>(s_LN)[tid] = make_uint4(l[0], l[1], l[2], l[3]);
        }
        if (!ONE) reinterpret_cast<uint4*>(s_hd)[tid] = make_uint4(hd[0], hd[1], hd[2], hd[3]);
        const int32_t gD = min(min(D[0], D[1]), min(D[2], D[3]));
        {
            int32_t y = gD;
            int node = TR_LEAVES + tid;
            tD[node] = y;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                y = min(y, __shfl_xor_sync(ALP_FULL_MASK, y, d));
                node >>= 1;
                if ((lane & (2 * d - 1)) == 0) tD[node] = y;
            }
        }
        __syncthreads();
        // ---- the tree's top, and which positions are on the tile's staircase
        uint32_t stairs = 0;
        {
            int32_t y = lane < NW ? tD[NW + lane] : TR_NONE;
            // the minimum of the later warps: a warp whose own is not below it has no entry
            const int32_t aD = __reduce_min_sync(ALP_FULL_MASK, lane > warp ? y : TR_NONE);
            const bool has = __shfl_sync(ALP_FULL_MASK, y, warp) < aD;
            if (warp == 0) {
                int node = NW + lane;
#pragma unroll
                for (int d = 1; d < NW; d <<= 1) {
                    y = min(y, __shfl_xor_sync(ALP_FULL_MASK, y, d));
                    node >>= 1;
                    if (lane < NW && (lane & (2 * d - 1)) == 0) tD[node] = y;
                }
            }
            if (has) {
                int32_t s = gD;  // minimum over this lane and the later ones
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int32_t o = __shfl_down_sync(ALP_FULL_MASK, s, d);
                    if (lane + d < 32) s = min(s, o);
                }
                int32_t run = __shfl_down_sync(ALP_FULL_MASK, s, 1);
                run = lane == 31 ? aD : min(run, aD);
#pragma unroll
                for (int j = PP_ITEMS - 1; j >= 0; --j) {
                    if (D[j] < run) { stairs |= 1u << j; run = D[j]; }
                }
            }
        }
        const uint32_t sc = (uint32_t)__popc(stairs);
        const uint32_t swt = __reduce_add_sync(ALP_FULL_MASK, sc);
        if (lane == 0) s_st[warp] = swt;
        __syncthreads();
        if (swt || warp == 0) {
            const uint32_t v = lane < NW ? s_st[lane] : 0u;
            uint32_t o = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? v : 0u) + warp_scan_add(sc, lane) - sc;
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j)
                if ((stairs >> j) & 1u)
                    a.stair[tile * PP_TILE + o++] = make_uint2((uint32_t)D[j], (uint32_t)(4 * tid + j) | (nof[j] << 16));
            const uint32_t tot = __reduce_add_sync(ALP_FULL_MASK, v);
            if (tid == 0) {
                a.tiles[tile].stair = tot;
                a.tile_min[tile] = tD[1];
            }
        }
        auto reject = [&](int pl) {
            if (ONE) a.doc_valid[0] = 0;
            else tr_reject(a.tok_off, a.n_docs, a.doc_valid, tile * PP_TILE + pl);
        };
        // The right `me` (stack entry) that leaves depth d against its left at position q: the
        // document is rejected when they differ; the parent is the node that waits for it.
        // (An entry past the pair's is read only where a rejected document's depths cross
        // into another document.)
        auto match = [&](int q, int32_t d, uint32_t me, uint32_t head, int pl) -> uint32_t {
            const uint32_t w = s_LN[q];
            const uint32_t left = s_se[min((w & 0xffffu) + (uint32_t)(d - s_D[q]), last_se)];
            if ((left ^ me) & 0xffffu) reject(pl);
            const uint32_t k = left >> 16;
            return k == TR_ROOT ? 0u : tp.nodes + (w >> 16) + k - head;
        };
        // ---- near searches, for the first right of each position
        uint32_t par[PP_ITEMS] = {0, 0, 0, 0};
        uint32_t far = 0;  // not answered here
        {
            const int4 pD = tid > 0 ? reinterpret_cast<const int4*>(s_D)[tid - 1] : make_int4(TR_NONE, TR_NONE, TR_NONE, TR_NONE);
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                const int32_t d = dep[j] - 1;
                int q = tr_last4(pD, 4, d);
#pragma unroll
                for (int i = 0; i < j; ++i)
                    if (D[i] <= d) q = 4 + i;
                if (tr_nr(cnt[j])) {
                    if (q >= 0) par[j] = match(4 * tid - 4 + q, d, s_se[beg[j] >> 16], ONE ? 0u : s_hd[4 * tid + j], 4 * tid + j);
                    else far |= 1u << j;
                }
            }
        }
        // ---- the queue of the warp.  An entry: position in the warp | right << 7 | rights after it
        // << 11 | (depth the right leaves, since the tile's start or the last ⊢ in it) << 16; the parent for a first right comes back in its place
        {
            uint32_t c = __popc(far);
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) c += max(tr_nr(cnt[j]), 1u) - 1u;
            const uint32_t inc = warp_scan_add(c, lane);
            const uint32_t total = __shfl_sync(ALP_FULL_MASK, inc, 31);
            uint32_t* q = s_q + warp * TR_QUEUE;
            int32_t g[5];  // g[k] = the least D of the 2^k threads ending at this one
            g[0] = gD;
            if (total) {
#pragma unroll
                for (int k = 1; k < 5; ++k) g[k] = min(g[k - 1], __shfl_up_sync(ALP_FULL_MASK, g[k - 1], 1 << (k - 1)));
            }
            for (uint32_t b = 0; b < total; b += TR_QUEUE) {
                uint32_t o = inc - c - b;  // entries before this chunk wrap around and are skipped
                uint32_t slot[PP_ITEMS];
#pragma unroll
                for (int j = 0; j < PP_ITEMS; ++j) {
                    slot[j] = o;
                    const uint32_t nr = tr_nr(cnt[j]);
                    for (uint32_t r = (far >> j) & 1u ? 0u : 1u; r < nr; ++r, ++o)
                        if (o < (uint32_t)TR_QUEUE)
                            q[o] = (uint32_t)(lane * PP_ITEMS + j) | (r << 7) | ((nr - 1u - r) << 11) |
                                   ((uint32_t)(dep[j] - ((uint32_t)(4 * tid + j) < fh ? tp.depth : 0) - 1 - (int32_t)r) << 16);
                }
                __syncwarp();
                const uint32_t nq = min(total - b, (uint32_t)TR_QUEUE);
                for (uint32_t e0 = 0; e0 < nq; e0 += 32) {
                    const uint32_t e = e0 + lane;
                    const uint32_t w = e < nq ? q[e] : 0u;
                    const int pl = warp * 128 + (int)(w & 127u);
                    const uint32_t r = (w >> 7) & 15u, r2 = (w >> 11) & 15u;  // its number, and of the rights after it
                    const int32_t d = ((int32_t)w >> 16) + ((uint32_t)pl < fh ? tp.depth : 0);
                    // the warp's earlier threads, by runs: the longest above d are stepped over first
                    int pos = (int)((w & 127u) >> 2) - 1;
#pragma unroll
                    for (int k = 4; k >= 0; --k) {
                        const int32_t v = __shfl_sync(ALP_FULL_MASK, g[k], pos & 31);
                        if (pos >= 0 && v > d) pos -= 1 << k;
                    }
                    if (e < nq) {
                        // the own thread's earlier positions come first
                        int at = tr_last4(reinterpret_cast<const int4*>(s_D)[pl >> 2], pl & 3, d);
                        if (at >= 0) {
                            at += pl & ~3;
                        } else {
                            int grp = pos >= 0 ? warp * 32 + pos : -1;
                            if (grp < 0) {
                                // earlier warps: up the tree from this warp's node, then down
                                int node = NW + warp;
                                while (node > 1 && !((node & 1) && tD[node - 1] <= d)) node >>= 1;
                                if (node > 1) {
                                    --node;
                                    while (node < TR_LEAVES) node = (tD[2 * node + 1] <= d) ? 2 * node + 1 : 2 * node;
                                    grp = node - TR_LEAVES;
                                }
                            }
                            if (grp >= 0) at = 4 * grp + max(tr_last4(reinterpret_cast<const int4*>(s_D)[grp], 4, d), 0);
                        }
                        const uint32_t ln = s_LN[pl];
                        const uint32_t me = s_se[min((ln & 0xffffu) - 1u - r2, last_se)];
                        const uint32_t node = me >> 16 == TR_END ? TR_NO_NODE : (ln >> 16) + (me >> 16);  // tile-local
                        const long long gi = (long long)tp.nodes + node;
                        if (at >= 0) {
                            const uint32_t p = match(at, d, me, ONE ? 0u : s_hd[pl], pl);
                            if (r == 0) q[e] = p;
                            else if (a.parent && node != TR_NO_NODE && gi < a.cap_nodes) a.parent[gi] = (long long)p;
                        } else if (tr_listed(d, node)) {
                            const long long k = (long long)tp.nodes + tile + atomicAdd(&s_en, 1u);
                            if (k < a.esc_cap) a.esc[k] = make_uint2((uint32_t)d, (uint32_t)pl | (r << 11) | (node << 16));
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < PP_ITEMS; ++j)
                    if (((far >> j) & 1u) && slot[j] < (uint32_t)TR_QUEUE) par[j] = q[slot[j]];
                __syncwarp();
            }
        }
        if (sp_n) ex_cp_wait_all();  // this thread's span copies; the barriers below publish them
        __syncthreads();             // the searches are done: their arrays become owners and parents
        if (tid == 0) {
            a.tiles[tile].node_base = tp.nodes;
            a.tiles[tile].esc = (uint32_t)max(0ll, min(a.esc_cap - (long long)tp.nodes - tile, (long long)s_en));
        }
        reinterpret_cast<uint4*>(sPar)[tid] = make_uint4(par[0], par[1], par[2], par[3]);
        // ---- nodes, one window at a time ---------------------------------------------
        const uint32_t lim = (uint32_t)max(0ll, min((long long)tn, a.cap_nodes - (long long)tp.nodes));
        const uint32_t slo_l = (uint32_t)sp_lo;
        uint32_t* o_tag = a.tag + tp.nodes;
        uint8_t* o_kind = a.kind + tp.nodes;
        int64_t* o_start = a.nstart + tp.nodes;
        int64_t* o_end = a.nend + tp.nodes;
        long long* o_par = a.parent ? a.parent + tp.nodes : nullptr;
        for (uint32_t w0 = 0; w0 < lim; w0 += EX_WIN) {
            const uint32_t wn = min(lim - w0, (uint32_t)EX_WIN);
#pragma unroll
            for (int j = 0; j < PP_ITEMS; ++j) {
                const uint32_t b = nof[j], n = tr_np(cnt[j]);
                const uint32_t lo = max(b, w0), hi = min(b + n, w0 + wn);
                for (uint32_t x = lo; x < hi; ++x) s_own[x - w0] = (uint16_t)(tid * PP_ITEMS + j);
            }
            __syncthreads();
#pragma unroll 2
            for (uint32_t e = tid; e < wn; e += PP_THREADS) {
                const uint32_t g = w0 + e;
                const uint32_t pl = s_own[e];
                const uint2 rec = s_rec[(int32_t)g + sA[pl]];
                const uint32_t code = rec.y >> 24;
                uint32_t st = 0, en = 0;
                if (rec.x >> 16) {
                    // the k-th terminal production of a document takes its k-th token's span
                    const uint32_t ti = sTok[pl] + (rec.y & 0xffu);
                    const uint32_t d = ti - slo_l;
                    if (d < sp_n) {
                        st = s_span[d];
                        en = s_span[a.span_cap + d];
                    } else if ((long long)ti < a.L) {
                        st = __ldg(&a.pstart[ti]);
                        en = __ldg(&a.pend[ti]);
                    }
                }
                o_tag[g] = rec.x & 0xffffu;
                o_kind[g] = (uint8_t)(rec.x >> 16);
                o_start[g] = (int64_t)st;
                o_end[g] = (int64_t)en;
                if (o_par && code != TR_OTHER)
                    o_par[g] = code == TR_FIRST ? (long long)sPar[pl] : (long long)(tp.nodes + g - code - (ONE ? 0u : s_hd[pl]));
            }
            __syncthreads();
        }
    }
}

// Minima of the tiles' least D over 32 and 1024 tiles, as tile_min_levels_kernel.
__global__ void tree_levels_kernel(TreeArgs a, long long tiles) {
    after_prior_kernel();
    tiles = (position_count(tiles * PP_TILE, a.dL) + PP_TILE - 1) / PP_TILE;
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int32_t m = INT32_MAX;
    if (g < (tiles + 31) / 32) {
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const long long t = g * 32 + k;
            if (t < tiles) m = min(m, a.tile_min[t]);
        }
        a.m32[g] = m;
    }
    m = __reduce_min_sync(ALP_FULL_MASK, m);
    if ((threadIdx.x & 31) == 0 && g / 32 < (tiles + 1023) / 1024) a.m1024[g / 32] = m;
}

// The nearest earlier tile than t with tile_min <= d, as prev_tile_leq, for the searches of
// one tile: s_min holds the minima of t's 32-group, s_m32 those of the 32-groups of its
// 1024-block, so that only a search that goes further reads memory step by step (each step
// some 500 cycles: a walk over a group took up to 8 us).  In a group found further off, 32
// minima are read at once.
constexpr long long TR_LEVELS = 1024;  // up to these tiles tree_escape_kernel needs no levels
__device__ __forceinline__ long long tr_last_leq(const int32_t* v, int32_t d) {
    int at = -1;
#pragma unroll
    for (int k = 0; k < 32; ++k)
        if (v[k] <= d) at = k;
    return at;
}
__device__ __forceinline__ long long tr_prev_tile(const TreeArgs& a, const int32_t* s_min, const int32_t* s_m32, long long t,
                                                  int32_t d) {
    const int tl = (int)(t & 31), gl = (int)((t >> 5) & 31);
    for (int u = tl - 1; u >= 0; --u)
        if (s_min[u] <= d) return t - tl + u;
    long long g = -1;
    for (int u = gl - 1; u >= 0 && g < 0; --u)
        if (s_m32[u] <= d) g = (t >> 5) - gl + u;
    if (g < 0) {
        long long h = (t >> 10) - 1;
        while (h >= 0 && a.m1024[h] > d) --h;
        if (h < 0) return -1;
        g = h * 32 + tr_last_leq(a.m32 + h * 32, d);
    }
    return g * 32 + tr_last_leq(a.tile_min + g * 32, d);
}

// The searches that left their tile: the nearest earlier tile with a small enough minimum,
// then the last small enough entry of its staircase.  A search is some ten dependent loads.
// A warp takes a tile's first `head` searches, the eight warps of a block the rest, so that
// deep nesting, where a run of tiles lists thousands each, is spread over the warps, and over
// warps that read the same staircases.  Most tiles have no rest: a lane looks at one of the
// warp's next 32 parts, so that the idle ones cost one load together.  Up to 1024 tiles
// `head` is 32, for latency; past them 64, which holds json's 40 a tile.  Against one warp a
// tile: 1 Mi closers at the end of a document 0.73 -> 0.14 ms, 4 Mi levels of nesting 0.86 ->
// 0.41, 1000 documents nested 5000 deep 0.60 -> 0.32; 256 MiB of json 40 us as before.
// With the minima staged in shared memory, 22 -> 17 us at 4 MB of json.
__global__ void __launch_bounds__(256) tree_escape_kernel(TreeArgs a, long long cap_tiles, uint32_t head) {
    __shared__ int32_t s_min[8][32], s_m32[8][32];
    after_prior_kernel();
    const uint32_t tiles = (uint32_t)((position_count(cap_tiles * PP_TILE, a.dL) + PP_TILE - 1) / PP_TILE);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // items: the tiles' first parts, then eight to a tile of the rest, one to each warp of a block
    const uint32_t rest = (tiles + 7u) & ~7u, items = rest + 8u * tiles, warps = gridDim.x * 8u;
    auto part = [&](uint32_t w, uint32_t& first) -> uint32_t {  // its tile and first search
        first = w < rest ? 0u : head + 32u * ((w - rest) & 7u);
        return w < rest ? w : (w - rest) >> 3;
    };
    uint32_t next = blockIdx.x * 8u + (uint32_t)warp, w0 = 0, busy = 0;
    while (true) {
        while (!busy && next < items) {
            w0 = next;
            next += 32u * warps;
            const uint32_t w = w0 + (uint32_t)lane * warps;
            uint32_t first;
            const uint32_t u = part(w, first);
            busy = __ballot_sync(ALP_FULL_MASK, w < items && u < tiles && a.tiles[u].esc > first);
        }
        if (!busy) break;
        const uint32_t wt = w0 + (uint32_t)(__ffs(busy) - 1) * warps;
        busy &= busy - 1u;
        uint32_t first;
        const long long t = part(wt, first);
        const TreeTile tt = a.tiles[t];
        const uint32_t end = first ? tt.esc : min(tt.esc, head), stride = first ? 256u : 32u;
        {
            const long long u = (t & ~31ll) + lane, g = ((t >> 5) & ~31ll) + lane;
            __syncwarp();
            s_min[warp][lane] = u < t ? a.tile_min[u] : INT32_MAX;
            int32_t m = INT32_MAX;
            if (g < (t >> 5)) {
                if (tiles > TR_LEVELS) {
                    m = a.m32[g];
                } else {  // no level was built: a lane reads its group of the one block
                    const int4* v = reinterpret_cast<const int4*>(a.tile_min + g * 32);
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int4 x = v[k];
                        m = min(m, min(min(x.x, x.y), min(x.z, x.w)));
                    }
                }
            }
            s_m32[warp][lane] = m;
            __syncwarp();
        }
        for (uint32_t e = first + lane; e < end; e += stride) {
            const uint2 q = a.esc[(size_t)tt.node_base + t + e];
            const int32_t d = (int32_t)q.x;
            const long long pos = t * PP_TILE + (q.y & 2047u);
            const long long g = (long long)tt.node_base + (q.y >> 16);
            const uint32_t me = a.t.stack[(a.t.pairs[a.pid[pos]].y >> 16) + ((q.y >> 11) & 15u)];
            long long ans = -1;
            bool bad = true;
            const long long u = tr_prev_tile(a, s_min[warp], s_m32[warp], t, d);
            if (u >= 0) {
                const TreeTile tu = a.tiles[u];
                const uint2* sv = a.stair + (size_t)u * PP_TILE;
                int lo = 0, hi = (int)tu.stair - 1;  // the last entry <= d (they ascend)
                while (hi - lo >= 4) {  // three probes at a time: a round is one trip to memory
                    const int s4 = (hi - lo) >> 2, p1 = lo + s4, p2 = p1 + s4, p3 = p2 + s4;
                    const bool b1 = (int32_t)sv[p1].x <= d, b2 = (int32_t)sv[p2].x <= d, b3 = (int32_t)sv[p3].x <= d;
                    if (!b1) hi = p1 - 1;
                    else if (!b2) { lo = p1; hi = p2 - 1; }
                    else if (!b3) { lo = p2; hi = p3 - 1; }
                    else lo = p3;
                }
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if ((int32_t)sv[mid].x <= d) lo = mid; else hi = mid - 1;
                }
                if (hi >= 0) {
                    const uint2 s = sv[lo];
                    const uint2 pr = a.t.pairs[a.pid[u * PP_TILE + (s.y & 2047u)]];
                    const uint32_t l = (uint32_t)(d - (int32_t)s.x);
                    if (l < tr_nl(pr.x)) {
                        const uint32_t left = a.t.stack[(pr.y >> 16) + tr_nr(pr.x) + l];
                        bad = ((left ^ me) & 0xffffu) != 0;
                        ans = left >> 16 == TR_ROOT ? -2 : (long long)tu.node_base + (s.y >> 16) + (left >> 16);
                    }
                }
            }
            if (a.parent && q.y >> 16 != TR_NO_NODE && g < a.cap_nodes) {
                long long dbase = 0;
                if (a.n_docs > 1) dbase = a.node_off[seg_upper(a.node_off, 0, a.n_docs - 1, g)];
                a.parent[g] = ans == -2 ? 0 : (ans < 0 ? -1 : ans - dbase);
            }
            if (bad) {
                if (a.n_docs == 1) a.doc_valid[0] = 0;
                else tr_reject(a.tok_off, a.n_docs, a.doc_valid, pos);
            }
        }
    }
}

}  // namespace alp
