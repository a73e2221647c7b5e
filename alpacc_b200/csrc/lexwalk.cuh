// The lexer's two passes over known chunk states (sm_100a): counts and tokens.
//
// The state entering every 64 bytes is known (lex3_scan_kernel).  lex3_walk_kernel runs the
// DFA over them and keeps, beside each 32-byte chunk's token count and last token start, one
// 16-bit record per token that ends in the chunk: its end and its start as offsets in the
// chunk (or that it started before) and the state it ended in.  After the tile scan of the
// counts, lex3_write_kernel makes the tokens from the records alone: a warp lists the chunk
// and record of each of its 2 KiB's tokens, then takes them 32 at a time, a lane a token, and
// stores them straight to their places, coalesced.
// A second DFA walk (lex3_emit_kernel, kept for the speculative lexer, whose front end
// writes no records) costs 13 instructions and two to three wavefronts of shared-memory
// lookups a byte, and its per-thread token loops run as long as the densest lane's.
//
// The walk is bound by its shared-memory lookups (77 % of the data pipe) and its instruction
// stream; the write pass by the latency of its record loads and its instruction stream.  For
// 512 MiB of json (75 M tokens, 64-bit positions): walk 0.39 ms, write 0.50 ms, against 0.36 ms
// for a counting walk and 0.68 ms for a second walk; the state scan over 64-byte units takes
// 0.086 ms against 0.148 over chunks.  20,000 documents (245 MB): walk 0.24 and write 0.32 ms
// against 0.26 and 0.47: a warp with a document boundary takes the same unrolled walk with two
// tests a byte more, not a loop over the bytes of each boundary's thread.
//
// Traffic: 16 bytes of records a chunk (its first eight; more where more tokens end), written
// and read once, against the chunk's 32 bytes that a second walk reads again.
#pragma once
#include "common.cuh"
#include "lex3.cuh"

namespace alp {

// walk table: [S][LW_ROW] bytes: next state | LW_START (a kept token starts at this byte) |
// LW_EMIT (a kept token ends before it).  One byte an entry: the 128 entries of ASCII text are one
// word in every bank, so that lanes in the same state never conflict; the pitch is odd in
// words, which spreads the states.  (16-bit entries took 3.6 wavefronts a lookup, these 2.4.)
constexpr int LW_ROW = 260;
constexpr uint32_t LW_STATE = 31u, LW_START = 32u, LW_EMIT = 64u;
// a token record: state | end offset << 5 | start offset << 10 (LW_BEFORE: it started before
// the chunk).  A document's last byte has a record too, with that byte's offset as its end;
// the records of a chunk that was walked for document boundaries end with LW_STOP.
constexpr uint32_t LW_BEFORE = 63u;
constexpr uint32_t LW_STOP = 62u << 10;
constexpr int LW_FIRST = 8;       // records of a chunk in chunk_r; the others in chunk_x
constexpr int LW_WARP = 32 * 2 * LX_CHUNK;  // bytes of a warp of the write pass, and its most tokens
// A chunk has a record for each token that ends before one of its bytes and for the last byte
// of each document, and LW_STOP: at most 34, or 65 where the initial state itself ends (empty)
// tokens.
// In shared memory a row's pitch is an odd number of words.
constexpr int LW_SLOTS = 34, LW_SLOTS_EMPTY = 66;
__host__ __device__ inline int lw_more(int slots) { return (slots - LW_FIRST + 7) & ~7; }  // records of a chunk in chunk_x
__host__ __device__ inline size_t lw_table_bytes(int S) { return ((size_t)S * LW_ROW + 15) & ~(size_t)15; }
__host__ __device__ inline size_t lex3_walk_smem(int S, int slots) { return lw_table_bytes(S) + 2 * (size_t)LX_THREADS * slots + 16; }

// The walk of one 32-byte chunk.  e: the entry of the byte before (its next state is the
// state now).  ro: the thread's row of records in shared memory.
// EDGE: document heads, document ends and the input's end, at the bytes of `hd`, `ls` and
// from `lim` on: a head restarts in the initial state and starts a token; a document's last
// byte has a record with the state after it, for one more token unless that is ignored.
// k: tokens, rows: records (LW_STOP among them), off: last start offset.
template <bool EDGE>
__device__ __forceinline__ uint32_t lw_chunk(uint8_t* smem, uint32_t ro, const uint4 (&w)[2], uint32_t e, uint32_t& k,
                                             uint32_t& rows, uint32_t& off, uint32_t hd, uint32_t ls, int lim,
                                             const uint32_t* s_tok, uint32_t* endinfo) {
    uint32_t o = ro, ignored = 0, cur = LW_BEFORE << 10;
#pragma unroll
    for (int j = 0; j < LX_CHUNK; ++j) {
        if (EDGE && ((hd >> j) & 1u)) {
            e = 1u;
            cur = (uint32_t)j << 10;
        }
        const uint32_t st = e & LW_STATE;
        e = smem[st * LW_ROW + byte_of(w, j)];
        if (EDGE && j >= lim) e = st;
        if (e & LW_EMIT) {
            *reinterpret_cast<uint16_t*>(smem + o) = (uint16_t)(st + cur + ((uint32_t)j << 5));
            o += 2;
        }
        if (e & LW_START) cur = (uint32_t)j << 10;
        if (EDGE && ((ls >> j) & 1u)) {
            const uint32_t nx = e & LW_STATE, t = s_tok[nx];
            *endinfo = t;
            if (t & TOK_IGNORE) ++ignored;
            *reinterpret_cast<uint16_t*>(smem + o) = (uint16_t)(nx + cur + ((uint32_t)j << 5));
            o += 2;
        }
    }
    rows = (o - ro) >> 1;
    k = rows - ignored;
    if (EDGE) {
        *reinterpret_cast<uint16_t*>(smem + o) = (uint16_t)LW_STOP;
        ++rows;
    }
    off = (cur >> 10) < (uint32_t)LX_CHUNK ? cur >> 10 : LX_NOOFF;
    return e;
}

__global__ void __launch_bounds__(LX_THREADS, 6) lex3_walk_kernel(Lex3Args a, LexSeg sg) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int S = a.t.S;
    __shared__ uint32_t s_tok[32];
    __shared__ uint32_t s_head[LX_WIDE / LX_CHUNK], s_last[LX_WIDE / LX_CHUNK];
    __shared__ uint32_t s_wc[LX_THREADS / 32], s_wp[LX_THREADS / 32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const uint4* src = reinterpret_cast<const uint4*>(a.t.walk);
        uint4* dst = reinterpret_cast<uint4*>(smem);
        const int words = (int)(lw_table_bytes(S) / 16);
        for (int i = tid; i < words; i += LX_THREADS) dst[i] = __ldg(src + i);
    }
    if (tid < S) s_tok[tid] = a.t.tokinfo[tid];
    after_prior_kernel();
    const uint32_t ro = (uint32_t)lw_table_bytes(S) + tid * 2 * (uint32_t)a.t.slots;
    const long long n = a.n;
    for (unsigned ft = blockIdx.x; ft < a.num_wide; ft += gridDim.x) {
        const long long t0 = (long long)ft * LX_WIDE;
        const long long t1 = min(t0 + LX_WIDE, n) - 1;
        const long long my = t0 + (long long)tid * (2 * LX_CHUNK);
        const int lim = (int)max(0ll, min((long long)(2 * LX_CHUNK), n - my));
        uint4 w[2];
        uint32_t s0 = 1u;
        if (lim > 0) {
            lx_load<2>(a, my, min(lim, LX_CHUNK), w);
            s0 = a.unit_s[my / (2 * LX_CHUNK)];
        }
        const bool edges = sg.n_docs > 1 || t0 == 0 || t0 + LX_WIDE >= n;  // the same in every thread
        uint2 hd = make_uint2(0, 0), ls = make_uint2(0, 0);
        __syncthreads();  // the tables are loaded; the tile before is done with the shared words
        if (edges) {
            *reinterpret_cast<uint2*>(s_head + 2 * tid) = hd;
            *reinterpret_cast<uint2*>(s_last + 2 * tid) = ls;
            __syncthreads();
            lx_mark_docs(sg, n, sg.n_docs > 1 ? a.tile_doc[2 * (size_t)ft] : 0, t0, t1, s_head, s_last, nullptr);
            __syncthreads();
            hd = *reinterpret_cast<const uint2*>(s_head + 2 * tid);
            ls = *reinterpret_cast<const uint2*>(s_last + 2 * tid);
        }
        const bool edge = edges && __any_sync(ALP_FULL_MASK, lim < 2 * LX_CHUNK || (hd.x | hd.y | ls.x | ls.y) != 0);
        uint32_t cnt = 0, lastp = ALP_NONE32;
        if (lim > 0) {
            const long long c = my / LX_CHUNK;
            uint32_t e = s0, mid = 0, ei = 0;
            uint32_t cc[2], off[2], rw;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int l = min(max(lim - h * LX_CHUNK, 0), LX_CHUNK);
                if (h) {
                    mid = e & LW_STATE;
                    if (l > 0) lx_load<2>(a, my + LX_CHUNK, l, w);
                }
                if (edge) e = lw_chunk<true>(smem, ro, w, e, cc[h], rw, off[h], h ? hd.y : hd.x, h ? ls.y : ls.x, l, s_tok, &ei);
                else e = lw_chunk<false>(smem, ro, w, e, cc[h], rw, off[h], 0, 0, LX_CHUNK, s_tok, nullptr);
                if (rw) {
                    // the records to their place (an odd pitch: word by word)
                    const uint32_t* u = reinterpret_cast<const uint32_t*>(smem + ro);
                    reinterpret_cast<uint4*>(a.chunk_r)[c + h] = make_uint4(u[0], u[1], u[2], u[3]);
                    uint4* out = reinterpret_cast<uint4*>(a.chunk_x + (size_t)(c + h) * lw_more(a.t.slots));
                    for (uint32_t q = LW_FIRST; q < rw; q += 8)
                        out[q / 8 - 1] = make_uint4(u[q / 2], u[q / 2 + 1], u[q / 2 + 2], u[q / 2 + 3]);
                }
            }
            if (lim > LX_CHUNK) {
                *reinterpret_cast<uint16_t*>(a.chunk_s + c) = (uint16_t)(s0 | (mid << 8));
                *reinterpret_cast<uint32_t*>(a.chunk_c + c) = (cc[0] | (off[0] << 8)) | ((cc[1] | (off[1] << 8)) << 16);
            } else {
                a.chunk_s[c] = (uint8_t)s0;
                a.chunk_c[c] = (uint16_t)(cc[0] | (off[0] << 8));
            }
            // one document: accepted or not, known before its tokens are written
            if (sg.n_docs == 1 && (ls.x | ls.y)) a.res->aux[7] = (ei & TOK_ACCEPT) ? 1 : 0;
            cnt = cc[0] + cc[1];
            lastp = off[1] != LX_NOOFF ? (uint32_t)(my + LX_CHUNK + off[1])
                                       : (off[0] != LX_NOOFF ? (uint32_t)(my + off[0]) : ALP_NONE32);
        }
        // per 8 KiB tile (threads 0..127 and 128..255): count and last start (starts grow with
        // the position: the last is the greatest, NONE + 1 = 0 the least)
        const uint32_t wc = __reduce_add_sync(ALP_FULL_MASK, cnt), wp = __reduce_max_sync(ALP_FULL_MASK, lastp + 1u);
        if (lane == 0) { s_wc[warp] = wc; s_wp[warp] = wp; }
        __syncthreads();
        if (tid == 0 || tid == LX_THREADS / 2) {
            const int w0 = tid / 32;
            uint32_t c = 0, p = 0;
            for (int w2 = w0; w2 < w0 + LX_THREADS / 64; ++w2) {
                c += s_wc[w2];
                p = max(p, s_wp[w2]);
            }
            const size_t t8 = 2 * (size_t)ft + (tid ? 1 : 0);
            if (t8 < a.num_tiles) a.tile_cs[t8] = ((unsigned long long)c << 32) | (p - 1u);
        }
    }
}

__host__ __device__ inline size_t lex3_write_smem() { return (size_t)(LX_THREADS / 32) * (2 * LW_WARP + 64 * 4); }

// ONE: a single document, whose boundaries are the input's ends.  Its form has no searches for
// documents, which leaves the registers to the token loop: 512 MiB take 500 us in it, 585 in
// the form for several.
template <typename TermT, typename PosT, bool ONE>
__global__ void __launch_bounds__(LX_THREADS, 5) lex3_write_kernel(Lex3Args a, LexSeg sg) {
    const int S = a.t.S;
    __shared__ unsigned long long s_dmax;
    __shared__ uint32_t s_tok[32];
    __shared__ uint32_t s_head[LX_WIDE / LX_CHUNK], s_last[LX_WIDE / LX_CHUNK];
    __shared__ uint32_t s_wc[2][LX_THREADS / 32], s_wp[2][LX_THREADS / 32];
    __shared__ uint32_t s_doff[LX_DOCS];  // offsets of the tile's documents d0.. (up to LX_DOCS)
    extern __shared__ __align__(16) uint8_t smem[];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = LX_THREADS / 32;
    // of this warp: per token its chunk (of 64) << 6 | its record, per chunk the last start before it
    uint16_t* s_slot = reinterpret_cast<uint16_t*>(smem) + warp * LW_WARP;
    uint32_t* s_cur = reinterpret_cast<uint32_t*>(smem + 2 * NW * LW_WARP) + warp * 64;
    if (tid < S) s_tok[tid] = a.t.tokinfo[tid];
    after_prior_kernel();
    const long long n = a.n;
    const long long ND = ONE ? 1 : sg.n_docs;
    // document holding position p of this tile: the largest d in [d0, dmax]
    // with off[d] <= p, from the shared offsets when the tile has few documents
    auto doc_of = [&](long long d0, long long dmax, long long p) -> long long {
        if (ONE || dmax == d0) return d0;
        if (dmax - d0 < LX_DOCS) {
            int lo = 0, hi = (int)(dmax - d0);
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((long long)s_doff[mid] <= p) lo = mid; else hi = mid - 1;
            }
            return d0 + lo;
        }
        return doc_upper(sg.doc_off, d0, dmax, p);
    };
    auto base_of = [&](long long d0, long long dmax, long long d) -> long long {
        return (ONE || dmax - d0 < LX_DOCS) ? (long long)s_doff[d - d0] : sg.doc_off[d];
    };
    TermT* o_term = reinterpret_cast<TermT*>(a.out_term);
    PosT* o_start = reinterpret_cast<PosT*>(a.out_start);
    PosT* o_end = reinterpret_cast<PosT*>(a.out_end);
    const long long sent = sg.sentinels ? 1 : 0;
    // a stream piece places its tokens after the earlier pieces' and maps
    // positions to the stream; a start of NONE is the carried token start
    const long long tbase = (a.carry && a.carry_tokens) ? a.carry->tokens - a.tok_first : 0;
    const long long pb = a.pos_base;
    const long long snone = a.carry ? a.carry->start : 0;
    auto put = [&](long long idx, uint32_t term, long long st, long long en) {
        idx += tbase;
        if (idx < 0) return;  // before the stream's output window
        if (idx < a.cap) {
            o_term[idx] = (TermT)term;
            o_start[idx] = (PosT)st;
            o_end[idx] = (PosT)en;
        } else {
            atomicOr(&a.res->error, ALP_DEV_ERR_CAPACITY);
        }
    };
    const uint16_t* rec_r = reinterpret_cast<const uint16_t*>(a.chunk_r);
    const uint16_t* rec_x = a.chunk_x;
    const int more = lw_more(a.t.slots);
    // the i-th record of a chunk
    auto record = [&](size_t c, uint32_t i) -> uint32_t {
        return i < (uint32_t)LW_FIRST ? __ldg(rec_r + c * LW_FIRST + i) : __ldg(rec_x + c * more + (i - LW_FIRST));
    };
    int par = 0;
    for (unsigned ft = blockIdx.x; ft < a.num_wide; ft += gridDim.x, par ^= 1) {
        const long long t0 = (long long)ft * LX_WIDE;
        const long long t1 = min(t0 + LX_WIDE, n) - 1;
        const long long d0 = ND > 1 ? a.tile_doc[2 * (size_t)ft] : 0;
        const long long my = t0 + (long long)tid * (2 * LX_CHUNK);
        const int lim = (int)max(0ll, min((long long)(2 * LX_CHUNK), n - my));
        // the two chunks' counts and last starts
        const size_t c = (size_t)(my / LX_CHUNK);
        uint32_t cc = (LX_NOOFF << 8) | (LX_NOOFF << 24);
        if (lim > LX_CHUNK) cc = *reinterpret_cast<const uint32_t*>(a.chunk_c + c);
        else if (lim > 0) cc = (uint32_t)a.chunk_c[c] | (LX_NOOFF << 24);
        const unsigned long long X = a.tile_cs[2 * (size_t)ft];
        const bool edges = ND > 1 || t0 == 0 || t1 == n - 1;  // the same in every thread
        uint2 heads = make_uint2(0, 0), lasts = make_uint2(0, 0);
        if (edges) {
            __syncthreads();  // the tile before is done with the shared words
            if (tid == 0) s_dmax = (unsigned long long)d0;
            *reinterpret_cast<uint2*>(s_head + 2 * tid) = heads;
            *reinterpret_cast<uint2*>(s_last + 2 * tid) = lasts;
            __syncthreads();
            lx_mark_docs(sg, n, d0, t0, t1, s_head, s_last, &s_dmax, s_doff);
        }
        const uint32_t cnt0 = cc & 0xffu, cnt = cnt0 + ((cc >> 16) & 0xffu);
        const uint32_t off0 = (cc >> 8) & 0xffu, off1 = cc >> 24;
        const uint32_t last0 = off0 != LX_NOOFF ? (uint32_t)my + off0 : ALP_NONE32;
        const uint32_t lastp = off1 != LX_NOOFF ? (uint32_t)my + LX_CHUNK + off1 : last0;
        // ---- this thread's place: tile prefix + block scan of stored counts.  Starts grow
        // with the position, so the last one before a thread is a maximum (0: none)
        uint32_t ic = cnt, ip = lastp + 1u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t oc = __shfl_up_sync(ALP_FULL_MASK, ic, d), op = __shfl_up_sync(ALP_FULL_MASK, ip, d);
            if (lane >= d) { ic += oc; ip = max(ip, op); }
        }
        uint32_t ep = __shfl_up_sync(ALP_FULL_MASK, ip, 1);
        if (lane == 0) ep = 0;
        if (lane == 31) { s_wc[par][warp] = ic; s_wp[par][warp] = ip; }
        __syncthreads();
        long long dmax = d0;
        if (edges) {
            dmax = ONE ? 0 : (long long)s_dmax;
            heads = *reinterpret_cast<const uint2*>(s_head + 2 * tid);
            lasts = *reinterpret_cast<const uint2*>(s_last + 2 * tid);
        }
        const uint32_t vc = lane < NW ? s_wc[par][lane] : 0u, vp = lane < NW ? s_wp[par][lane] : 0u;
        const uint32_t wc = __reduce_add_sync(ALP_FULL_MASK, lane < warp ? vc : 0u);
        const uint32_t wp = __reduce_max_sync(ALP_FULL_MASK, lane < warp ? vp : 0u);
        const uint32_t Xc = (uint32_t)(X >> 32), Xp = (uint32_t)X;
        const uint32_t before = max(ep, wp);
        const uint32_t cur0 = before ? before - 1u : Xp;         // last start before this thread's bytes
        const uint32_t cur1 = last0 != ALP_NONE32 ? last0 : cur0;  // and before its second chunk
        const bool edge = (heads.x | heads.y | lasts.x | lasts.y) != 0;

        if (edge) {
            // documents that start or end in this thread's bytes: record by record and
            // boundary by boundary, in the order token before the byte, head, last token
            // (a head's own end flag, from an accepting initial state, comes after the head)
            // The chunk's record i and the one after it are held, the next load in flight while a
            // token is stored, and a head's documents follow from the one before: with a load for
            // each test of a record and a search for each head 300,000 documents of one byte took
            // 412 us here, 161 so (a second DFA walk 168); 40,000 of ten bytes 127 and 78 (63).
            uint32_t t = Xc + wc + ic - cnt, i = 0, h = 0, cur = cur0;
            uint32_t r0 = record(c, 0), r1 = record(c, 1);
            long long doc = doc_of(d0, dmax, my);
            long long base = base_of(d0, dmax, doc);
            const unsigned long long hd = heads.x | ((unsigned long long)heads.y << 32), ls = lasts.x | ((unsigned long long)lasts.y << 32);
            auto tok = [&](uint32_t r, uint32_t ch, uint32_t end) {
                const uint32_t at = (uint32_t)my + ch * LX_CHUNK, so = r >> 10;
                const uint32_t st = so < (uint32_t)LX_CHUNK ? at + so : cur;
                put((long long)t + sent * (2 * doc + 1), s_tok[r & 31u] & TOK_TERM_MASK,
                    st == ALP_NONE32 ? snone : (long long)st - base + pb, (long long)(at + end) - base + pb);
                ++t;
            };
            uint32_t left = cnt0;  // tokens of the current chunk to come
            auto step = [&]() { r0 = r1; r1 = record(c + h, ++i + 1u); };
            for (int j = 0; j < lim;) {
                // the next boundary at or after byte j, or the end of the chunk
                const unsigned long long ev = (hd | ls) >> j;
                const int cend = j < LX_CHUNK ? LX_CHUNK : 2 * LX_CHUNK;
                const int b = ev ? min(cend, j + __ffsll((long long)ev) - 1) : cend;
                const bool bnd = b < cend;
                const bool head = bnd && ((hd >> b) & 1ull), last = bnd && ((ls >> b) & 1ull);
                const uint32_t bo = (uint32_t)(b - (int)h * LX_CHUNK);  // its offset in the chunk
                auto next = [&]() { tok(r0, h, (r0 >> 5) & 31u); --left; step(); };
                // a token ends before byte b itself (its last byte's own record comes after it)
                auto at_b = [&]() {
                    if (!left || ((r0 >> 5) & 31u) != bo) return false;
                    return !last || ((r1 >> 10) != (LW_STOP >> 10) && ((r1 >> 5) & 31u) == bo);
                };
                while (left && ((r0 >> 5) & 31u) < bo) next();
                if (head) {
                    // every document starting here (empty ones first, then the real one): past the
                    // thread's first byte the ones right after the current document
                    const long long pos = my + b;
                    long long dl = doc;
                    if (b > 0) {
                        dl = doc + 1;
                        while (++doc < dmax && base_of(d0, dmax, doc + 1) <= pos) {}
                    } else {
                        while (dl > 0 && sg.doc_off[dl - 1] >= pos) --dl;
                    }
                    base = pos;
                    for (long long e2 = dl; e2 <= doc; ++e2) {
                        sg.tok_off[e2] = t;
                        if (sent) put((long long)t + 2 * e2, sg.sent_l, 0, 0);
                        if (e2 < doc) {
                            sg.valid[e2] = 0;
                            if (sent) put((long long)t + 2 * e2 + 1, sg.sent_r, 0, 0);
                        }
                    }
                }
                if (bnd && at_b()) next();
                if (last) {
                    const uint32_t ti = s_tok[r0 & 31u];
                    if (!(ti & TOK_IGNORE)) {
                        tok(r0, h, bo + 1u);
                        --left;
                    }
                    step();
                    sg.valid[doc] = (ti & TOK_ACCEPT) ? 1 : 0;
                    if (sent) put((long long)t + 2 * doc + 1, sg.sent_r, 0, 0);
                }
                j = bnd ? b + 1 : b;
                if (j >= LX_CHUNK && h == 0) {
                    h = 1;
                    i = 0;
                    left = cnt - cnt0;
                    cur = cur1;
                    if (lim > LX_CHUNK) {
                        r0 = record(c + 1, 0);
                        r1 = record(c + 1, 1);
                    }
                }
            }
        }
        if (my <= n - 1 && n - 1 < my + 2 * LX_CHUNK) {
            // documents that start at n (empty, at the end) and the closing offset
            const uint32_t t = Xc + wc + ic;
            for (long long e2 = doc_of(d0, dmax, n - 1) + 1; e2 < ND; ++e2) {
                sg.tok_off[e2] = t;
                sg.valid[e2] = 0;
                if (sent) {
                    put((long long)t + 2 * e2, sg.sent_l, 0, 0);
                    put((long long)t + 2 * e2 + 1, sg.sent_r, 0, 0);
                }
            }
            sg.tok_off[ND] = t;
            a.res->count = t;
            a.res->valid = 1;
        }

        // ---- the warp's other tokens, 32 at a time.  Their numbers r run over the threads
        // without boundaries; `shift`: what the tokens of those with boundaries add to r
        uint32_t in = ic, shift = 0;  // numbers up to and including this thread's
        const uint32_t c1 = edge ? 0u : cnt;
        const bool shift_none = !__any_sync(ALP_FULL_MASK, edge);
        if (!shift_none) {
            in = warp_scan_add(c1, lane);
            shift = (ic - cnt) - (in - c1);
        }
        const uint32_t total = __shfl_sync(ALP_FULL_MASK, in, 31);
        __syncwarp();  // the tile before is done with the slots
        *reinterpret_cast<uint2*>(s_cur + 2 * lane) = make_uint2(cur0, cur1);
        if (c1) {
            uint16_t* p = s_slot + (in - c1);
            uint32_t v = (uint32_t)lane << 7;
            for (uint32_t i = 0; i < cnt0; ++i) *p++ = (uint16_t)v++;
            v = ((uint32_t)lane << 7) + 64u;
            for (uint32_t i = cnt0; i < cnt; ++i) *p++ = (uint16_t)v++;
        }
        __syncwarp();
        const uint32_t wpos = (uint32_t)t0 + warp * (uint32_t)LW_WARP;
        const uint16_t* wr = rec_r + ((size_t)(t0 / LX_CHUNK) + warp * 64) * LW_FIRST;
        const uint16_t* wx = rec_x + ((size_t)(t0 / LX_CHUNK) + warp * 64) * more;
        auto load = [&](uint32_t sl) -> uint32_t {
            const uint32_t q = sl >> 6, i = sl & 63u;
            return i < (uint32_t)LW_FIRST ? __ldg(wr + (q * LW_FIRST + i)) : __ldg(wx + (q * (uint32_t)more + i - LW_FIRST));
        };
        // one document in the tile: its tokens' indices and positions shift alike
        if (dmax == d0 && shift_none) {
            const long long ib = (long long)Xc + wc + tbase + sent * (2 * d0 + 1);
            const long long off = ND > 1 ? pb - base_of(d0, dmax, d0) : pb;
            // (elements before the output window or past the capacity are not stored)
            const uint32_t lo = ib < 0 ? (uint32_t)min((long long)total, -ib) : 0u;
            const uint32_t hi = (uint32_t)max((long long)lo, min((long long)total, a.cap - ib));
            if (hi < total && lane == 0) atomicOr(&a.res->error, ALP_DEV_ERR_CAPACITY);
            TermT* pt = o_term + ib;
            PosT* ps = o_start + ib;
            PosT* pe = o_end + ib;
            const PosT poff = (PosT)off, none = (PosT)snone;
#pragma unroll 2
            for (uint32_t r = lo + lane; r < hi; r += 32) {
                const uint32_t sl = s_slot[r];
                const uint32_t rec = load(sl);
                const uint32_t at = wpos + (sl >> 6) * LX_CHUNK, so = rec >> 10;
                const uint32_t st = so < (uint32_t)LX_CHUNK ? at + so : s_cur[sl >> 6];
                pt[r] = (TermT)(s_tok[rec & 31u] & TOK_TERM_MASK);
                ps[r] = st == ALP_NONE32 ? none : (PosT)((PosT)st + poff);
                pe[r] = (PosT)((PosT)(at + ((rec >> 5) & 31u)) + poff);
            }
        } else {
            long long ib = 0, off = 0;
            if (!edge && cnt) {
                const long long d = doc_of(d0, dmax, my);
                ib = (long long)Xc + wc + shift + sent * (2 * d + 1);
                off = pb - base_of(d0, dmax, d);
            }
            for (uint32_t r0 = 0; r0 < total; r0 += 32) {
                const uint32_t r = r0 + lane;
                const uint32_t sl = r < total ? s_slot[r] : 0u;
                const long long tib = __shfl_sync(ALP_FULL_MASK, ib, sl >> 7), toff = __shfl_sync(ALP_FULL_MASK, off, sl >> 7);
                if (r < total) {
                    const uint32_t rec = load(sl);
                    const uint32_t at = wpos + (sl >> 6) * LX_CHUNK, so = rec >> 10;
                    const uint32_t st = so < (uint32_t)LX_CHUNK ? at + so : s_cur[sl >> 6];
                    put(tib + r, s_tok[rec & 31u] & TOK_TERM_MASK, st == ALP_NONE32 ? snone : (long long)st + toff,
                        (long long)(at + ((rec >> 5) & 31u)) + toff);
                }
            }
        }
    }
}

}  // namespace alp
