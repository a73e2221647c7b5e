// The searches that parse_tree_kernel lists a tile (tr_listed), on the host: for batches of
// documents given as pair ids, those that the tile cannot answer are counted against the room
// of its list, its nodes and one more.  Reads the tables and the batches as numbers from the
// file named (tests/test_tree_room.py writes it); prints "ok <most listed past the nodes>".
#include <cstdio>
#include <vector>

#include "../alpacc_b200/csrc/tree.cuh"

using namespace alp;

static FILE* in;
static long long number() {
    long long v = 0;
    if (fscanf(in, "%lld", &v) != 1) { printf("short file\n"); exit(2); }
    return v;
}

int main(int argc, char** argv) {
    in = argc > 1 ? fopen(argv[1], "r") : nullptr;
    if (!in) return 2;
    const size_t n_pairs = (size_t)number();
    std::vector<PairInfo> info(n_pairs);
    std::vector<uint8_t> use(n_pairs);
    for (size_t i = 0; i < n_pairs; ++i) {
        info[i].stack_begin = (uint32_t)number();
        info[i].n_br = (uint16_t)number();
        info[i].prod_begin = (uint32_t)number();
        info[i].n_prod = (uint16_t)number();
        use[i] = (uint8_t)number();
    }
    std::vector<uint32_t> stack((size_t)number());
    for (auto& v : stack) v = (uint32_t)number();
    std::vector<uint32_t> pseq((size_t)number());
    for (auto& v : pseq) v = (uint32_t)number();
    std::vector<int32_t> arity((size_t)number()), pterm(arity.size());
    for (auto& v : arity) v = (int32_t)number();
    for (auto& v : pterm) v = (int32_t)number();
    TreeHost h;
    if (!build_tree_tables(info, use, stack, pseq, arity, pterm, h)) { printf("no compact tables\n"); return 1; }
    long long most = -1, unlisted = 0;
    for (long long batches = number(); batches > 0; --batches) {
        const size_t L = (size_t)number();
        std::vector<uint32_t> id(L);
        std::vector<uint8_t> head(L);
        for (size_t i = 0; i < L; ++i) {
            id[i] = (uint32_t)number();
            head[i] = (uint8_t)number();
        }
        std::vector<int32_t> D(L);
        std::vector<uint8_t> below(L, 0);  // the position takes its document's depth below zero
        int32_t depth = 0;
        for (size_t t = 0; t < L; t += PP_TILE) {
            long long nodes = 0, listed = 0;
            for (size_t i = t; i < L && i < t + PP_TILE; ++i) {
                if (head[i]) depth = 0;
                const uint32_t p = id[i] == NO_PAIR ? (uint32_t)n_pairs : id[i];
                const uint32_t x = h.pairs[2 * p], sb = h.pairs[2 * p + 1] >> 16;
                const int32_t nl = (int32_t)((x >> 8) & 15u), nr = (int32_t)((x >> 12) & 15u);
                D[i] = nl ? depth - nr : TR_NONE;
                below[i] = depth < nr;
                for (int32_t r = 0; r < nr; ++r) {
                    const int32_t d = depth - 1 - r;
                    bool here = false;
                    for (size_t q = i; q > t && !here; --q) here = D[q - 1] <= d;
                    if (here) continue;
                    const uint32_t se = h.stack[sb + r] >> 16;
                    if (tr_listed(d, se == TR_END ? TR_NO_NODE : (uint32_t)nodes + se)) {
                        ++listed;
                    } else {
                        ++unlisted;
                        if (!below[i]) { printf("an unlisted search of a document that may be valid\n"); return 1; }
                    }
                }
                nodes += x & 31u;
                depth += nl - nr;
            }
            if (listed - nodes > most) most = listed - nodes;
            if (listed > nodes + 1) {
                printf("position %zu: %lld searches listed, room for %lld\n", t, listed, nodes + 1);
                return 1;
            }
        }
    }
    printf("ok %lld %lld\n", most, unlisted);
    return 0;
}
