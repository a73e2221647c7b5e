// Table loading on the host with tables that no front end makes: what a context's creation
// reads on the host must stay in range and in bounded memory, and end in a refusal or the
// general kernels.  The argument names the case; prints "ok".
#include <cstdio>
#include <cstring>

#include "../alpacc_b200/csrc/keys.cuh"
#include "../alpacc_b200/csrc/tree.cuh"

using namespace alp;

// One ⊢ pair (end marker and start symbol) and one inner pair of one node with `arity` children.
static bool arity(int32_t children) {
    std::vector<PairInfo> info(2);
    info[0].stack_begin = 0; info[0].n_br = 2; info[0].prod_begin = 0; info[0].n_prod = 0;
    info[1].stack_begin = 2; info[1].n_br = 1; info[1].prod_begin = 0; info[1].n_prod = 1;
    const std::vector<uint8_t> use = {2, 1};
    const std::vector<uint32_t> stack = {0x80000007u, 0x80000001u, 1u}, pseq = {0};
    TreeHost h;
    return build_tree_tables(info, use, stack, pseq, {children}, {-1}, h);
}

// The parser section of a blob with two terminals and the sentinels given; no pairs, no keys.
static std::vector<uint8_t> section(uint32_t q, uint32_t k, uint32_t T, uint32_t empty, uint32_t start, uint32_t end,
                                    const std::vector<uint32_t>& pseq = {}) {
    std::vector<uint32_t> w = {q, k, T, empty, start, end, 1, 2, 0, 0xffffffffu, 0, 0, (uint32_t)pseq.size()};
    w.insert(w.end(), pseq.begin(), pseq.end());
    w.push_back(0);
    std::vector<uint8_t> b(4 * w.size());
    memcpy(b.data(), w.data(), b.size());
    return b;
}

// load_parser's refusal, or "" where it got as far as the uploads (which fail without a device)
static std::string refusal(const std::vector<uint8_t>& b) {
    ParseTables pt{};
    ParseHost ph;
    std::vector<void*> owned;
    std::string err;
    load_parser(pt, ph, b.data(), b.data() + b.size(), owned, err);
    return err.compare(0, 10, "cudaMalloc") == 0 ? "" : err;
}

static bool sentinels() {
    const std::string no = "parser sentinel ids out of range";
    return refusal(section(1, 1, 5, 2, 3, 4)).empty() && refusal(section(0, 1, 5, 5, 3, 4)).empty() &&
           refusal(section(1, 1, 5, 5, 3, 4)) == no && refusal(section(1, 3, 5, 0x7fffffffu, 3, 4)) == no &&
           refusal(section(1, 1, 5, 2, 5, 4)) == no && refusal(section(0, 1, 5, 2, 3, 0x40000000u)) == no;
}

// productions that no pair takes are read all the same
static bool productions() {
    const std::string no = "production id out of range";
    return refusal(section(1, 1, 5, 2, 3, 4, {0, 0})).empty() && refusal(section(1, 1, 5, 2, 3, 4, {0, 1})) == no &&
           refusal(section(1, 1, 5, 2, 3, 4, {0x7fffffffu, 0})) == no;
}

int main(int argc, char** argv) {
    const char* name = argc > 1 ? argv[1] : "";
    bool ok = false;
    if (!strcmp(name, "arity")) ok = arity(0) && !arity(1) && !arity(64) && !arity(INT32_MAX);
    if (!strcmp(name, "sentinels")) ok = sentinels();
    if (!strcmp(name, "productions")) ok = productions();
    if (ok) printf("ok\n");
    return ok ? 0 : 1;
}
