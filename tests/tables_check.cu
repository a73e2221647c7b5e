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

int main(int argc, char** argv) {
    const char* name = argc > 1 ? argv[1] : "";
    bool ok = false;
    if (!strcmp(name, "arity")) ok = arity(0) && !arity(1) && !arity(64) && !arity(INT32_MAX);
    if (ok) printf("ok\n");
    return ok ? 0 : 1;
}
