// position_count on the host: a launch sized for `cap` positions never takes more, whatever
// count is in memory, in positions and in whole tiles.  Prints "ok".
#include <cstdio>

#include "../alpacc_b200/csrc/parser.cuh"

using namespace alp;

int main() {
    const long long caps[] = {1, 3, PP_TILE - 1, PP_TILE, PP_TILE + 1, 9016, 3ll * PP_TILE * ST_CHUNK + 5, 0x7fffffffll};
    for (long long cap : caps) {
        const long long tiles = (cap + PP_TILE - 1) / PP_TILE;
        if (position_count(cap, nullptr) != cap) return 1;
        const long long counts[] = {0, 1, cap - 1, cap, cap + 1, cap + cap / 2, 4 * cap, 1ll << 40};
        for (long long n : counts) {
            const long long got = position_count(cap, &n);
            if (got > cap || (n <= cap && got != n)) return 1;
            // as the kernels over whole tiles cut it
            const long long t = (position_count(tiles * PP_TILE, &n) + PP_TILE - 1) / PP_TILE;
            if (t > tiles || (n <= cap && t != (n + PP_TILE - 1) / PP_TILE)) return 1;
        }
    }
    printf("ok\n");
    return 0;
}
