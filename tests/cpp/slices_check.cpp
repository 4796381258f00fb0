// Scratch of the dense chain against the launches that use it, for every count of points and slice around the borders.
#include <cstdio>
#include <set>

#include "../../superkmeans_b200/csrc/host_logic.h"

using namespace skmb;

int main() {
    size_t sharing = 0, wrong = 0;
    for (const size_t pairs : {size_t{1}, size_t{4}, size_t{66}, size_t{74}, size_t{80}}) {
        const size_t most = pairs / kChainUnits * kChainTileRows;   // the largest launch whose tiles are shared
        for (const size_t slice : {size_t{1}, size_t{256}, most, most + 1, pairs * 256, 13 * pairs * 256}) {
            if (slice == 0) continue;
            std::set<size_t> rests{0, 1, 255, 256, 257, most, most + 1, slice - 1};
            for (const size_t whole : {0, 1, 2, 13}) {
                for (const size_t rest : rests) {
                    if (rest >= slice || whole + rest == 0) continue;
                    const size_t n = whole * slice + rest, rows = chain_scratch_rows(n, slice, pairs);
                    // as the points go through
                    for (size_t r0 = 0; r0 < n; r0 += slice) {
                        const size_t cnt = std::min(slice, n - r0);
                        const bool shares = chain_shares_tiles(cnt, pairs);
                        if (shares) ++sharing;
                        if (shares != (cnt <= most) || (shares && cnt > rows)) {
                            std::printf("pairs %zu slice %zu n %zu: a launch of %zu, scratch for %zu\n", pairs, slice, n, cnt, rows);
                            ++wrong;
                        }
                    }
                    if (rows > slice) ++wrong;
                }
            }
        }
    }
    std::printf("%s (%zu launches share tiles)\n", wrong == 0 && sharing > 100 ? "OK" : "WRONG", sharing);
    return wrong != 0 || sharing <= 100;
}
