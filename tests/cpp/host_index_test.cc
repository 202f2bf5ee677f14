// The host's look at an index read from a file (host_index.h): which lists the
// library's builders could have made, and how often a list repeats an id.
#include <cstdio>

#include "../../genie_gb300/csrc/host_index.h"

using namespace gg;

static int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)

int main() {
    // 5 objects x 2 dims; dim 0 has values 3..5, dim 1 values 0..1
    const int32_t values[] = {3, 0, 4, 1, 3, 1, 5, 0, 4, 0};
    HostIndex ix;
    CHECK(build_host_index(values, 5, 2, ix));
    CHECK(ix.whole && lists_every_object_once(ix) && most_repeats(ix) == 1);

    HostIndex missing = ix;            // object 4 in no list of dim 1
    missing.ids.erase(missing.ids.begin() + 7);
    for (int64_t k = 4; k <= 5; ++k) missing.key_off[(size_t)k] -= 1;
    CHECK(!lists_every_object_once(missing) && most_repeats(missing) == 1);

    HostIndex twice = ix;              // object 0 in two lists of dim 0, object 1 in none
    twice.ids[2] = 0;
    CHECK(!lists_every_object_once(twice) && most_repeats(twice) == 1);

    HostIndex repeated = ix;           // object 0 twice in one list, object 2 in none
    repeated.ids[1] = 0;
    CHECK(!lists_every_object_once(repeated) && most_repeats(repeated) == 2);

    HostIndex outside = ix;            // the last list of dim 0 is past its largest value
    outside.dim_max[0] = 4;
    CHECK(!lists_every_object_once(outside));
    std::printf(bad ? "FAILED\n" : "OK\n");
    return bad;
}
