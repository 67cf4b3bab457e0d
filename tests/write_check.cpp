/* Host check of write_octree (octree_write.h) with ranges from a made-up
 * fetch of three words a window.  argv: the path, the word before which the
 * fetch fails (-1: none).  Prints the result and the words fetched. */
#include <cstdio>
#include <cstdlib>

#include "octree_write.h"

int main(int argc, char** argv) {
    if (argc < 3) return 1;
    vtoct::Levels L = {0.5f, 8, {7, 5, 8}, 3, {0, 1, 2, 3}, 3u};
    const long fail = atol(argv[2]);
    const uint64_t words[12] = {512, 513, 600, 601, 700, 700, 64, 65, 80, 80, 8, 9};   /* level 3 first */
    const size_t first[4] = {0, 10, 6, 0};
    long fetched = 0;
    const int r = vtoct::write_octree(argv[1], L, [&](int l, size_t k0, size_t* n) -> const uint64_t* {
        const size_t at = first[l] + k0;
        *n = at + 3 < 12 ? 3 : 12 - at;
        if (fail >= 0 && at + *n > (size_t)fail) return nullptr;
        fetched += (long)*n;
        return words + at;
    });
    printf("%d %ld\n", r, fetched);
    return 0;
}
