/*
 * octree_write.h -- the octree file from a builder's levels (host).
 */
#pragma once
#include <fcntl.h>
#include <stdint.h>
#include <stdio.h>
#include <sys/stat.h>
#include <unistd.h>

#include <atomic>

#include "vt_search.h"

namespace vtoct {

enum { WRITE_OK = 0, WRITE_FETCH, WRITE_OPEN, WRITE_SHORT };

/* What a level's range array is written from, in windows. */
struct Levels {
    float iso;
    int dimension, realDim[3], nLevels;
    unsigned long long runs[16];   /* of level l >= 1 */
    uint32_t bits1;                /* level 1's eight cells */
};

/* Header, then levels nLevels .. 0 as a word count and that many range words
 * (writeToFile, src/CreateOctree.cu:342-371).  fetch(l, k0, out): range words
 * of level l from k0 on, running over into the following levels, as many as
 * fit its window (*n of them); NULL if that fails. */
template <class Fetch>
int write_levels(FILE* f, const Levels& L, Fetch fetch) {
    const int magic = 919278872;
    bool ok = fwrite(&magic, 4, 1, f) == 1 && fwrite(&L.iso, 4, 1, f) == 1 && fwrite(&L.dimension, 4, 1, f) == 1 &&
              fwrite(L.realDim, 4, 3, f) == 3 && fwrite(&L.nLevels, 4, 1, f) == 1;
    const uint64_t* e = nullptr;
    size_t have = 0;               /* fetched and not yet written */
    for (int l = L.nLevels; ok && l >= 1; l--) {
        const int words = (int)(2 * L.runs[l]);
        ok = fwrite(&words, 4, 1, f) == 1;
        for (size_t k = 0; ok && k < (size_t)words;) {
            if (!have && !(e = fetch(l, k, &have))) return WRITE_FETCH;
            const size_t m = have < (size_t)words - k ? have : (size_t)words - k;
            ok = fwrite(e, 8, m, f) == m;
            e += m; have -= m; k += m;
        }
    }
    /* root (src/CreateOctree.cu:532-540), from level 1's eight bits */
    uint64_t e1[8], root[2] = {1ull, 1ull};
    int n1 = 0;
    for (int k = 0; k < 8; k++) {
        if (!((L.bits1 >> k) & 1u)) continue;
        if (k == 0 || !((L.bits1 >> (k - 1)) & 1u)) e1[n1++] = 8ull + k;
        if (k == 7 || !((L.bits1 >> (k + 1)) & 1u)) e1[n1++] = 8ull + k;
    }
    const int n0 = vtsearch::search_children_host(e1, n1, 1ull) > 0 ? 2 : 0;
    ok = ok && fwrite(&n0, 4, 1, f) == 1 && (n0 == 0 || fwrite(root, 8, 2, f) == 2);
    return ok ? WRITE_OK : WRITE_SHORT;
}

/* A new file beside `path` to take its place, with the mode of the one there;
 * NULL where that would not be the same as writing into it (a link, a device,
 * another's file, one that may not be written) or cannot be. */
inline FILE* open_beside(const char* path, char* name, size_t size, bool* there_) {
    static std::atomic<unsigned int> count(0);
    struct stat st;
    const bool there = *there_ = lstat(path, &st) == 0;
    if (there && (!S_ISREG(st.st_mode) || st.st_nlink != 1 || st.st_uid != geteuid() ||
                  faccessat(AT_FDCWD, path, W_OK, AT_EACCESS) != 0))
        return nullptr;
    const int n = snprintf(name, size, "%s.%ld-%u.tmp", path, (long)getpid(), count++);
    if (n < 0 || (size_t)n >= size) return nullptr;
    const int fd = open(name, O_WRONLY | O_CREAT | O_EXCL | O_CLOEXEC, 0666);
    if (fd < 0) return nullptr;
    FILE* f = !there || fchmod(fd, st.st_mode & 07777) == 0 ? fdopen(fd, "wb") : nullptr;
    if (!f) { close(fd); unlink(name); }
    return f;
}

/* The file is written beside the path and put in its place when it is whole,
 * so that a build whose device work fails half way leaves what was there.
 * Where that does not work (see open_beside; no room for two) it is written
 * in place.  An earlier file is exchanged and removed, not renamed over: over
 * a file, ext4 starts writing the new one out before the call returns (13 MB
 * written: 6.5 ms renamed over or truncated and written into, 1.75 ms
 * exchanged).  Holding all ranges in memory before opening the path would do
 * too, but costs a pass through fresh pages (512^3 blobs, 13 MB: 8.3 -> 13 ms
 * a build). */
template <class Fetch>
int write_octree(const char* path, const Levels& L, Fetch fetch) {
    char name[4096];
    bool there;
    if (FILE* f = open_beside(path, name, sizeof(name), &there)) {
        int r = write_levels(f, L, fetch);
        if (fclose(f) != 0 && r == WRITE_OK) r = WRITE_SHORT;
        if (r == WRITE_OK && there && renameat2(AT_FDCWD, name, AT_FDCWD, path, RENAME_EXCHANGE) == 0) {
            unlink(name);
            return WRITE_OK;
        }
        if (r == WRITE_OK && rename(name, path) == 0) return WRITE_OK;
        unlink(name);
        if (r == WRITE_FETCH) return r;
    }
    FILE* f = fopen(path, "wb");
    if (!f) return WRITE_OPEN;
    int r = write_levels(f, L, fetch);
    if (fclose(f) != 0 && r == WRITE_OK) r = WRITE_SHORT;
    return r;
}

}  // namespace vtoct
