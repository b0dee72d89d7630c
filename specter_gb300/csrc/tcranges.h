// How launches over the lanes of several transforms are cut to the room that their digits have.
#pragma once

#include <algorithm>
#include <cstddef>

namespace sg {

struct TcRange {
    int jobs;        // transforms of one launch, at most
    unsigned tiles;  // tiles of 128 lanes of each, at most
};

// njobs transforms of `tiles` tiles each into room for cap >= 1 tiles: launches of as many whole transforms as
// fit, else of one transform's tiles in ranges.  Launches are of equal size, so that none is a small rest.
inline TcRange tc_range(int njobs, unsigned tiles, size_t cap) {
    auto even = [](size_t n, size_t most) {  // n in the fewest parts of at most `most`: the largest part
        const size_t parts = (n + most - 1) / most;
        return (n + parts - 1) / parts;
    };
    if (tiles > cap) return {1, (unsigned)even(tiles, cap)};
    return {(int)even((size_t)njobs, cap / tiles), tiles};
}

}  // namespace sg
