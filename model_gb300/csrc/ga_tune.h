// Choice of a level tile by its time (host).
#pragma once

namespace ga {

// `keep`, whose time is `best`, unless another power of two from kmin to kmax
// that fits is faster by more than 0.4%, about what the least of a few samples
// of one tile varies by (a context already at its best tile must stay there).
// keep 0: no tile yet, `best` is what a tile has to beat.  Returns the tile and
// leaves its time in `best`.
template <typename Fits, typename Time>
inline int faster_tile(int keep, int kmin, int kmax, float &best, Fits fits, Time time)
{
    const int stay = keep;
    for (int kt = kmin; kt <= kmax; kt <<= 1) {
        if (!fits(kt)) break;
        if (kt == stay) continue;
        const float t = time(kt);
        if (t < 0.996f * best) {
            best = t;
            keep = kt;
        }
    }
    return keep;
}

}  // namespace ga
