// tile_slots.h -- the shared-memory slots of one gram_tile launch: the distinct
// columns of its operands, and whether they fit.  Host code without CUDA types,
// so that a host test can run it on every shape.
//
// A column of L or R is a[i], or a[i] - sigma b[i] where b[i] is not null; its
// partner b[i] then needs a slot of its own.  Without shifts at most 4 (tl + tr)
// <= 36 columns are distinct.  With them it may be twice as many; the
// projections, whose R repeats the columns of L and their partners, stay at 32.
#pragma once
#include <cstddef>

namespace de {

constexpr int kTile = 4;        // outputs of a warp: kTile x kTile
constexpr int kTileWarps = 8;   // output tiles x row groups of a CTA
constexpr int kMaxSlots = 40;   // distinct columns of a launch
constexpr int kMaxTiles = 36;   // output tiles over all launches
constexpr size_t kTileSmem = 112 * 1024;  // two CTAs per SM

template <class S>
struct TileSlots {
    const S *col[kMaxSlots], *sub[kMaxSlots];              // slot: col, or col - sigma sub
    unsigned char shifted[kMaxSlots], partner[kMaxSlots];  // slots that become col - sigma sub, and sub's
    unsigned char l[kTile * kTileWarps], r[kTile * kTileWarps];
    int n, nshift;
};

// The blocks of L and R columns a launch takes, at most kTileWarps tiles: the
// side with fewer tiles stays whole.
inline void tile_block(int nl, int nr, int &bl, int &br)
{
    const int tl = (nl + kTile - 1) / kTile, tr = (nr + kTile - 1) / kTile;
    bl = kTile * (tr <= tl ? (tr <= kTileWarps ? kTileWarps / tr : 1) : tl);
    br = kTile * (tr <= tl ? tr : (tl <= kTileWarps ? kTileWarps / tl : 1));
}

// rows a stage, and row groups of a CTA, for a number of tiles
inline int tile_groups(int tiles) { return kTileWarps / tiles; }
inline int tile_rows(int tiles)
{
    const int groups = tile_groups(tiles);
    return groups >= 8 ? 256 : groups >= 4 ? 128 : 64;
}

// False where the columns need more slots or two stages more shared memory than
// there is; t is then incomplete.
template <class S>
bool tile_slots(TileSlots<S> &t, const S *const *la, const S *const *lb, int nl, const S *const *ra, const S *const *rb,
                int nr)
{
    const int tl = (nl + kTile - 1) / kTile, tr = (nr + kTile - 1) / kTile;
    if (nl < 1 || nr < 1 || tl * tr > kTileWarps) return false;
    t.n = t.nshift = 0;
    auto find = [&](const S *a, const S *b) {
        for (int s = 0; s < t.n; ++s)
            if (t.col[s] == a && t.sub[s] == b) return s;
        if (t.n == kMaxSlots) return -1;
        t.col[t.n] = a;
        t.sub[t.n] = b;
        return t.n++;
    };
    for (int i = 0; i < nl + nr; ++i) {
        const int s = i < nl ? find(la[i], lb[i]) : find(ra[i - nl], rb[i - nl]);
        if (s < 0) return false;
        (i < nl ? t.l[i] : t.r[i - nl]) = (unsigned char)s;
    }
    for (int s = 0, n = t.n; s < n; ++s)
        if (t.sub[s]) {
            const int p = find(t.sub[s], nullptr);
            if (p < 0) return false;
            t.shifted[t.nshift] = (unsigned char)s;
            t.partner[t.nshift++] = (unsigned char)p;
        }
    for (int i = nl; i < tl * kTile; ++i) t.l[i] = t.l[0];  // padding, its outputs are dropped
    for (int j = nr; j < tr * kTile; ++j) t.r[j] = t.r[0];
    return 2 * (size_t)t.n * tile_rows(tl * tr) * sizeof(S) <= kTileSmem;
}

// Whether every launch of L (nl columns) against R (nr columns) fits.
template <class S>
bool tiles_fit(const S *const *la, const S *const *lb, int nl, const S *const *ra, const S *const *rb, int nr)
{
    const int tl = (nl + kTile - 1) / kTile, tr = (nr + kTile - 1) / kTile;
    if (nl < 1 || nr < 1 || (tl > kTileWarps && tr > kTileWarps) || tl * tr > kMaxTiles) return false;
    bool shifts = false;
    for (int i = 0; i < nl; ++i) shifts = shifts || lb[i];
    for (int j = 0; j < nr; ++j) shifts = shifts || rb[j];
    if (!shifts) return true;
    int bl, br;
    tile_block(nl, nr, bl, br);
    TileSlots<S> t;
    for (int i = 0; i < nl; i += bl)
        for (int j = 0; j < nr; j += br)
            if (!tile_slots(t, la + i, lb + i, nl - i < bl ? nl - i : bl, ra + j, rb + j, nr - j < br ? nr - j : br))
                return false;
    return true;
}

}  // namespace de
