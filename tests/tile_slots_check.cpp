// Runs the slot assignment of the shared-memory Gram (tile_slots.h) over every
// shape, with guard bytes behind its arrays and the distinct columns counted
// independently.  Prints one line per violated property.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <set>
#include <utility>
#include <vector>

#include "tile_slots.h"

using namespace de;

template <class S>
struct Guarded {
    TileSlots<S> t;
    unsigned char guard[64];
};

template <class S>
int check(int nl, int nr, int kind, std::vector<S> &mem, int &accepted)
{
    int bad = 0;
    std::vector<const S *> la(nl), lb(nl, nullptr), ra(nr), rb(nr, nullptr);
    int next = 0;
    for (int i = 0; i < nl; ++i) la[i] = &mem[next++];
    for (int j = 0; j < nr; ++j) ra[j] = &mem[next++];
    if (kind == 1 || kind == 3)  // L shifted, every partner of its own
        for (int i = 0; i < nl; ++i) lb[i] = &mem[next++];
    if (kind == 2 || kind == 3)  // R shifted likewise
        for (int j = 0; j < nr; ++j) rb[j] = &mem[next++];
    if (kind == 4)  // the projections: R = [L's shifted columns, their partners, ..]
        for (int i = 0; i < nl; ++i) lb[i] = &mem[next++];
    if (kind == 4)
        for (int j = 0; j < nr; ++j) {
            ra[j] = j < nl ? la[j] : lb[(j - nl) % nl];
            rb[j] = j < nl ? lb[j] : nullptr;
        }
    const int tl = (nl + 3) / 4, tr = (nr + 3) / 4;
    const bool shape = (tl <= 8 || tr <= 8) && tl * tr <= 36;
    bool fit = shape;
    if (shape) {
        int bl, br;
        tile_block(nl, nr, bl, br);
        for (int i = 0; i < nl; i += bl)
            for (int j = 0; j < nr; j += br) {
                const int ni = std::min(bl, nl - i), nj = std::min(br, nr - j);
                if (((ni + 3) / 4) * ((nj + 3) / 4) > 8) bad |= 1;
                std::set<std::pair<const S *, const S *>> cols;
                for (int u = 0; u < ni; ++u) cols.insert({la[i + u], lb[i + u]});
                for (int u = 0; u < nj; ++u) cols.insert({ra[j + u], rb[j + u]});
                std::set<std::pair<const S *, const S *>> all = cols;
                for (auto &c : cols)
                    if (c.second) all.insert({c.second, nullptr});
                const int tiles = ((ni + 3) / 4) * ((nj + 3) / 4);
                const bool want = all.size() <= 40 && 2 * all.size() * tile_rows(tiles) * sizeof(S) <= kTileSmem;
                Guarded<S> g;
                std::memset(g.guard, 0x5a, sizeof g.guard);
                const bool got = tile_slots(g.t, la.data() + i, lb.data() + i, ni, ra.data() + j, rb.data() + j, nj);
                for (unsigned char b : g.guard)
                    if (b != 0x5a) bad |= 2;
                if (got != want) bad |= 4;
                if (got) {
                    if (g.t.n != (int)all.size()) bad |= 8;
                    for (int u = 0; u < ni; ++u)
                        if (g.t.col[g.t.l[u]] != la[i + u] || g.t.sub[g.t.l[u]] != lb[i + u]) bad |= 16;
                    for (int u = 0; u < nj; ++u)
                        if (g.t.col[g.t.r[u]] != ra[j + u] || g.t.sub[g.t.r[u]] != rb[j + u]) bad |= 16;
                    for (int k = 0; k < g.t.nshift; ++k)
                        if (g.t.col[g.t.partner[k]] != g.t.sub[g.t.shifted[k]] || g.t.sub[g.t.partner[k]]) bad |= 32;
                }
                fit = fit && want;
            }
    }
    if (tiles_fit(la.data(), lb.data(), nl, ra.data(), rb.data(), nr) != fit) bad |= 64;
    // no column is shifted, or the projection's shape: always accepted
    if (shape && kind == 0 && !fit) bad |= 128;
    if (shape && kind == 4 && nr == 2 * nl && !fit) bad |= 256;
    accepted += fit;
    if (bad) std::printf("%zu bytes, %d x %d, kind %d: %d\n", sizeof(S), nl, nr, kind, bad);
    return bad;
}

struct C64 {
    float x, y;
};
struct C128 {
    double x, y;
};

int main()
{
    std::vector<C64> a(512);
    std::vector<C128> b(512);
    int bad = 0, accepted = 0;
    for (int nl = 1; nl <= 64; ++nl)
        for (int nr = 1; nr <= 128; ++nr)
            for (int kind = 0; kind < 5; ++kind) {
                bad |= check<C64>(nl, nr, kind, a, accepted);
                bad |= check<C128>(nl, nr, kind, b, accepted);
            }
    std::printf("accepted %d\n", accepted);
    return bad ? 1 : 0;
}
