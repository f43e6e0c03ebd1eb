// Walks the dealing of csrc/stream_deal.h as the kernel's CTAs do (test infrastructure, built by tests/test_stream_deal.py).
#include <vector>
#include "stream_deal.h"

// 0, or which rule is broken: 1 a unit not dealt exactly once, 2 a contributor missing between the first and the last CTA of a tile (it
// would be waited for), 3 two partial sums in one place, 4 more than two shared tiles to finish in one CTA, 5 a CTA with nothing to do,
// 6 a run that is longer than another by more than one unit, 7 refused as too large, 8 more() says otherwise than next(), 9 waves and
// shared tiles do not add up to the tiles.  SHORT: as the pair form walks, past whose last tile a short wave ends; the streaming form's
// walk knows no short wave.
template <bool SHORT>
static int check(const afb::StreamDeal& d, uint32_t tiles, uint32_t blocks) {
    if (!d.fits()) return 7;
    if (!SHORT && d.shared_tiles + (uint64_t)d.whole_waves * d.grid != tiles) return 9;
    std::vector<uint8_t> seen((size_t)tiles * blocks, 0);
    std::vector<uint32_t> arrivals(d.shared_tiles, 0);
    std::vector<uint8_t> slots((size_t)2 * d.grid, 0);
    uint32_t shortest = ~0u, longest = 0;
    for (uint32_t c = 0; c < d.grid; ++c) {
        afb::Walk w;
        w.start(d, c);
        if (c < d.dealers && d.shared_tiles) {
            const uint32_t run = w.u_end - w.u;
            shortest = run < shortest ? run : shortest;
            longest = run > longest ? run : longest;
        }
        afb::Piece x;
        bool more = true;
        uint32_t pieces = 0, parts = 0;
        while (w.next<SHORT>(d, c, x)) {
            ++pieces;
            if (!more) return 8;
            more = w.more(d, c);
            if (x.t >= tiles || x.kb0 >= x.kb1 || x.kb1 > blocks) return 1;
            for (uint32_t kb = x.kb0; kb < x.kb1; ++kb)
                if (seen[(size_t)x.t * blocks + kb]++) return 1;
            if (x.kb0 == 0 && x.kb1 == blocks) continue;
            if (x.t >= d.shared_tiles || c < d.first_cta(x.t) || c > d.last_cta(x.t)) return 2;
            ++arrivals[x.t];
            if (++parts > 2) return 4;
            if (slots[d.slot(c, x.t)]++) return 3;
        }
        if (!pieces) return 5;
        if (more) return 8;
    }
    for (uint8_t s : seen) if (!s) return 1;
    for (uint32_t t = 0; t < d.shared_tiles; ++t)
        if (arrivals[t] && arrivals[t] != d.last_cta(t) - d.first_cta(t) + 1) return 2;
    if (d.shared_tiles && longest - shortest > 1) return 6;
    return 0;
}
extern "C" int check_deal(uint32_t tiles, uint32_t blocks, uint32_t sms) { return check<false>(afb::deal_tiles(tiles, blocks, sms), tiles, blocks); }
// what the walks of both forms make of a dealing with `waves` whole waves more than there are: the tiles dealt past the end
extern "C" uint32_t tiles_past_the_end(uint32_t tiles, uint32_t blocks, uint32_t sms, uint32_t waves, int as_pairs) {
    afb::StreamDeal d = afb::deal_tiles(tiles, blocks, sms);
    d.whole_waves += waves;
    uint32_t past = 0;
    for (uint32_t c = 0; c < d.grid; ++c) {
        afb::Walk w;
        w.start(d, c);
        afb::Piece x;
        while (as_pairs ? w.next<true>(d, c, x) : w.next(d, c, x)) past += x.t >= tiles;
    }
    return past;
}
extern "C" int check_waves(uint32_t tiles, uint32_t blocks, uint32_t sms, uint32_t more_waves) {
    afb::StreamDeal d = afb::deal_tiles(tiles, blocks, sms);
    d.whole_waves += more_waves;
    return check<false>(d, tiles, blocks);
}
// as the pair form deals: whatever does not fill whole waves shared, or nothing
extern "C" uint32_t check_pair_range(uint32_t tiles_end, uint32_t blocks_end, uint32_t pairs, uint32_t* where) {
    for (uint32_t t = 1; t < tiles_end; ++t)
        for (uint32_t b = 1; b < blocks_end; ++b)
            for (int share = 0; share < 2; ++share)
                if (const int rc = check<true>(share ? afb::deal_tiles(t, b, pairs, 0) : afb::deal_whole(t, b, pairs), t, b)) { where[0] = t; where[1] = b; return (uint32_t)rc; }
    return 0;
}
extern "C" uint32_t check_range(uint32_t tiles_end, uint32_t blocks_end, uint32_t sms, uint32_t* where) {
    for (uint32_t t = 1; t < tiles_end; ++t)
        for (uint32_t b = 1; b < blocks_end; ++b)
            if (const int rc = check_deal(t, b, sms)) { where[0] = t; where[1] = b; return (uint32_t)rc; }
    return 0;
}
extern "C" int fits(uint32_t tiles, uint32_t blocks, uint32_t sms) { return afb::deal_tiles(tiles, blocks, sms).fits(); }
