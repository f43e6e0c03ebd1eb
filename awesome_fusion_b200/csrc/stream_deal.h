// How the tiles of the streaming form are dealt to its CTAs.  Plain arithmetic that host and device share; tests/test_stream_deal.py
// compiles it for the host and walks it.
//
// A tile is `blocks` units (raw weight blocks along K).  The first `shared_tiles` tiles are dealt in units: `dealers` CTAs take
// consecutive runs of them, the same number but for one.  The other tiles are dealt whole, one per CTA and wave.
// No dealer's run is empty (dealers <= units): all CTAs from the first to the last one with a unit of a tile hold some of it, which is
// what the count of a tile's arrivals and the adding up of its partial sums rely on.
// 32-bit arithmetic (units * (dealers + 1) < 2^32, which fits() says): the division in begin() comes before a CTA's first load.
#pragma once
#include <stdint.h>
#ifdef __CUDACC__
#define AFB_DEAL __host__ __device__ __forceinline__
#else
#define AFB_DEAL inline
#endif

namespace afb {

struct StreamDeal {
    uint32_t blocks;         // units of a tile
    uint32_t shared_tiles;   // tiles [0, shared_tiles) are dealt in units
    uint32_t whole_waves;    // the tiles after them, `grid` per wave
    uint32_t grid;           // CTAs
    uint32_t dealers;        // CTAs [0, dealers) hold units of shared tiles
    uint32_t tiles;          // all of them

    bool fits() const { return ((uint64_t)shared_tiles * blocks * (dealers + 1)) >> 32 == 0; }
    AFB_DEAL uint32_t units() const { return shared_tiles * blocks; }
    // first unit of CTA c (= end of CTA c - 1)
    AFB_DEAL uint32_t begin(uint32_t c) const { return c >= dealers ? units() : c * units() / dealers; }
    // the CTA holding unit u: the largest c with begin(c) <= u
    AFB_DEAL uint32_t cta_of(uint32_t u) const { return ((u + 1) * dealers + units() - 1) / units() - 1u; }
    AFB_DEAL uint32_t first_cta(uint32_t t) const { return cta_of(t * blocks); }
    AFB_DEAL uint32_t last_cta(uint32_t t) const { return cta_of(t * blocks + blocks - 1); }
    // Where CTA c leaves its partial sums of shared tile t: slot 2c for the tile its run begins in, 2c + 1 for the one it ends in
    // (tiles between them are whole and leave none).
    AFB_DEAL uint32_t slot(uint32_t c, uint32_t t) const { return 2 * c + (begin(c) / blocks != t ? 1u : 0u); }
};

// The pieces of work of one CTA, in order: units [kb0, kb1) of tile t.
struct Piece { uint32_t t, kb0, kb1; };
struct Walk {
    uint32_t u, u_end, it;
    AFB_DEAL void start(const StreamDeal& d, uint32_t cta) { u = d.begin(cta); u_end = d.begin(cta + 1); it = 0; }
    AFB_DEAL bool more(const StreamDeal& d, uint32_t cta) const { return u < u_end || (it < d.whole_waves && d.shared_tiles + cta + it * d.grid < d.tiles); }
    // SHORT: the last wave may be short (deal_whole)
    template <bool SHORT = false>
    AFB_DEAL bool next(const StreamDeal& d, uint32_t cta, Piece& x) {
        if (u < u_end) {
            x.t = u / d.blocks; x.kb0 = u - x.t * d.blocks;
            x.kb1 = u_end - u < d.blocks - x.kb0 ? x.kb0 + (u_end - u) : d.blocks;
            u += x.kb1 - x.kb0;
            return true;
        }
        if (it >= d.whole_waves) return false;
        x.t = d.shared_tiles + cta + it * d.grid; x.kb0 = 0; x.kb1 = d.blocks;
        if (SHORT && x.t >= d.tiles) return false;
        ++it;
        return true;
    }
};

// Tiles that fill whole waves stay whole; a short rest is shared together with the last full wave, so that no CTA gets less than
// a quarter of a tile of it.
// `least`: of a tile, in quarters.
inline StreamDeal deal_tiles(uint32_t tiles, uint32_t blocks, uint32_t sms, uint32_t least = 1) {
    StreamDeal d;
    d.blocks = blocks;
    d.grid = sms;
    d.tiles = tiles;
    const uint32_t waves = tiles / sms, rest = tiles - waves * sms;
    if (rest == 0) { d.shared_tiles = 0; d.whole_waves = waves; }
    else if (waves == 0) { d.shared_tiles = tiles; d.whole_waves = 0; }
    else if (rest * 4 >= least * sms) { d.shared_tiles = rest; d.whole_waves = waves; }
    else { d.shared_tiles = sms + rest; d.whole_waves = waves - 1; }
    const uint64_t units = (uint64_t)d.shared_tiles * blocks;
    d.dealers = units < sms ? (uint32_t)units : sms;
    if (d.whole_waves == 0) d.grid = d.dealers;
    return d;
}

// All tiles whole; the last wave may be short.
inline StreamDeal deal_whole(uint32_t tiles, uint32_t blocks, uint32_t sms) {
    StreamDeal d;
    d.blocks = blocks; d.tiles = tiles;
    d.shared_tiles = d.dealers = 0;
    d.grid = tiles < sms ? tiles : sms;
    d.whole_waves = (tiles + sms - 1) / sms;
    return d;
}

}  // namespace afb
#undef AFB_DEAL
