// How a grid is cut into tiles for the z-marching kernels, and the blocks that take them. Host code that a
// plain C++ compiler takes too.
#pragma once

#include <stddef.h>

namespace pm {

// The tiling every step kernel walks: 32 × 8 columns of cells (one warp row per y), each
// marched through `zc` planes by its thread. A persistent grid of blocks takes tiles
// blockIdx.x, blockIdx.x + gridDim.x, ... in that fixed order, so every thread's share of a
// reduction is summed in the same order on every run.
struct Tiles {
    int nx, ny, nz, zc;
    int ntx, nty, ntz;
    long long ntiles;
    int rows;  // rows of a tile: the block's y extent (8 but in the many-step heat kernels)
};

inline Tiles make_tiles(int nx, int ny, int nz, int zc, int rows = 8) {
    Tiles t;
    t.nx = nx; t.ny = ny; t.nz = nz; t.zc = zc;
    t.rows = rows;
    t.ntx = (nx + 31) / 32;
    t.nty = (ny + rows - 1) / rows;
    t.ntz = (nz + zc - 1) / zc;
    t.ntiles = (long long)t.ntx * t.nty * t.ntz;
    return t;
}

// The z-chunk of a z-marching kernel, a multiple of the `lo` planes it takes at a time less `off`. A
// block takes ceil(tiles / wave) tiles one after another, and a tile costs its planes and about one more
// (the planes below and above its first and last): the chunk with the least of that product is taken,
// with a quarter of a tile for the uneven end. Large grids keep chunks of 6 to 20 planes; a grid that
// does not fill the SMs takes the thinnest, since a step is then as long as one tile. Measured,
// µs a step, chunks of 4, 8, 16 or 32 planes by their even spread alone and by this rule: a radiating f64
// block of 150 × 121 × 93 cells 67.6 and 55.8, a filled f64 32³ one 9.9 and 6.4, a lossy f64 32 × 24 × 31
// cavity 11.3 and 9.5, an FP32 31 × 27 × 43 one 17.2 and 15.6.
inline int choose_zc(int nx, int ny, int nz, unsigned resident, int lo = 1, int off = 0) {
    int best = lo - off;
    double best_cost = -1.0;
    for (int zc = lo - off; zc < nz + lo && zc <= 64; zc += lo) {
        const long long rounds = (make_tiles(nx, ny, nz, zc).ntiles + resident - 1) / resident;
        const double cost = ((double)rounds + 0.25) * (zc + 1);
        if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = zc; }
    }
    return best;
}
// The z-chunk of a hall's step, a multiple of its `lo` planes a stage. A hall's tile is light, so besides the
// rounds of a block the planes count that an SM's blocks march between them, mostly on the fullest SM. Chunks
// of more than eight stages gain nothing more. Fitted to sweeps of the chunk over 59 grids of the cp.async
// form and 14 of the TMA one: its choices are 1.5 and 0.5 % from the best on the mean (choose_zc's 3.0 and
// 1.6), and none is slower than chunks of 4, 8, 16 or 32 planes by their even spread by more than 4 %. Measured,
// µs a step by choose_zc and by this: 255 × 64 × 64 nodes in FP32 16.7 and 14.8, 65 × 90 × 50 10.7 and 9.5;
// 33 × 33 × 200 in f64 10.6 and 9.9; by TMA 64 × 64 × 256 10.6 and 10.3, 128³ 16.0 and 15.0.
inline int choose_hall_zc(int nx, int ny, int nz, unsigned sms, unsigned resident, int lo) {
    int best = lo;
    double best_cost = -1.0;
    for (int zc = lo; zc < nz + lo && zc <= 8 * lo; zc += lo) {
        const long long tiles = make_tiles(nx, ny, nz, zc).ntiles;
        const double mean = (double)tiles / sms, most = (double)((tiles + sms - 1) / sms);
        const double rounds = (double)((tiles + resident - 1) / resident);
        const double cost = (0.75 * most + 0.25 * mean + rounds) * (zc + 0.8);
        if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = zc; }
    }
    return best;
}
// The blocks of a wave of yee_tma_step that take tiles: with a near-field box one is the box's. Tiles cut for
// the whole wave and stepped by one block less took a round more wherever they filled their rounds, a cavity
// in a hundred. Those, µs a step for the whole wave and for the blocks there are: 64 × 64 × 256 of mixed ε
// 24.9 and 21.0, 192 × 32 × 256 32.4 and 30.0, 217 × 145 × 255 of one medium 89.6 and 81.9; the smallest,
// whose last round is a few tiles long, lose as they leave their thin chunks: 59 × 46 × 146 13.5 and 14.4,
// 64 × 32 × 256 of mixed ε 17.1 and 18.2.
inline unsigned yee_tile_blocks(unsigned wave, bool near) { return near && wave > 1 ? wave - 1 : wave; }
// The row pitch, in floats, of a cavity's padded FP32 lattice. Rows start on 32-byte sectors: with the 16
// bytes that TMA asks for, every store of a warp's 32 nodes cut a sector in two at both ends on every other
// row (384³ 560 -> 528 us a step, 256³ 174 -> 160, 160³ 51.4 -> 48.9, 128³ of mixed ε 37.5 -> 36.8; 96³, which
// L2 holds, 17.2 both ways). Whole 128-byte lines gave 384³ 517 but 96³ 17.6 and 128³ of mixed ε 38.3: the
// wider rows crowd a lattice out of L2. Four floats stay for a lattice that only they leave indexable by 32
// bits, and where the free memory may not hold all that a cavity ever allocates at the wider pitch: two sets
// of fields, three gains, Mur's three, a checkpoint's six, and media, masks and staging of 24 arrays' size.
inline unsigned cavity_row_pitch(int nx, int ny, int nz, size_t free_bytes) {
    const unsigned narrow = (unsigned)((nx + 1 + 3) & ~3), wide = (unsigned)((nx + 1 + 7) & ~7);
    const size_t lattice = (size_t)wide * ((size_t)ny + 1) * ((size_t)nz + 1);
    return lattice < ((size_t)1 << 32) && lattice <= free_bytes / (48 * sizeof(float)) ? wide : narrow;
}
inline unsigned grid_for(const Tiles& t, unsigned resident) {
    return (unsigned)(t.ntiles < (long long)resident ? t.ntiles : (long long)resident);
}

}  // namespace pm
