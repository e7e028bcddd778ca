// The engine's own layout of an IQ3_S matrix: four bits a weight, no codebook.
//
// Every IQ3_S weight is d (1 + 2 s) m with m odd, |m| <= 15 (the codebook's magnitudes are 1, 3, ..., 15 and the sign bit gives
// the rest), so m = 2 t + 1 with t = -8 .. 7: one two's-complement nibble holds it exactly.  A matrix in this layout takes 4.25
// bits a weight against the 3.44 of block_iq3_s and its tiles (iq3s_tile.h), and needs no table: a nibble becomes an int8 operand
// 8 m = 16 t + 8 with one logic operation (and one shift for every second one), where an index, its codebook entry and its signs took
// about seven instructions and a 64 KB table per block.  The windows' products are bound by those instructions and by the table's place in
// shared memory, not by the bytes; the two layouts hold the same numbers.
//
// A half tile is 16 rows x 256 columns, 2176 bytes, for one warp that feeds mma.sync.m16n8k32 (lane = 4 g + q: fragment row g, thread
// q of its group); like the other layout's, the lane owns the weights 8 q .. 8 q + 7 of every 32-weight sub-block of rows g and g + 8:
//   0      2048   words [j 0..3][lane] of 16 bytes: row half h = j / 2, sub-blocks 4 (j & 1) .. + 3, one u32 each; byte i of a word:
//                 low nibble = weight 8 q + i, high nibble = weight 8 q + 4 + i
//   2048    128   [g] 16 bytes: scale nibbles of row g, of row g + 8 (nibble sb = the sub-block's s), d of the two rows (f16), zero
// A tile is two half tiles over the same 256 columns, so that one load of the rows' operands serves both: 32 consecutive rows, or (a
// stacked [gate; up] matrix) 16 gate rows and the 16 up rows of the same features.  A matrix of R x K is the sequence of tiles
// [R / 32 rounded up][K / 256]; rows past R have d = 0.
#pragma once

#include "iq3s_tile.h"

namespace fnxb {

constexpr int NAT_HALF_BYTES = 2176, NAT_TILE_BYTES = 2 * NAT_HALF_BYTES;
constexpr int NAT_META = 2048;

FNX_HD size_t nat_bytes(size_t rows, size_t cols) { return (rows + 31) / 32 * (cols / 256) * NAT_TILE_BYTES; }
// byte offset of the half tile that holds 16-row group i (of n) and 256-column block b (of KB)
FNX_HD size_t nat_half_at(size_t i, size_t n, size_t b, size_t KB, bool gate_up) {
    const size_t tile = gate_up ? (i < n / 2 ? i : i - n / 2) : i / 2, half = gate_up ? i >= n / 2 : i % 2;
    return (tile * KB + b) * NAT_TILE_BYTES + half * NAT_HALF_BYTES;
}

// row r (0..15) of a half tile from its GGML block; `grid`: the 512 codebook entries
FNX_HD void nat_put_block(uint8_t* tile, int r, const uint8_t* blk, const uint32_t* grid) {
    const uint8_t *qs = blk + 2, *qh = blk + 66, *signs = blk + 74, *scales = blk + 106;
    const int g = r & 7, h = r >> 3;
    for (int sb = 0; sb < 8; ++sb)
        for (int q = 0; q < 4; ++q) {
            uint32_t w = 0;
            for (int e = 0; e < 2; ++e) {
                const int k = 2 * q + e;
                const uint32_t mag = grid[(uint32_t) qs[8 * sb + k] | ((((uint32_t) qh[sb] >> k) & 1u) << 8)];
                for (int j = 0; j < 4; ++j) {
                    const int m = (int) ((mag >> (8 * j)) & 255u), s = (signs[4 * sb + q] >> (4 * e + j)) & 1;
                    const uint32_t t = (uint32_t) (((s ? -m : m) - 1) >> 1) & 15u;
                    w |= t << (8 * j + 4 * e);
                }
            }
            memcpy(tile + (((2 * h + (sb >> 2)) * 32 + 4 * g + q) * 16 + (sb & 3) * 4), &w, 4);
        }
    uint8_t* m = tile + NAT_META + g * 16;
    for (int j = 0; j < 4; ++j) m[4 * h + j] = scales[j];
    m[8 + 2 * h] = blk[0];
    m[9 + 2 * h] = blk[1];
    if (h == 0)
        for (int j = 12; j < 16; ++j) m[j] = 0;
}

// the inverse; `inv`: codebook index of four magnitudes, at (m0 >> 1) | (m1 >> 1) << 3 | (m2 >> 1) << 6 | (m3 >> 1) << 9 (every entry
// of the codebook is there once, so the block comes back bit for bit)
FNX_HD void nat_get_block(const uint8_t* tile, int r, uint8_t* blk, const uint16_t* inv) {
    for (int i = 0; i < IQ3S_BLOCK_BYTES; ++i) blk[i] = 0;
    uint8_t *qs = blk + 2, *qh = blk + 66, *signs = blk + 74, *scales = blk + 106;
    const int g = r & 7, h = r >> 3;
    for (int sb = 0; sb < 8; ++sb)
        for (int q = 0; q < 4; ++q) {
            const uint8_t* p = tile + (((2 * h + (sb >> 2)) * 32 + 4 * g + q) * 16 + (sb & 3) * 4);
            for (int e = 0; e < 2; ++e) {
                uint32_t key = 0;
                for (int j = 0; j < 4; ++j) {
                    const int t = (int) ((p[j] >> (4 * e)) & 15), m = 2 * (t < 8 ? t : t - 16) + 1, a = m < 0 ? -m : m;
                    key |= (uint32_t) (a >> 1) << (3 * j);
                    if (m < 0) signs[4 * sb + q] |= (uint8_t) (1u << (4 * e + j));
                }
                const int k = 2 * q + e;
                qs[8 * sb + k] = (uint8_t) (inv[key] & 255u);
                qh[sb] |= (uint8_t) (((inv[key] >> 8) & 1u) << k);
            }
        }
    const uint8_t* m = tile + NAT_META + g * 16;
    for (int j = 0; j < 4; ++j) scales[j] = m[4 * h + j];
    blk[0] = m[8 + 2 * h];
    blk[1] = m[9 + 2 * h];
}

}  // namespace fnxb
