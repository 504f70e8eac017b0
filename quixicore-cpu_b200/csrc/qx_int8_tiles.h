// Tiles of the W8A8 tensor-core GEMM (qx_int8_gemm_tc.cu); host code without CUDA.
#pragma once

namespace qx {

// A tile's channels (na tiles of 128) and tokens.
struct Int8Tile {
  int na, bn;
};

// Cycles until the slowest SM has done its tiles. A 32-byte step of K takes what shared memory has to take in and give out
// at 128 bytes a cycle, (na * 128 + bn) rows fetched and na * (128 + bn) read, above the tensor pipe's na * bn / 2 for every
// tile; and no less than the 96 (256 channels: 200) at which the codes themselves come, however few the tokens: tiles of 32
// instead of 64 read them twice as often (36 rows 8192 x 4096 16.6 us with its two small kernels, 15.8 with 64). The results of a tile of 128 channels are stored beside the next one's products (two accumulators), those of
// 256 channels and of an SM's last tile with nothing beside them.
inline long long int8_tile_cycles(long long m, long long n, long long k, int na, int bn, int sm_count, long long* tiles_out) {
  const long long channels = na * 128;
  const long long tiles = (n + channels - 1) / channels * ((m + bn - 1) / bn);
  const long long rounds = (tiles + sm_count - 1) / sm_count;
  const long long moved = (channels + bn + na * (128 + bn)) / 4;
  const long long least = na == 2 ? 200 : 96;
  const long long products = (k + 31) / 32 * (moved > least ? moved : least), results = 8LL * na * bn;
  *tiles_out = tiles;
  if (na == 2) return rounds * (products + results);
  return rounds * (products > results ? products : results) + results;
}

// The largest of the tiles that are within a fiftieth of the fewest cycles, or within two twenty-fifths where they fill the
// SMs: smaller ones cost power in padding, which large products are short of (1024 rows 14336 x 4096 in a row 61 us with 224
// tiles of 256 tokens, 63 with 280 of 224). `only`: 1 or 2 leaves tiles of 128 or 256 channels, 0 both.
//
// Measured (us, this rule | tiles of 256 tokens, and of 256 channels wherever they gave six of ten SMs a tile) on 77 shapes
// of 33 to 6500 rows with every tile: 2.1 % above the best tile in the mean (16 % at most) | 21 % (twice at most); four slower
// by more than a hundredth, by less than a fiftieth.  200 rows 2048 x 8192 14.0 | 23.4, 512 rows 1024 x 4096 7.7 | 14.8, 300
// rows 14336 x 4096 24.8 | 36.9, 1300 rows 9000 x 2048 24.1 | 40.8, 547 rows 10140 x 4640 32.4 | 43.3.  The same tile for 2048
// rows 28672 x 8192 341 (128 x 256: 346), 4096 rows 14336 x 4096 181 (185), 2790 rows 18669 x 6560 258 (293), 243 rows
// 30851 x 976 20.3 (22.4).
inline Int8Tile choose_int8_tile(long long m, long long n, long long k, int sm_count, int only) {
  struct {
    Int8Tile tile;
    long long tiles, cycles;
  } choices[16];
  int count = 0;
  long long fewest = 0;
  for (int area = 512; area >= 32; area -= 32) {  // the largest first
    for (int na = 2; na >= 1; --na) {             // (of one size the one of more channels: less operand traffic)
      const int bn = area / na;
      if ((only != 0 && na != only) || bn * na != area || bn % 32 != 0 || bn > 256) continue;
      if (bn > 32 && bn - 32 >= m) continue;  // (nothing but padding in the last 32)
      auto& choice = choices[count++];
      choice.tile = Int8Tile{na, bn};
      choice.cycles = int8_tile_cycles(m, n, k, na, bn, sm_count, &choice.tiles);
      if (count == 1 || choice.cycles < fewest) fewest = choice.cycles;
    }
  }
  int at = 0;
  while (choices[at].cycles * (choices[at].tiles >= sm_count ? 46 : 49) > fewest * 50) ++at;  // (the fewest's own ends it)
  return choices[at].tile;
}

}  // namespace qx
