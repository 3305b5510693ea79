// How the search of many vectors (fm_rvq_tiles.cu) deals its tiles to pairs of blocks, and when it is the faster form.  Host code.
#pragma once

namespace fm {

struct RvqDeal {
  static constexpr int kMaxPairs = 80, kTileRows = 256;
  int first[2][kMaxPairs + 1];         // pair i has the tiles first[s][i] .. first[s][i + 1] of stack s
  int pairs, layers[2];                // of the stacks, the longer one first; 0: there is no second one

  // Tiles of the longer stack evenly, those of the other to whoever has fewest layers so far.
  void make(long long rows, int longer, int shorter, int sms) {
    const int tiles = static_cast<int>((rows + kTileRows - 1) / kTileRows), all = shorter > 0 ? 2 * tiles : tiles;
    pairs = sms / 2 < kMaxPairs ? sms / 2 : kMaxPairs;
    if (pairs > all) pairs = all;
    if (pairs < 1) pairs = 1;
    layers[0] = longer;
    layers[1] = shorter;
    int load[kMaxPairs], count[2][kMaxPairs] = {};
    for (int p = 0; p < pairs; ++p) {
      count[0][p] = tiles / pairs + (p < tiles % pairs ? 1 : 0);
      load[p] = count[0][p] * longer;
    }
    for (int left = shorter > 0 ? tiles : 0; left > 0;) {
      int least = load[0];
      for (int p = 1; p < pairs; ++p) least = load[p] < least ? load[p] : least;
      for (int p = 0; p < pairs && left > 0; ++p) {
        if (load[p] != least) continue;
        ++count[1][p];
        load[p] += shorter;
        --left;
      }
    }
    for (int s = 0; s < 2; ++s) {
      first[s][0] = 0;
      for (int p = 0; p < pairs; ++p) first[s][p + 1] = first[s][p] + count[s][p];
    }
  }

  // The busiest pair's time, in us: 5 for the launch, 7.5 for each tile (its vectors, its first scores, its last decision), 9.4 for each
  // layer of one and 6 for every 1024 entries of a layer.  Vectors that a tile could still hold cost as much as others.
  double us(int n_codes) const {
    double most = 0.0;
    for (int p = 0; p < pairs; ++p) {
      const int n0 = first[0][p + 1] - first[0][p], n1 = first[1][p + 1] - first[1][p];
      const double t = 5.0 + 7.5 * (n0 + n1) + (9.4 + 6.0 * n_codes / 1024) * (n0 * layers[0] + n1 * layers[1]);
      most = t > most ? t : most;
    }
    return most;
  }
};

// The chain of kernels (fm_rvq.cu): a layer takes 7.8 us, for every 1000 vectors 0.42 and 0.46 times its thousands of entries, and 0.1 for those
// past 32000, whose records and residuals no longer stay in L2.
inline double rvq_chain_us(long long rows, int layers, int n_codes) {
  const double k = static_cast<double>(rows) / 1000;
  return layers * (7.8 + k * (0.42 + 0.46 * n_codes / 1024) + (k > 32.0 ? 0.1 * (k - 32.0) : 0.0));
}

// A pair takes as long for a layer however few vectors it has, whereas the chain spreads a layer over the whole device, so what counts is how evenly
// tiles come out, and how many layers share what a tile costs besides.  Chain -> tiles, in us, 2048 entries:
//   1 layer     12000 vectors 24 -> 34, 18944 (the most that a tile per pair holds) 32 -> 36, 37888 60 -> 60, 64000 90 -> 109
//   2 layers    12000 47 -> 55, 18944 64 -> 57, 37888 119 -> 103, 64000 194 -> 207
//   8 layers    9600 165 -> 177, 12000 190 -> 178, 18944 259 -> 184, 19200 272 -> 336, 32000 415 -> 360, 48000 644 -> 532, 64000 827 -> 706
//   32 layers   9600 677 -> 705, 16000 931 -> 702, 25000 1314 -> 1415, 32000 1644 -> 1393
//   1 + 7       9600 166 -> 159, 16000 235 -> 180, 19200 277 -> 295, 32000 403 -> 365, 48000 633 -> 529, 64000 821 -> 683
// and of 256: 1 layer of 128000 vectors 77 -> 169, 8 of 9600 103 -> 101, 1 + 7 of 64000 405 -> 407.  Of 1250 calls of 256 to 2048 entries, 1 to 32
// layers, one stack or two, the rule takes the slower form in few, and loses 5 % where that is the tiles, 11 % where it is the chain.
inline bool rvq_tiles_pay(const RvqDeal& deal, long long rows, int n_codes) {
  return deal.us(n_codes) < rvq_chain_us(rows, deal.layers[0] + deal.layers[1], n_codes);
}

}  // namespace fm
