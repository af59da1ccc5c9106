// Host test of the copies into several destinations (host_copy.h): every byte
// of every piece and nothing past it, for piece sizes from one byte to a few
// MB, empty ones among them, in chunks that cut the pieces anywhere.
#include <cstdio>
#include <algorithm>
#include <random>
#include <vector>

#include "host_copy.h"

int main() {
  std::mt19937 rng(5);
  int bad = 0;
  for (int round = 0; round < 60; round++) {
    const int n = 1 + rng() % 6;
    std::vector<std::vector<char>> dst(n);
    std::vector<lbm::host_copy::Piece> pieces;
    size_t total = 0;
    for (auto& d : dst) {
      const size_t bytes = round % 3 == 0 ? rng() % 5 : round % 3 == 1 ? rng() % 100000 : rng() % (size_t(7) << 20);
      d.assign(bytes + 64, 0);
      pieces.push_back({d.data(), bytes});
      total += bytes;
    }
    std::vector<char> src(total + 1);
    for (size_t i = 0; i < total; i++) src[i] = (char)(i * 131 + round + 1);
    const size_t chunk = 1 + rng() % (total + 1);
    for (size_t o = 0; o < total; o += chunk)
      lbm::host_copy::copy_parallel(pieces.data(), o, std::min(chunk, total - o), src.data() + o, round % 2);
    size_t at = 0;
    for (int i = 0; i < n; i++) {
      for (size_t b = 0; b < pieces[i].bytes; b++) bad += dst[i][b] != src[at + b];
      for (size_t b = pieces[i].bytes; b < dst[i].size(); b++) bad += dst[i][b] != 0;
      at += pieces[i].bytes;
    }
  }
  std::printf("wrong bytes %d\n", bad);
  return bad == 0 ? 0 : 1;
}
