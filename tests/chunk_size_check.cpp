// Host check of even_chunk (lgpu_chunks.h), compiled with g++ by test_chunk_size.py.
//
// Usage: chunk_size_check blocks most least n...  (a negative n: an excluded condition
// of -n electrons). Prints the chunk, the chunks that the layout makes of it, and the
// chunks with one electron less and with the most.
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>

#include "lgpu_chunks.h"

int main(int argc, char** argv) {
  const int blocks = std::atoi(argv[1]), most = std::atoi(argv[2]), least = std::atoi(argv[3]);
  std::vector<int> n;
  std::vector<unsigned char> take;
  for (int k = 4; k < argc; ++k) {
    const int v = std::atoi(argv[k]);
    n.push_back(std::abs(v));
    take.push_back(v > 0);
  }
  const int ns = (int)n.size();
  auto chunks = [&](int chunk) {
    std::vector<int> prefix(ns + 1), part(ns);
    std::vector<std::pair<int, int>> rem;
    const auto lay = lgpu::layout_pass(ns, n.data(), take.data(), chunk, prefix.data(), part.data(), rem);
    return lay.first + lay.second;
  };
  const int c = lgpu::even_chunk(ns, n.data(), take.data(), blocks, most, least);
  std::printf("%d %d %d %d\n", c, chunks(c), c > 1 ? chunks(c - 1) : 1 << 30, chunks(most));
  return 0;
}
