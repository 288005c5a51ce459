// Host check of noalloc_factor_block (csrc/noalloc_setup.h), the elimination the
// kernel runs: it stops where the columns repeat, writes the repeated ones and
// resumes for the last.  Bitwise the plain elimination for every length the entry
// point takes.
#include <cstdio>
#include <cstring>
#include <vector>

#include "noalloc_setup.h"

using namespace owt;

int main() {
  int bad = 0;
  for (int NY = 7; NY <= kNoallocMaxNY; ++NY) {
    const size_t nb = (size_t)kNoallocBandRows * NY;
    std::vector<unsigned char> m[2];
    NoallocSetup s[2];
    for (int q = 0; q < 2; ++q) {
      m[q].resize(noalloc_setup_bytes(NY));
      s[q] = noalloc_layout(m[q].data(), NY);
      noalloc_assemble(s[q], NY, 2.0);
    }
    int state[2] = {0, 0};
    noalloc_factor(s[0], NY);
    noalloc_factor_block(s[1], NY, 0, 1, state, [] {});
    if (std::memcmp(s[0].ab, s[1].ab, nb * sizeof(double)) || std::memcmp(s[0].piv, s[1].piv, NY)) {
      std::printf("NY=%d: factors differ\n", NY);
      ++bad;
    }
  }
  return bad ? 1 : 0;
}
