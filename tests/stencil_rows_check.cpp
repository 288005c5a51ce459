// Host check of stencil_rows (csrc/setup_host.h): the kernels take a row's
// entries by their place in it.  The packed rows hold the whole stencil at both
// orders, a coefficient that is zero keeps the others' places, and a coefficient
// at a node the kernels do not read is refused.
#include <cstdio>
#include <stdexcept>

#include "setup_host.h"

using namespace owt;

static int unpack_mismatches(const Stencils &st, int which, const std::vector<int> &cols, const std::vector<double> &vals) {
  int bad = 0;
  for (int j = 0; j < st.N; ++j)
    for (int c = 0; c < st.N; ++c) {
      double s = 0.0;
      for (int e = 0; e < 5; ++e)
        if (cols[(size_t)j * 5 + e] == c) s += vals[(size_t)j * 5 + e];
      bad += s != st.b(which, j, c);
    }
  return bad;
}

int main() {
  int bad = 0;
  for (int N : {7, 8, 9, 10, 33})
    for (int order : {8, 6})
      for (int which : {0, 1}) {
        Stencils st = make_stencils(N, 2.0 / (N - 1.0), order);
        std::vector<int> cols, c2;
        std::vector<double> vals, v2;
        stencil_rows(st, which, cols, vals);
        int q = unpack_mismatches(st, which, cols, vals);
        // every coefficient in turn set to zero
        for (int j = 0; j < N; ++j)
          for (int e = 0; e < 5; ++e) {
            if (vals[(size_t)j * 5 + e] == 0.0) continue;
            Stencils z = st;
            z.B[which][(size_t)j * N + cols[(size_t)j * 5 + e]] = 0.0;
            stencil_rows(z, which, c2, v2);
            std::vector<double> want = vals;
            want[(size_t)j * 5 + e] = 0.0;
            q += c2 != cols || v2 != want;
          }
        // a coefficient beside the row's
        for (int j = 0; j < N; ++j)
          for (int c = 0; c < N; ++c) {
            bool in = false;
            for (int e = 0; e < 5; ++e) in = in || (vals[(size_t)j * 5 + e] != 0.0 && cols[(size_t)j * 5 + e] == c);
            if (in) continue;
            Stencils z = st;
            z.B[which][(size_t)j * N + c] = 1.0;
            bool refused = false;
            try {
              stencil_rows(z, which, c2, v2);
            } catch (const std::logic_error &) {
              refused = true;
            }
            q += !refused;
          }
        if (q) std::printf("N=%d order %d derivative %d: %d mismatches\n", N, order, which + 1, q);
        bad += q;
      }
  return bad ? 1 : 0;
}
