// Host build of the two ways from a float pair to a double
// (qcware_unitair_gb300/csrc/dfloat.cuh).
#include "dfloat.cuh"

using namespace gbsv;

struct Pair {
  double x, y;
};

extern "C" void dfj_join(const float* re, const float* im, int count,
                         double* by_integers, double* by_addition) {
  for (int i = 0; i < count; ++i) {
    DC a;
    a.re = DF{re[2 * i], re[2 * i + 1]};
    a.im = DF{im[2 * i], im[2 * i + 1]};
    Pair p;
    df_join2(a, &p);
    by_addition[2 * i] = p.x;
    by_addition[2 * i + 1] = p.y;
    by_integers[2 * i] = df_join(a.re);
    by_integers[2 * i + 1] = df_join(a.im);
  }
}
