// The FP64 form's face flux in FP32 pairs (csrc/face_split.cuh), built for the CPU by the tests.
#include "face_split.cuh"

using namespace mhdgb;

extern "C" void halve(int n, const double* x, double* y) {
  for (int i = 0; i < n; i++) y[i] = d_half(x[i]);
}

// n faces: left and right states (12 primitives each, normal component first), fluxes (10 each), and
// whether the split applies.
extern "C" void faces(int n, const double* left, const double* right, double chg, int hllc, double* F, int* ok) {
  for (int i = 0; i < n; i++) {
    double l[NPRIM], r[NPRIM], f[NCONS];
    for (int q = 0; q < NPRIM; q++) {
      l[q] = left[i * NPRIM + q];
      r[q] = right[i * NPRIM + q];
    }
    ok[i] = face_flux_split(l, r, [&](int q, bool up) { return up ? l[q] : r[q]; }, 0.5 * chg, chg * chg, f, hllc != 0);
    for (int m = 0; m < NCONS; m++) F[i * NCONS + m] = f[m];
  }
}
