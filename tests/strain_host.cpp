// The device header's strain decomposition compiled for the host. The
// approximate units it uses (reciprocal square root, quick division) are exact
// to rounding here.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

using std::max;
using std::min;
static inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
static inline float __fdividef(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }
static inline float __uint_as_float(uint32_t a) {
  float r;
  memcpy(&r, &a, sizeof r);
  return r;
}

#include "xpbi_math.cuh"

using namespace xpbi;

// H = F - I by columns -> sigma, log of the clamped sigma, U and V by columns,
// and F with its singular values clamped to [lo, hi]
extern "C" void strain_svd(const float* H, int n, float* sig, float* e, float* U, float* V, float lo, float hi,
                           float* G) {
  for (int k = 0; k < n; ++k) {
    M3 h;
    for (int c = 0; c < 3; ++c) h.c[c] = v3(H[9 * k + 3 * c], H[9 * k + 3 * c + 1], H[9 * k + 3 * c + 2]);
    V3 l;
    bool near;
    const SVD s = strainSVD(h, l, near);
    const M3 g = withSigma(h, s, vclamp(s.sig, lo, hi), near);
    for (int c = 0; c < 3; ++c) {
      sig[3 * k + c] = s.sig[c];
      e[3 * k + c] = l[c];
      for (int r = 0; r < 3; ++r) {
        U[9 * k + 3 * c + r] = s.U.c[c][r];
        V[9 * k + 3 * c + r] = s.V.c[c][r];
        G[9 * k + 3 * c + r] = g.c[c][r];
      }
    }
  }
}
