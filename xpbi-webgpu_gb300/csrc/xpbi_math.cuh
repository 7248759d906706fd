// Device math of the XPBI substep: SPH kernels, grid helpers, 3x3 SVD,
// StVK-Hencky and the five return mappings. Restates the math of
// web/js/shaders/common.js (cited per function) in f32 with the same
// operation order, so results track the WGSL to rounding.
#pragma once
#include "xpbi_internal.h"

namespace xpbi {

// ----------------------------------------------------------------- vectors
struct V3 {
  float x, y, z;
  __device__ __forceinline__ float& operator[](int k) { return k == 0 ? x : (k == 1 ? y : z); }
  __device__ __forceinline__ float operator[](int k) const { return k == 0 ? x : (k == 1 ? y : z); }
};
__device__ __forceinline__ V3 v3(float a, float b, float c) { return V3{a, b, c}; }
__device__ __forceinline__ V3 splat(float s) { return V3{s, s, s}; }
__device__ __forceinline__ V3 xyz(const float4& a) { return V3{a.x, a.y, a.z}; }
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator-(V3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ V3 operator*(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 operator*(float s, V3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ V3 operator*(V3 a, V3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ V3 operator/(V3 a, float s) { return {a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ V3 operator/(V3 a, V3 b) { return {a.x / b.x, a.y / b.y, a.z / b.z}; }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float length(V3 a) { return sqrtf(dot(a, a)); }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
__device__ __forceinline__ V3 vclamp(V3 v, float lo, float hi) {
  return {clampf(v.x, lo, hi), clampf(v.y, lo, hi), clampf(v.z, lo, hi)};
}
__device__ __forceinline__ V3 vmaxs(V3 v, float m) { return {fmaxf(v.x, m), fmaxf(v.y, m), fmaxf(v.z, m)}; }
__device__ __forceinline__ V3 vlog(V3 v) { return {logf(v.x), logf(v.y), logf(v.z)}; }
__device__ __forceinline__ V3 vexp(V3 v) { return {expf(v.x), expf(v.y), expf(v.z)}; }
__device__ __forceinline__ V3 vsqrt(V3 v) { return {sqrtf(v.x), sqrtf(v.y), sqrtf(v.z)}; }

// Two f32 lanes in one 64-bit register pair (sm_100's packed add / multiply /
// fused multiply-add, each lane rounded like the scalar operation): the
// neighbour passes are issue-bound, and these do two candidates' or two
// neighbours' arithmetic per instruction.
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float lo2(F2 a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi2(F2 a) { return __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Column-major 3x3, c[j] = column j (WGSL mat3x3f).
struct M3 {
  V3 c[3];
};
__device__ __forceinline__ M3 mzero() { return {{splat(0.f), splat(0.f), splat(0.f)}}; }
__device__ __forceinline__ M3 mident() { return {{v3(1.f, 0.f, 0.f), v3(0.f, 1.f, 0.f), v3(0.f, 0.f, 1.f)}}; }
__device__ __forceinline__ M3 minusIdent(const M3& A) {
  return {{v3(A.c[0].x - 1.f, A.c[0].y, A.c[0].z), v3(A.c[1].x, A.c[1].y - 1.f, A.c[1].z),
           v3(A.c[2].x, A.c[2].y, A.c[2].z - 1.f)}};
}
__device__ __forceinline__ V3 mul(const M3& A, V3 v) { return A.c[0] * v.x + A.c[1] * v.y + A.c[2] * v.z; }
__device__ __forceinline__ M3 mul(const M3& A, const M3& B) {
  return {{mul(A, B.c[0]), mul(A, B.c[1]), mul(A, B.c[2])}};
}
__device__ __forceinline__ M3 transpose(const M3& A) {
  return {{v3(A.c[0].x, A.c[1].x, A.c[2].x), v3(A.c[0].y, A.c[1].y, A.c[2].y),
           v3(A.c[0].z, A.c[1].z, A.c[2].z)}};
}
__device__ __forceinline__ M3 madd(const M3& A, const M3& B) {
  return {{A.c[0] + B.c[0], A.c[1] + B.c[1], A.c[2] + B.c[2]}};
}
__device__ __forceinline__ M3 mscale(const M3& A, float s) { return {{A.c[0] * s, A.c[1] * s, A.c[2] * s}}; }
__device__ __forceinline__ float det(const M3& A) { return dot(A.c[0], cross(A.c[1], A.c[2])); }

// Plane-major 3x3 storage: entry (col c, row r) of particle i at [(3c+r)*N + i].
__device__ __forceinline__ M3 loadM(const float* __restrict__ P, uint32_t N, uint32_t i) {
  M3 m;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    m.c[c] = v3(P[(3 * c + 0) * (size_t)N + i], P[(3 * c + 1) * (size_t)N + i], P[(3 * c + 2) * (size_t)N + i]);
  return m;
}
__device__ __forceinline__ void storeM(float* __restrict__ P, uint32_t N, uint32_t i, const M3& m) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    P[(3 * c + 0) * (size_t)N + i] = m.c[c].x;
    P[(3 * c + 1) * (size_t)N + i] = m.c[c].y;
    P[(3 * c + 2) * (size_t)N + i] = m.c[c].z;
  }
}

// The SPH kernels are formed in the pair loops of solve.cu: Wendland C2 and its
// gradient (support 2h, common.js:63-79) in radial2 and xsph, the PBF kernels
// (common.js:81-94) in pbfPair.

// ----------------------------------------------------------------- grid
// common.js:97-103. Saturating f32->i32 (NaN -> 0) before clamping.
__device__ __forceinline__ int axisCell(float p, float o, float cs, int dim) {
  float fl = floorf((p - o) / cs);
  fl = fminf(fmaxf(fl, 0.f), (float)(dim - 1));
  return (int)fl;
}
struct I3 {
  int x, y, z;
};
__device__ __forceinline__ I3 cellCoord(const SceneDev& S, V3 p) {
  return I3{axisCell(p.x, S.origin[0], S.cs, S.dims[0]), axisCell(p.y, S.origin[1], S.cs, S.dims[1]),
            axisCell(p.z, S.origin[2], S.cs, S.dims[2])};
}
__device__ __forceinline__ uint32_t cellIndex(const SceneDev& S, int x, int y, int z) {
  return (uint32_t)x + (uint32_t)y * (uint32_t)S.dims[0] + (uint32_t)z * (uint32_t)(S.dims[0] * S.dims[1]);
}

// ----------------------------------------------------------------- svd3
struct SVD {
  M3 U;
  V3 sig;
  M3 V;
};

__device__ __forceinline__ void swapf(float& a, float& b) { float t = a; a = b; b = t; }
__device__ __forceinline__ void swapv(V3& a, V3& b) { V3 t = a; a = b; b = t; }

// One Jacobi rotation of two columns bp, bq of F V (squared lengths np, nq)
// that makes them orthogonal, V's columns vp, vq rotated along; nothing if
// they are already, to rounding, or one is negligible against the other.
// `more`: another sweep is needed (a sweep of angles below 2e-4 leaves
// columns orthogonal to their square). MUFU based: the angle is off by a few
// ulp.
__device__ __forceinline__ void jacobiRot(V3& bp, V3& bq, float& np, float& nq, V3& vp, V3& vq, bool& more) {
  const float g = dot(bp, bq);
  if (g * g <= 1e-14f * (np * nq)) return;
  const float tau = __fdividef(nq - np, 2.f * g);
  if (!(fabsf(tau) < 1e9f)) return;
  const float h2 = 1.f + tau * tau;
  const float root = h2 * rsqrtf(h2);
  const float t = __fdividef(1.f, tau >= 0.f ? tau + root : tau - root);
  more |= fabsf(t) > 2e-4f;
  const float c = rsqrtf(1.f + t * t);
  const float s = t * c;
  np -= t * g;
  nq += t * g;
  const V3 b = bp, v = vp;
  bp = c * b - s * bq;
  bq = s * b + c * bq;
  vp = c * v - s * vq;
  vq = s * v + c * vq;
}

// 1 / sqrt(d): the MUFU's value after one Newton step
__device__ __forceinline__ float rsqrtNewton(float d) {
  const float r = rsqrtf(d);
  return r * fmaf(-0.5f * d * r, r, 1.5f);
}
__device__ __forceinline__ V3 normalizeFast(V3 a) { return a * rsqrtNewton(dot(a, a)); }

// A vector whose length is 1 up to the rounding of approximate cosines, with
// the error's first order taken off.
__device__ __forceinline__ V3 renormalize(V3 a) { return a * fmaf(-0.5f, dot(a, a), 1.5f); }

// SVD with the reference's conventions (common.js:105-184: sigma descending,
// the last one negative if det F < 0, U and V rotations) by one-sided Jacobi
// sweeps: the columns of F V are made orthogonal instead of diagonalising
// F^T F, so the squared condition number of F never enters (a singular value
// keeps its relative accuracy) and F V hands over U sigma. The sweeps, at most
// the reference's six, end once their angles are small: three for a warp of
// strained particles.
__device__ __forceinline__ SVD svd3Fast(const M3& F) {
  V3 b0 = F.c[0], b1 = F.c[1], b2 = F.c[2];
  V3 a0 = v3(1.f, 0.f, 0.f), a1 = v3(0.f, 1.f, 0.f), a2 = v3(0.f, 0.f, 1.f);
  float n0 = dot(b0, b0), n1 = dot(b1, b1), n2 = dot(b2, b2);
#pragma unroll 1
  for (int sweep = 0; sweep < 6; ++sweep) {
    bool more = false;
    jacobiRot(b0, b1, n0, n1, a0, a1, more);
    jacobiRot(b0, b2, n0, n2, a0, a2, more);
    jacobiRot(b1, b2, n1, n2, a1, a2, more);
    if (!more) break;
  }
  // the approximate cosines leave V's columns, and F V's with them, a few ulp
  // off length 1: the first order of that off both
  const float k0 = fmaf(-0.5f, dot(a0, a0), 1.5f), k1 = fmaf(-0.5f, dot(a1, a1), 1.5f),
              k2 = fmaf(-0.5f, dot(a2, a2), 1.5f);
  a0 = a0 * k0;
  a1 = a1 * k1;
  a2 = a2 * k2;
  b0 = b0 * k0;
  b1 = b1 * k1;
  b2 = b2 * k2;
  V3 sig = v3(sqrtf(dot(b0, b0)), sqrtf(dot(b1, b1)), sqrtf(dot(b2, b2)));
  if (sig.x < sig.y) { swapf(sig.x, sig.y); swapv(a0, a1); swapv(b0, b1); }
  if (sig.x < sig.z) { swapf(sig.x, sig.z); swapv(a0, a2); swapv(b0, b2); }
  if (sig.y < sig.z) { swapf(sig.y, sig.z); swapv(a1, a2); swapv(b1, b2); }
  if (dot(cross(a0, a1), a2) < 0.f) {
    a2 = -a2;
    b2 = -b2;
  }
  if (dot(cross(b0, b1), b2) < 0.f) sig.z = -sig.z;  // det F (V is a rotation)
  SVD out;
  out.V = {{a0, a1, a2}};
  V3 u0, u1;
  const float eps = 1e-8f;
  if (sig.x > eps) u0 = normalizeFast(b0);
  else u0 = v3(1.f, 0.f, 0.f);
  if (sig.y > eps) {
    u1 = b1 - dot(b1, u0) * u0;
    const float l2 = dot(u1, u1);
    if (l2 > eps * eps) u1 = u1 * rsqrtNewton(l2);
    else u1 = normalizeFast(cross(v3(0.f, 1.f, 0.f), u0) + splat(1e-4f));
  } else {
    V3 a = cross(u0, v3(0.f, 1.f, 0.f));
    if (dot(a, a) < 1e-8f) a = cross(u0, v3(1.f, 0.f, 0.f));
    u1 = normalizeFast(a);
  }
  const V3 u2 = cross(u0, u1);
  out.U = {{u0, u1, u2}};
  out.sig = sig;
  return out;
}

// Eigenvalues d and eigenvectors (the columns a) of a symmetric 3x3 matrix by
// Jacobi rotations, in no particular order. A rotation zeroes one off-diagonal
// exactly, moves its diagonals by t apq and turns the other two off-diagonals
// and the vectors; off-diagonals below 1e-9 of the largest entry are left.
struct Sym3 {
  float xx, yy, zz, xy, xz, yz;
};
__device__ __forceinline__ void eigRot(float& dp, float& dq, float& apq, float& arp, float& arq, V3& vp, V3& vq,
                                       float small, bool& more) {
  if (!(fabsf(apq) > small)) return;
  const float tau = __fdividef(dq - dp, 2.f * apq);
  const float h2 = 1.f + tau * tau;
  const float root = h2 * rsqrtf(h2);
  const float t = __fdividef(1.f, tau >= 0.f ? tau + root : tau - root);
  more |= fabsf(t) > 2e-4f;
  const float c = rsqrtf(1.f + t * t);
  const float s = t * c;
  dp -= t * apq;
  dq += t * apq;
  apq = 0.f;
  const float x = arp, y = arq;
  arp = c * x - s * y;
  arq = s * x + c * y;
  const V3 p = vp, q = vq;
  vp = c * p - s * q;
  vq = s * p + c * q;
}
__device__ __forceinline__ float maxAbs(const Sym3& S) {
  return fmaxf(fmaxf(fmaxf(fabsf(S.xx), fabsf(S.yy)), fabsf(S.zz)),
               fmaxf(fmaxf(fabsf(S.xy), fabsf(S.xz)), fabsf(S.yz)));
}
__device__ __forceinline__ void eigSym(Sym3 S, V3& d, M3& V) {
  V3 a0 = v3(1.f, 0.f, 0.f), a1 = v3(0.f, 1.f, 0.f), a2 = v3(0.f, 0.f, 1.f);
  const float small = 1e-9f * maxAbs(S);
#pragma unroll 1
  for (int sweep = 0; sweep < 6; ++sweep) {
    bool more = false;
    eigRot(S.xx, S.yy, S.xy, S.xz, S.yz, a0, a1, small, more);
    eigRot(S.xx, S.zz, S.xz, S.xy, S.yz, a0, a2, small, more);
    eigRot(S.yy, S.zz, S.yz, S.xy, S.xz, a1, a2, small, more);
    if (!more) break;
  }
  d = v3(S.xx, S.yy, S.zz);
  V = {{renormalize(a0), renormalize(a1), renormalize(a2)}};
}

// U diag(d) V^T (common.js:182-184)
__device__ __forceinline__ M3 diagMul(const M3& U, V3 d, const M3& V) {
  M3 Ud = {{U.c[0] * d.x, U.c[1] * d.y, U.c[2] * d.z}};
  return mul(Ud, transpose(V));
}

// ----------------------------------------------------------------- StVK-Hencky
// common.js:186-201
__device__ __forceinline__ V3 safeSig(V3 s) { return vclamp(s, 1e-3f, 1e3f); }
// The SVD of F = I + H and the logs of its (clamped) singular values. Near the
// identity, where a granular body flows, f32 singular values of 1 + O(1e-4)
// keep three digits of the strain; there the eigenvalues x of
// F^T F - I = H + H^T + H^T H are taken instead, which H's own digits carry,
// with log sigma = log(1 + x) / 2. (The singular values then come in no
// particular order: the material models do not depend on it.) That needs
// det F > 0 (the eigenvalues of F^T F do not see an inversion, whose smallest
// singular value is negative) and a bound on x away from -1: with the entries
// of F^T F - I below 0.5 and its absolute row sums below 0.75, |x| < 0.75 and
// sigma lies in (0.5, 1.33), inside safeSig's bounds. (The entries alone do
// not: flattened to nothing along (1, 1, 1), every one is -1/3 and an
// eigenvalue is -1.) Elsewhere, NaN included, the SVD of F itself keeps the
// small singular values and the sign. near: which of the two it was.
__device__ __forceinline__ SVD strainSVD(const M3& H, V3& e, bool& near) {
  const V3 x = H.c[0], y = H.c[1], z = H.c[2];
  const Sym3 S = {fmaf(2.f, x.x, dot(x, x)), fmaf(2.f, y.y, dot(y, y)), fmaf(2.f, z.z, dot(z, z)),
                  (x.y + y.x) + dot(x, y),   (x.z + z.x) + dot(x, z),   (y.z + z.y) + dot(y, z)};
  const M3 F = {{v3(1.f + x.x, x.y, x.z), v3(y.x, 1.f + y.y, y.z), v3(z.x, z.y, 1.f + z.z)}};
  const float xy = fabsf(S.xy), xz = fabsf(S.xz), yz = fabsf(S.yz);
  const float rows = fmaxf(fmaxf(fabsf(S.xx) + xy + xz, fabsf(S.yy) + xy + yz), fabsf(S.zz) + xz + yz);
  near = maxAbs(S) < 0.5f && rows < 0.75f && det(F) > 0.f;
  if (near) {
    SVD out;
    V3 d;
    eigSym(S, d, out.V);
    e = v3(0.5f * log1pf(d.x), 0.5f * log1pf(d.y), 0.5f * log1pf(d.z));
    const V3 r = v3(rsqrtNewton(1.f + d.x), rsqrtNewton(1.f + d.y), rsqrtNewton(1.f + d.z));
    out.sig = v3((1.f + d.x) * r.x, (1.f + d.y) * r.y, (1.f + d.z) * r.z);
#pragma unroll
    for (int k = 0; k < 3; ++k) out.U.c[k] = (out.V.c[k] + mul(H, out.V.c[k])) * r[k];
    return out;
  }
  const SVD out = svd3Fast(F);
  e = vlog(safeSig(out.sig));
  return out;
}
// F = I + H with its singular values replaced by s. Near the identity what the
// map changed is added to F, which keeps the digits of a small strain; far from
// it that would leave the rounding of a large F on a result that the map may
// have brought back to sigma = 1 (F of size 30 to 2e-5, 2e-7 composed anew).
__device__ __forceinline__ M3 withSigma(const M3& H, const SVD& sv, V3 s, bool near) {
  return near ? madd(madd(H, diagMul(sv.U, s - sv.sig, sv.V)), mident()) : diagMul(sv.U, s, sv.V);
}
// energy from the logs e of the clamped singular values; its gradient is
// (2 mu e + lam tr e) / safeSig(sig)
__device__ __forceinline__ float stvkPsi(V3 e, float mu, float lam) {
  float tr = e.x + e.y + e.z;
  return mu * dot(e, e) + 0.5f * lam * tr * tr;
}

// ----------------------------------------------------------------- return maps
// A return map's result: the singular values and the logs of their clamped
// values (safeSig), which the energy and its gradient take. The maps that work
// on the logs (Drucker-Prager, von Mises) hand them on, not the rounded log of
// a rounded exponential.
struct Mapped {
  V3 sig, e;
};
__device__ __forceinline__ Mapped mappedLog(V3 e) {
  const V3 s = vexp(e);
  // log(clamp(exp e)) = clamp(e): the bounds are the logs of safeSig's
  return Mapped{s, vclamp(e, -6.90775528f, 6.90775528f)};
}
__device__ __forceinline__ Mapped mappedSig(V3 s) { return Mapped{s, vlog(safeSig(s))}; }
// Drucker-Prager (common.js:205-221); e0 = log(safeSig(sig))
__device__ __forceinline__ Mapped rmDruckerPrager(V3 sig, V3 e0, const MatDev& m, float mu, float lam) {
  float alpha = m.p0, coh = m.p1;
  V3 e = e0 - splat(coh);
  float tr = e.x + e.y + e.z;
  V3 dev = e - splat(tr / 3.f);
  float dn = length(dev);
  if (dn < 1e-9f || tr > 0.f) return mappedLog(splat(coh));
  float dg = dn + alpha * (3.f * lam + 2.f * mu) / (2.f * mu) * tr;
  if (dg <= 0.f) return Mapped{sig, e0};
  V3 en = e - (dg / dn) * dev;
  return mappedLog(en + splat(coh));
}
// Von Mises (common.js:223-234)
__device__ __forceinline__ Mapped rmVonMises(V3 sig, V3 e, const MatDev& m, float mu) {
  float sigY = m.p0;
  float tr = e.x + e.y + e.z;
  V3 dev = e - splat(tr / 3.f);
  float dn = length(dev);
  float dg = dn - sigY / (2.f * mu);
  if (dg <= 0.f || dn < 1e-9f) return Mapped{sig, e};
  return mappedLog(e - (dg / dn) * dev);
}
// Herschel-Bulkley, b-bar-e form with bisection (common.js:236-280)
__device__ __forceinline__ V3 rmHerschelBulkley(V3 sig, const MatDev& m, float mu, float dt) {
  float sigY = m.p0, hexp = m.p1, eta = m.p2;
  V3 s3 = safeSig(sig);
  float J = s3.x * s3.y * s3.z;
  V3 bbar = s3 * s3 * powf(J, (float)(-2.0 / 3.0));
  float trb = bbar.x + bbar.y + bbar.z;
  V3 devb = bbar - splat(trb / 3.f);
  float sPre = mu * length(devb);
  float sY = (float)0.816496580927726 * sigY;  // sqrt(2/3)
  if (sPre <= sY || sPre < 1e-12f) return sig;
  float muT = (trb / 3.f) * mu;
  float sNew;
  if (fabsf(hexp - 1.f) < 1e-3f || eta < 1e-9f) {
    sNew = sPre - (sPre - sY) / (1.f + eta / (2.f * muT * dt));
  } else {
    float ih = 1.f / hexp;
    float ei = powf(eta, ih);
    float lo = sY, hi = sPre;
#pragma unroll 1
    for (int it = 0; it < 18; ++it) {
      float mid = 0.5f * (lo + hi);
      float g = ei * (mid - sPre) + 2.f * muT * dt * powf(fmaxf(mid - sY, 0.f), ih);
      if (g > 0.f) hi = mid;
      else lo = mid;
    }
    sNew = 0.5f * (lo + hi);
  }
  V3 bNew = devb * (sNew / sPre) + splat(trb / 3.f);
  bNew = vmaxs(bNew, 1e-6f);
  float detB = bNew.x * bNew.y * bNew.z;
  bNew = bNew * powf(detB, (float)(-1.0 / 3.0));
  return vsqrt(bNew) * powf(J, (float)(1.0 / 3.0));
}
// NACC, b^E form with fracture-friendly hardening (common.js:287-364)
__device__ __forceinline__ V3 rmNACC(V3 sig, const MatDev& m, float mu, float lam, float alphaIn, float& alphaOut) {
  float beta = m.p1, xi = m.p2, Mf = m.p3;
  float kappa = (float)(2.0 / 3.0) * mu + lam;
  float alpha = alphaIn;
  V3 s3 = safeSig(sig);
  float Jtr = s3.x * s3.y * s3.z;
  V3 b2 = s3 * s3;
  float trb = b2.x + b2.y + b2.z;
  V3 devb = b2 - splat(trb / 3.f);
  V3 sHat = mu * powf(Jtr, (float)(-2.0 / 3.0)) * devb;
  float sNorm = length(sHat);
  const float sqrt15 = (float)1.224744871391589;  // sqrt(1.5)
  float q = sqrt15 * sNorm;
  float p = -0.5f * kappa * (Jtr * Jtr - 1.f);
  alpha = clampf(alpha, -0.25f, 0.4f);
  float p0 = kappa * (0.00001f + sinhf(fminf(xi * fmaxf(-alpha, 0.f), 4.f)));
  float b = 1.f + 2.f * beta;
  V3 outSig = sig;
  if (p > p0) {
    float Jn = sqrtf(fmaxf(-2.f * p0 / kappa + 1.f, 1e-6f));
    outSig = splat(powf(Jn, (float)(1.0 / 3.0)));
    alpha = alpha + logf(Jtr / Jn);
  } else if (p < -beta * p0) {
    float Jn = sqrtf(fmaxf(2.f * beta * p0 / kappa + 1.f, 1e-6f));
    outSig = splat(powf(Jn, (float)(1.0 / 3.0)));
    alpha = alpha + logf(Jtr / Jn);
  } else {
    float y = b * q * q + Mf * Mf * (p + beta * p0) * (p - p0);
    if (y > 1e-4f && sNorm > 1e-9f) {
      if (p0 > 1e-4f && p < p0 - 1e-4f && p > -beta * p0 + 1e-4f) {
        float pc = (1.f - beta) * p0 * 0.5f;
        float lenDir = sqrtf((pc - p) * (pc - p) + (-q) * (-q));
        if (lenDir > 1e-9f) {
          float Dp = (pc - p) / lenDir;
          float Dq = -q / lenDir;
          float Aq = Mf * Mf * Dp * Dp + b * Dq * Dq;
          float Bq = Mf * Mf * Dp * (2.f * pc - p0 + beta * p0);
          float Cq = Mf * Mf * (pc + beta * p0) * (pc - p0);
          float disc = Bq * Bq - 4.f * Aq * Cq;
          if (disc > 0.f && fabsf(Aq) > 1e-12f) {
            float l1 = (-Bq + sqrtf(disc)) / (2.f * Aq);
            float l2 = (-Bq - sqrtf(disc)) / (2.f * Aq);
            float px1 = pc + l1 * Dp;
            float px2 = pc + l2 * Dp;
            float px = px1;
            if ((p - pc) * (px2 - pc) > 0.f) px = px2;
            float Jx2 = -2.f * px / kappa + 1.f;
            if (Jx2 > 1e-8f) {
              float Jx = sqrtf(Jx2);
              if (Jx > 1e-4f) alpha = alpha + logf(Jtr / Jx);
            }
          }
        }
      }
      float qN = Mf * sqrtf(fmaxf(-(p + beta * p0) * (p - p0), 0.f) / b);
      float sNewNorm = qN / sqrt15;
      V3 bNew = (powf(Jtr, (float)(2.0 / 3.0)) / mu) * (sNewNorm / sNorm) * sHat + splat(trb / 3.f);
      bNew = vmaxs(bNew, 1e-6f);
      outSig = vsqrt(bNew);
    }
  }
  alphaOut = alpha;
  return outSig;
}
// Snow hardening of mu, lambda (common.js:366-375): the factor on both
__device__ __forceinline__ float hardening(const MatDev& m, float state) {
  return m.kind == kKindSnow ? expf(fminf(m.p2 * (1.f - state), 5.f)) : 1.f;
}
// Dispatch on the material kind (common.js:377-396) with the (hardened) mu,
// lambda; e = log(safeSig(sig)).
__device__ __forceinline__ Mapped returnMap(V3 sig, V3 e, const MatDev& m, float mu, float lam, float state, float dt,
                                            float& stateOut) {
  stateOut = state;
  switch (m.kind) {
    case 1u: return rmDruckerPrager(sig, e, m, mu, lam);
    case 2u: return mappedSig(rmNACC(sig, m, mu, lam, state, stateOut));
    case 3u: return rmVonMises(sig, e, m, mu);
    case 4u: return mappedSig(rmHerschelBulkley(sig, m, mu, dt));
    case 5u: {
      V3 sNew = v3(clampf(sig.x, 1.f - m.p0, 1.f + m.p1), clampf(sig.y, 1.f - m.p0, 1.f + m.p1),
                   clampf(sig.z, 1.f - m.p0, 1.f + m.p1));
      float jOld = sig.x * sig.y * sig.z;
      float jNew = sNew.x * sNew.y * sNew.z;
      stateOut = clampf(state * jOld / fmaxf(jNew, 1e-6f), 0.2f, 2.f);
      return mappedSig(sNew);
    }
    default: return Mapped{sig, e};
  }
}

}  // namespace xpbi
