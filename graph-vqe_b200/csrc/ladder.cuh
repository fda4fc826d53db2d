// Pauli-sum energies of ladder circuits: environments as Pauli components.
//
// Reference algorithm: ReverseMPS.sites / energy_chunk (test/tools/reverse_mps.py:39-82),
// the exact matrix product state in which every CX doubles a bond, contracted with each
// word; the SVD chain (sharded_mps.cuh:477-549) prepares the same state.
//
// A ladder circuit has layers of one-site gates, each followed by one CX on every bond in
// chain order (the linear and reverse_linear ansatz). Its exact site tensors need no SVD
// and no 16 x 16 products. CX = sum_b |b><b| (x) X^b (or, with the roles of the axes
// exchanged, sum_b Z^b (x) |x_b><x_b|), so with the right axis a site's tensor is
//   A[l, p, r] = prod_k V_k[r_k ^ l_k, r_{k-1}] W[p, r_4]
// with one bond bit per layer: 2 x 2 matrices V_k (the layer's gates) and W (the gates
// after the last CX). Sites are taken in the order in which each site's CX with its left
// neighbour comes before the one with its right neighbour (the chain is mirrored otherwise).
//
// An environment E[l, l'] over four bond bits is Hermitian, so it is kept as its 256 real
// Pauli components t = Tr(E s1 (x) s2 (x) s3 (x) s4), s in {I, X, Y, Z}, one digit per layer. In
// these a site is five sparse real stages, each on one digit or on two neighbouring ones:
//   S1  digit 1: flip of the first layer's Bloch vector n by l_1
//   Sk  digits k-1, k (k = 2, 3, 4): copy of the spin into r_{k-1}, rotation O_k (the Bloch matrix of
//       V_k), flip by l_k
//   SF  digit 4: copy into r_4, rotation W and the trace with the site's Pauli
// 8 + 3 x 36 multiply-adds per 4 + 16 components (fewer for real gates, whose rotations
// stay in the x-z plane) against two dense 16 x 16 x 32 products. The suffix environments are
// the dual components (w with value = sum t w), moved by the transposed stages. With real
// gates, components with an odd number of Y digits vanish while the word so far has an even
// number of Y codes, and the other way round: they are neither stored nor read.
//
// Layout: four lanes per environment, one per value of digit 4, each with the 64 components of
// digits 1-3 in registers, eight environments per warp (consecutive states of one path when
// there are eight). S1-S3 need no exchange; S4 and SF exchange digit 4 with one shuffle per
// component, and between identity codes not even that. A warp walks a whole path of trie
// nodes without touching memory except for the site's rotations (22 or 39 numbers) and the
// environments that several paths or a closure need. Those lie in global memory as
// [slot][digit 4][digits 1-3][state], so that eight states fill the 32-byte sectors.
#pragma once
#include "common.cuh"
#include "evolve.cuh"

namespace vqemps {

// Order of the digits' values (and of a quad's lanes): I 0, X 1, Y 2, Z 3.
constexpr int LAD_REAL_COEFS = 22;   // nx nz | k = 2, 3, 4: xx xz zx zz yy | W: xx xz zx zz yy
constexpr int LAD_COEFS = 39;        // n | k = 2, 3, 4: O row-major | W row-major
constexpr int LAD_MAX_LAYERS = 4;

struct LadGate {   // a one-site gate of a layer: fixed matrix or rotation
  int32_t mat, rot, param, pad;
  double angle;
};

struct LadCoefParams {
  const LadGate *gates;
  const int32_t *off;      // [n * (layers + 1) + 1]: gates of (ladder site, layer)
  const cplx *mats;
  const double *theta;     // B x P
  double *theta_keep;      // B x P copy of the angles
  int n, P, layers;
  int hadamard;            // the bond axis is x: gates are conjugated by H
  cplx prep[4];            // |0> -> initial state
  double *coef;            // [n][ncoef][B]
  int32_t *status;         // B
  double *poison;          // B: 0, or NaN when an angle is not finite
  double *leafval;         // B x nleaf: leaf 0 the norm, leaf 1 zero
  int nleaf;
};

__device__ __forceinline__ void mul2(const cplx *a, const cplx *b, cplx *o) {
  o[0] = cadd(cmul(a[0], b[0]), cmul(a[1], b[2]));
  o[1] = cadd(cmul(a[0], b[1]), cmul(a[1], b[3]));
  o[2] = cadd(cmul(a[2], b[0]), cmul(a[3], b[2]));
  o[3] = cadd(cmul(a[2], b[1]), cmul(a[3], b[3]));
}

// O[a][b] = Tr(s_a U s_b U^H) / 2 over x, y, z
__device__ __forceinline__ void bloch(const cplx *u, double *o) {
  const cplx ad = cmul(u[0], cconj(u[3])), bc = cmul(u[1], cconj(u[2]));
  const cplx ab = cmul(u[0], cconj(u[1])), cd = cmul(u[2], cconj(u[3]));
  const cplx ac = cmul(u[0], cconj(u[2])), bd = cmul(u[1], cconj(u[3]));
  o[0] = ad.x + bc.x;                      // M01 of U X U^H = a d* + b c*
  o[3] = -(ad.y + bc.y);
  o[6] = ab.x - cd.x;
  o[1] = ad.y - bc.y;                      // U Y U^H: M01 = -i a d* + i b c*
  o[4] = ad.x - bc.x;
  o[7] = ab.y - cd.y;
  o[2] = ac.x - bd.x;                      // U Z U^H: M01 = a c* - b d*
  o[5] = -(ac.y - bd.y);
  o[8] = 0.5 * ((cabs2(u[0]) - cabs2(u[1])) - (cabs2(u[2]) - cabs2(u[3])));
}

// Rotations of every site and layer, one CTA per state. A layer before the site's last CX with
// an angle that is not finite fails the state (as the SVD chain's nonfinite check does); such
// an angle in the last layer only makes the values NaN.
template <bool REAL>
__global__ void __launch_bounds__(256)
ladder_coef_kernel(LadCoefParams p) {
  const int b = blockIdx.x, B = gridDim.x, tid = threadIdx.x;
  const double *th = p.theta + (size_t)b * p.P;
  if (p.theta_keep != nullptr)
    for (int i = tid; i < p.P; i += 256) p.theta_keep[(size_t)b * p.P + i] = th[i];
  constexpr int NC = REAL ? LAD_REAL_COEFS : LAD_COEFS;
  const double r2 = 0.70710678118654752440;
  const cplx had[4] = {cmake(r2, 0), cmake(r2, 0), cmake(r2, 0), cmake(-r2, 0)};
  int bad = 0;
  const int pad = LAD_MAX_LAYERS - p.layers;        // leading layers without a CX
  for (int it = tid; it < p.n * 5; it += 256) {
    const int s = it / 5, k = it % 5, kk = k - pad;
    cplx u[4] = {cmake(1, 0), cmake(0, 0), cmake(0, 0), cmake(1, 0)};
    if (kk >= 0) {
      if (kk == 0)
        for (int i = 0; i < 4; ++i) u[i] = p.prep[i];
      else if (p.hadamard)
        for (int i = 0; i < 4; ++i) u[i] = had[i];
      const int g0 = p.off[s * (p.layers + 1) + kk], g1 = p.off[s * (p.layers + 1) + kk + 1];
      for (int g = g0; g < g1; ++g) {
        const LadGate lg = p.gates[g];
        DevGate dg{};
        dg.mat = lg.mat; dg.rot = lg.rot; dg.param = lg.param; dg.angle = lg.angle;
        cplx m[4], t[4];
        one_site_matrix(dg, p.mats, th, m);
        mul2(m, u, t);
        for (int i = 0; i < 4; ++i) u[i] = t[i];
      }
      if (k < 4 && p.hadamard) {
        cplx t[4];
        mul2(had, u, t);
        for (int i = 0; i < 4; ++i) u[i] = t[i];
      }
    }
    double o[9];
    bloch(u, o);
    double sum = 0.0;
    for (int i = 0; i < 9; ++i) sum += o[i];
    if (!isfinite(sum)) bad |= (k < 4) ? 1 : 2;
    double *c = p.coef + (size_t)s * NC * B + b;
    if (REAL) {
      if (k == 0) {
        c[0] = o[2];
        c[(size_t)B] = o[8];
      } else {
        double *d = c + (size_t)(2 + 5 * (k - 1)) * B;
        d[0] = o[0]; d[(size_t)B] = o[2]; d[(size_t)2 * B] = o[6]; d[(size_t)3 * B] = o[8]; d[(size_t)4 * B] = o[4];
      }
    } else {
      if (k == 0) {
        c[0] = o[2]; c[(size_t)B] = o[5]; c[(size_t)2 * B] = o[8];
      } else {
        double *d = c + (size_t)(3 + 9 * (k - 1)) * B;
        for (int i = 0; i < 9; ++i) d[(size_t)i * B] = o[i];
      }
    }
  }
  const int f1 = __syncthreads_or(bad & 1), f2 = __syncthreads_or(bad & 2);
  if (tid == 0) {
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const double ps = (f1 || f2) ? nan : 0.0;
    p.status[b] = f1 ? ST_NONFINITE : ST_OK;
    p.poison[b] = ps;
    p.leafval[(size_t)b * p.nleaf] = 1.0 + ps;
    p.leafval[(size_t)b * p.nleaf + 1] = ps;
  }
}

// ---- stages on a lane's 64 components x[d1 + 4 d2 + 16 d3] -------------------
// Digits 1-3 of component j hold an odd number of Y values.
__host__ __device__ constexpr int lad_ypar(int j) {
  return (((j & 3) == 2) ^ (((j >> 2) & 3) == 2) ^ (((j >> 4) & 3) == 2)) ? 1 : 0;
}

// S1: I' = I + nx X, X' = X + nx I, Y' = nz Y + ny Z, Z' = nz Z - ny Y.
// The transposed stage is the same with -ny.
template <bool REAL>
__device__ __forceinline__ void lad_s1(double (&x)[64], double nx, double ny, double nz) {
#pragma unroll
  for (int o = 0; o < 64; o += 4) {
    const double i = x[o], a = x[o + 1], y = x[o + 2], z = x[o + 3];
    x[o] = fma(nx, a, i);
    x[o + 1] = fma(nx, i, a);
    if (REAL) {
      x[o + 2] = nz * y;
      x[o + 3] = nz * z;
    } else {
      x[o + 2] = fma(ny, z, nz * y);
      x[o + 3] = fma(-ny, y, nz * z);
    }
  }
}

// Sk on the digit pair with strides SP (spin -> r_{k-1}) and SB (l_k -> spin). The
// transposed stage is the same with the entries odd in y (xy, yx, yz, zy) negated.
struct LadRot { double xx, xy, xz, yx, yy, yz, zx, zy, zz; };
template <bool REAL, int SP, int SB, int SO>
__device__ __forceinline__ void lad_sk(double (&x)[64], const LadRot &o) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int base = q * SO;
#define LX(P, Bt) x[base + (P) * SP + (Bt) * SB]
    {
      const double ii = LX(0, 0), ix = LX(0, 1), iy = LX(0, 2), iz = LX(0, 3);
      const double zi = LX(3, 0), zx = LX(3, 1), zy = LX(3, 2), zz = LX(3, 3);
      LX(0, 0) = fma(o.xz, zx, ii);
      LX(0, 1) = fma(o.xz, zi, ix);
      LX(3, 0) = fma(o.xz, ix, zi);
      LX(3, 1) = fma(o.xz, ii, zx);
      if (REAL) {
        LX(0, 2) = o.zz * zy;
        LX(0, 3) = o.zz * zz;
        LX(3, 2) = o.zz * iy;
        LX(3, 3) = o.zz * iz;
      } else {
        LX(0, 2) = fma(o.yz, zz, o.zz * zy);
        LX(0, 3) = fma(-o.yz, zy, o.zz * zz);
        LX(3, 2) = fma(o.yz, iz, o.zz * iy);
        LX(3, 3) = fma(-o.yz, iy, o.zz * iz);
      }
    }
    {
      const double xi = LX(1, 0), xx = LX(1, 1), xy = LX(1, 2), xz = LX(1, 3);
      const double yi = LX(2, 0), yx = LX(2, 1), yy = LX(2, 2), yz = LX(2, 3);
      if (REAL) {
        LX(1, 0) = o.xx * xx;
        LX(1, 1) = o.xx * xi;
        LX(1, 2) = fma(o.yy, yz, o.zx * xy);
        LX(1, 3) = fma(-o.yy, yy, o.zx * xz);
        LX(2, 0) = o.xx * yx;
        LX(2, 1) = o.xx * yi;
        LX(2, 2) = fma(-o.yy, xz, o.zx * yy);
        LX(2, 3) = fma(o.yy, xy, o.zx * yz);
      } else {
        LX(1, 0) = fma(o.xy, yx, o.xx * xx);
        LX(1, 1) = fma(o.xy, yi, o.xx * xi);
        LX(1, 2) = fma(o.yx, xz, fma(o.yy, yz, fma(o.zy, yy, o.zx * xy)));
        LX(1, 3) = fma(-o.yx, xy, fma(-o.yy, yy, fma(o.zy, yz, o.zx * xz)));
        LX(2, 0) = fma(-o.xy, xx, o.xx * yx);
        LX(2, 1) = fma(-o.xy, xi, o.xx * yi);
        LX(2, 2) = fma(o.yx, yz, fma(-o.yy, xz, fma(-o.zy, xy, o.zx * yy)));
        LX(2, 3) = fma(-o.yx, yy, fma(o.yy, xy, fma(-o.zy, xz, o.zx * yz)));
      }
    }
#undef LX
  }
}

// A site's rotations of one state (c points at component 0, stride B).
template <bool REAL>
__device__ __forceinline__ LadRot lad_rot(const double *__restrict__ c, int B, int k, double ysign) {
  LadRot o;
  if (REAL) {
    const double *d = c + (size_t)(2 + 5 * k) * B;
    o.xx = d[0]; o.xz = d[B]; o.zx = d[2 * B]; o.zz = d[3 * B]; o.yy = d[4 * B];
    o.xy = o.yx = o.yz = o.zy = 0.0;
  } else {
    const double *d = c + (size_t)(3 + 9 * k) * B;
    o.xx = d[0]; o.xy = ysign * d[B]; o.xz = d[2 * B];
    o.yx = ysign * d[3 * B]; o.yy = d[4 * B]; o.yz = ysign * d[5 * B];
    o.zx = d[6 * B]; o.zy = ysign * d[7 * B]; o.zz = d[8 * B];
  }
  return o;
}

// Lane q's rows of S4: what it keeps (ki, kz, kx, ky) and sends to lane q ^ 1 (sz, sx, sy); see
// lad_s4_*. Lanes I and X keep the identity part and send x; lanes Y and Z keep z and send -+ y.
struct LadS4 { double ki, kz, kx, ky, sz, sx, sy; };
template <bool REAL>
__device__ __forceinline__ LadS4 lad_s4_rows(const LadRot &o, int q) {
  LadS4 r;
  const bool yz = q >= 2;
  const double sg = q == 2 ? -1.0 : 1.0;
  r.ki = yz ? 0.0 : 1.0;
  r.kz = yz ? o.zz : 0.0;
  r.kx = yz ? o.zx : 0.0;
  r.ky = (!REAL && yz) ? o.zy : 0.0;
  r.sz = yz ? (REAL ? 0.0 : sg * o.yz) : o.xz;
  r.sx = yz ? (REAL ? 0.0 : sg * o.yx) : o.xx;
  r.sy = yz ? sg * o.yy : (REAL ? 0.0 : o.xy);
  return r;
}

constexpr unsigned LAD_FULL = 0xffffffffu;

// S4: digit 3 (registers) spin -> r_3, digit 4 (lanes) l_4 -> spin. exchange false: lanes X
// and Y hold zeros and only lanes I and Z are wanted (a run of identity codes).
template <bool REAL>
__device__ __forceinline__ void lad_s4(double (&x)[64], const LadS4 &r, bool exchange) {
#pragma unroll
  for (int o = 0; o < 16; ++o) {
    const double vi = x[o], vx = x[o + 16], vy = x[o + 32], vz = x[o + 48];
    x[o] = fma(r.ki, vi, r.kz * vz);
    x[o + 48] = fma(r.ki, vz, r.kz * vi);
    x[o + 16] = REAL ? r.kx * vx : fma(r.ky, vy, r.kx * vx);
    x[o + 32] = REAL ? r.kx * vy : fma(-r.ky, vx, r.kx * vy);
    if (exchange) {
      x[o] += __shfl_xor_sync(LAD_FULL, r.sz * vz, 1);
      x[o + 48] += __shfl_xor_sync(LAD_FULL, r.sz * vi, 1);
      x[o + 16] += __shfl_xor_sync(LAD_FULL, fma(r.sy, vy, r.sx * vx), 1);
      x[o + 32] += __shfl_xor_sync(LAD_FULL, fma(-r.sy, vx, r.sx * vy), 1);
    }
  }
}
// The transposed S4. exchange false: only lanes I and Z of the result are wanted and
// lanes X and Y hold zeros.
template <bool REAL>
__device__ __forceinline__ void lad_s4_t(double (&x)[64], const LadS4 &r, bool exchange) {
#pragma unroll
  for (int o = 0; o < 16; ++o) {
    const double vi = x[o], vx = x[o + 16], vy = x[o + 32], vz = x[o + 48];
    x[o] = fma(r.ki, vi, r.kz * vz);
    x[o + 48] = fma(r.ki, vz, r.kz * vi);
    x[o + 16] = REAL ? r.kx * vx : fma(-r.ky, vy, r.kx * vx);
    x[o + 32] = REAL ? r.kx * vy : fma(r.ky, vx, r.kx * vy);
    if (exchange) {
      const double wi = __shfl_xor_sync(LAD_FULL, vi, 1), wx = __shfl_xor_sync(LAD_FULL, vx, 1);
      const double wy = __shfl_xor_sync(LAD_FULL, vy, 1), wz = __shfl_xor_sync(LAD_FULL, vz, 1);
      x[o] = fma(r.sz, wz, x[o]);
      x[o + 48] = fma(r.sz, wi, x[o + 48]);
      x[o + 16] = fma(r.sx, wx, fma(-r.sy, wy, x[o + 16]));
      x[o + 32] = fma(r.sy, wx, fma(r.sx, wy, x[o + 32]));
    }
  }
}

// SF and its transpose (tsign -1): value <- u value + v value of lane q ^ 3.
struct LadSF { double u, v; };
template <bool REAL>
__device__ __forceinline__ LadSF lad_sf_row(const double *__restrict__ c, int B, int q, int code, double tsign) {
  LadSF r;
  const bool iz = q == 0 || q == 3;
  if (code == 0) {
    r.u = iz ? 1.0 : 0.0;
    r.v = 0.0;
    return r;
  }
  double a, bb, cc;                       // row of W for this Pauli: x, y, z
  if (REAL) {
    const double *d = c + (size_t)17 * B;
    a = code == 1 ? d[0] : code == 3 ? d[2 * B] : 0.0;
    cc = code == 1 ? d[B] : code == 3 ? d[3 * B] : 0.0;
    bb = code == 2 ? d[4 * B] : 0.0;
  } else {
    const double *d = c + (size_t)(30 + 3 * (code - 1)) * B;
    a = d[0]; bb = d[B]; cc = d[2 * B];
  }
  r.u = iz ? 0.0 : a;
  r.v = iz ? cc : (q == 1 ? tsign * bb : -tsign * bb);
  return r;
}
__device__ __forceinline__ void lad_sf(double (&x)[64], const LadSF &r) {
#pragma unroll
  for (int j = 0; j < 64; ++j) {
    const double w = __shfl_xor_sync(LAD_FULL, x[j], 3);
    x[j] = fma(r.u, x[j], r.v * w);
  }
}

// One path of trie nodes: the environment of start (a slot, or the chain's boundary) carried
// over len sites from site (up for prefix paths, down for suffix paths). Step bytes:
// bits 0-1 the Pauli code, bit 2 store the result in the path's next slot, bit 3 (suffix) the
// lanes X and Y of the stored result are wanted.
struct LadPath {
  int32_t start;     // slot, or -1: boundary
  int32_t site, len;
  int32_t code;      // offset of the step bytes
  int32_t slot;      // first stored slot
  int32_t flags;     // bit 0 odd Y count at the start, bit 1 suffix path, bit 2 lanes X, Y of the start
                     // are set, bit 3 store the boundary itself first
};

struct LadPathParams {
  const LadPath *paths;
  const uint8_t *codes;
  const double *coef;
  double *envp, *envs;   // prefix / suffix slots [slot][256][B]
  int npre, npaths;      // paths 0 .. npre - 1 prefix, npre .. npaths - 1 suffix
  int B;
};

template <bool REAL>
__device__ __forceinline__ void lad_store(double *__restrict__ dst, int B, const double (&x)[64], int par) {
#pragma unroll
  for (int j = 0; j < 64; ++j)
    if (!REAL || lad_ypar(j) == par) dst[(size_t)j * B] = x[j];
}
template <bool REAL>
__device__ __forceinline__ void lad_load(const double *__restrict__ src, int B, double (&x)[64], int par, bool set) {
#pragma unroll
  for (int j = 0; j < 64; ++j) x[j] = (set && (!REAL || lad_ypar(j) == par)) ? src[(size_t)j * B] : 0.0;
}

constexpr int LAD_THREADS = 128;

template <bool REAL>
__global__ void __launch_bounds__(LAD_THREADS, 2)
ladder_path_kernel(LadPathParams p) {
  constexpr int NC = REAL ? LAD_REAL_COEFS : LAD_COEFS;
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int B = p.B;
  // quads: prefix paths x states, padded to a whole warp, then suffix paths x states
  const long long quad = ((long long)blockIdx.x * LAD_THREADS + threadIdx.x) >> 2;
  const long long npre_q = (long long)p.npre * B, pre_pad = (npre_q + 7) & ~7LL;
  const bool suffix = quad >= pre_pad;                       // uniform over the warp
  const long long idx = suffix ? quad - pre_pad + npre_q : quad;
  const bool live = suffix ? idx < (long long)p.npaths * B : quad < npre_q;
  LadPath path{};
  int b = 0;
  if (live) {
    path = p.paths[idx / B];
    b = (int)(idx % B);
  }
  double *env = (suffix ? p.envs : p.envp) + b;
  auto slot_ptr = [&](int slot) { return env + ((size_t)slot * 256 + q * 64) * B; };
  double x[64];
  int par = path.flags & 1;
  const int ylane = q == 2 ? 1 : 0;
  int slot = path.slot;
  if (path.start >= 0 && live) {
    lad_load<REAL>(slot_ptr(path.start), B, x, par ^ ylane, (path.flags & 4) || q == 0 || q == 3);
  } else {
    // boundary: prefix |0> in every digit (I = Z = 1), suffix all ones (I = X = 1)
    const int other = suffix ? 1 : 3;
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const bool in = ((j & 3) == 0 || (j & 3) == other) && (((j >> 2) & 3) == 0 || ((j >> 2) & 3) == other) &&
                      (((j >> 4) & 3) == 0 || ((j >> 4) & 3) == other) && (q == 0 || q == other);
      x[j] = in ? 1.0 : 0.0;
    }
    if (live && (path.flags & 8)) {
      lad_store<REAL>(slot_ptr(slot), B, x, par ^ ylane);
      ++slot;
    }
  }
  int longest = path.len;
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(LAD_FULL, longest, o));
  bool xy_in = path.start < 0 ? suffix : (path.flags & 4) != 0;   // lanes X, Y of x may be nonzero
  for (int t = 0; t < longest; ++t) {
    const bool on = t < path.len;
    const int site = on ? (suffix ? path.site - t : path.site + t) : path.site;
    const int step = on ? p.codes[path.code + t] : 0;
    const int code = step & 3;
    const double *c = p.coef + (size_t)site * NC * B + b;
    if (!suffix) {
      if (REAL) lad_s1<REAL>(x, c[0], 0.0, c[B]);
      else lad_s1<REAL>(x, c[0], c[B], c[2 * (size_t)B]);
      lad_sk<REAL, 1, 4, 16>(x, lad_rot<REAL>(c, B, 0, 1.0));
      lad_sk<REAL, 4, 16, 1>(x, lad_rot<REAL>(c, B, 1, 1.0));
      const LadRot o4 = lad_rot<REAL>(c, B, 2, 1.0);
      LadS4 r4 = lad_s4_rows<REAL>(o4, q);
      const bool any = __any_sync(LAD_FULL, on && (code != 0 || xy_in));
      if (any) {
        lad_s4<REAL>(x, r4, true);
        if (__any_sync(LAD_FULL, on && code != 0)) {
          lad_sf(x, lad_sf_row<REAL>(c, B, q, code, 1.0));
        } else if (q == 1 || q == 2) {
#pragma unroll
          for (int j = 0; j < 64; ++j) x[j] = 0.0;
        }
      } else {
        if (q == 1 || q == 2) r4.ki = r4.kz = r4.kx = r4.ky = 0.0;
        lad_s4<REAL>(x, r4, false);
      }
      xy_in = code != 0;
      par ^= (code == 2);
      if (on && (step & 4)) {
        if (code != 0 || q == 0 || q == 3) lad_store<REAL>(slot_ptr(slot), B, x, par ^ ylane);
        ++slot;
      }
    } else {
      const int next = (on && t + 1 < path.len) ? (p.codes[path.code + t + 1] & 3) : 0;
      if (__any_sync(LAD_FULL, on && code != 0)) {
        lad_sf(x, lad_sf_row<REAL>(c, B, q, code, -1.0));
      } else if (q == 1 || q == 2) {
#pragma unroll
        for (int j = 0; j < 64; ++j) x[j] = 0.0;
      }
      const LadRot o4 = lad_rot<REAL>(c, B, 2, 1.0);
      LadS4 r4 = lad_s4_rows<REAL>(o4, q);
      const bool want = code != 0 || next != 0 || (step & 8);
      if (__any_sync(LAD_FULL, on && want)) {
        lad_s4_t<REAL>(x, r4, true);
      } else {
        if (q == 1 || q == 2) r4.ki = r4.kz = r4.kx = r4.ky = 0.0;
        lad_s4_t<REAL>(x, r4, false);
      }
      lad_sk<REAL, 4, 16, 1>(x, lad_rot<REAL>(c, B, 1, -1.0));
      lad_sk<REAL, 1, 4, 16>(x, lad_rot<REAL>(c, B, 0, -1.0));
      if (REAL) lad_s1<REAL>(x, c[0], 0.0, c[B]);
      else lad_s1<REAL>(x, c[0], -c[B], c[2 * (size_t)B]);
      par ^= (code == 2);
      if (on && (step & 4)) {
        if ((step & 8) || q == 0 || q == 3) lad_store<REAL>(slot_ptr(slot), B, x, par ^ ylane);
        ++slot;
      }
    }
  }
}

// Closures: value of a word = sum over components of its prefix and suffix environments, four
// lanes per (word, state) as the paths, every sum in the same order whatever the batch size.
struct LadPair {
  int32_t pslot, sslot, leaf;
  int32_t flags;    // bit 0 odd Y count of the prefix, bit 1 lanes X and Y count (prefix ends with X, Y or Z)
};

template <bool REAL>
__global__ void __launch_bounds__(256)
ladder_close_kernel(const double *__restrict__ envp, const double *__restrict__ envs, const LadPair *__restrict__ pairs,
                    int npairs, int B, const int32_t *__restrict__ status, const double *__restrict__ poison,
                    double *__restrict__ leafval, int nleaf) {
  const long long quad = ((long long)blockIdx.x * 256 + threadIdx.x) >> 2;
  const int q = threadIdx.x & 3;
  const bool live = quad < (long long)npairs * B;
  double v = 0.0;
  LadPair pr{};
  int b = 0;
  if (live) {
    pr = pairs[quad / B];
    b = (int)(quad % B);
    if ((pr.flags & 2) || q == 0 || q == 3) {
      const double *t = envp + ((size_t)pr.pslot * 256 + q * 64) * B + b;
      const double *w = envs + ((size_t)pr.sslot * 256 + q * 64) * B + b;
      const int par = (pr.flags & 1) ^ (q == 2 ? 1 : 0);
      if (!REAL) {
#pragma unroll 16
        for (int j = 0; j < 64; ++j) v = fma(t[(size_t)j * B], w[(size_t)j * B], v);
      } else if (par == 0) {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (lad_ypar(j) == 0) v = fma(t[(size_t)j * B], w[(size_t)j * B], v);
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (lad_ypar(j) == 1) v = fma(t[(size_t)j * B], w[(size_t)j * B], v);
      }
    }
  }
  v += __shfl_xor_sync(LAD_FULL, v, 1);
  v += __shfl_xor_sync(LAD_FULL, v, 2);
  if (live && q == 0) leafval[(size_t)b * nleaf + pr.leaf] = status[b] == 0 ? v + poison[b] : 0.0;
}

}  // namespace vqemps
