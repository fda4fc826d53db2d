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
// environments that several paths or a closure need. Those lie in global memory in 16-byte pairs of
// components (see lad_at): eight states side by side where the batch has them, so that a warp's access is
// full 128-byte lines, else one block per state.
#pragma once
#include "common.cuh"
#include "evolve.cuh"

namespace vqemps {

// Order of the digits' values (and of a quad's lanes): I 0, X 1, Y 2, Z 3.
constexpr int LAD_REAL_COEFS = 22;   // nx nz | k = 2, 3, 4: xx xz zx zz yy | W: xx xz zx zz yy
constexpr int LAD_COEFS = 40;        // n | k = 2, 3, 4: O row-major | W row-major | unused
constexpr int LAD_MAX_LAYERS = 4;

struct LadGate {   // a one-site gate of a layer: fixed matrix or rotation
  int32_t mat, rot, param;
  int32_t slot;            // index of its angle derivative, -1 without a parameter
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
  double *coef;            // [n][B][ncoef]: a state's row of a site is one run of 16-byte pieces
  int32_t *status;         // B
  double *poison;          // B: 0, or NaN when an angle is not finite
  double *leafval;         // B x nleaf: leaf 0 the norm, leaf 1 zero
  int nleaf;
  double *consts;          // LAD_CONSTS environments: the prefix and the suffix boundary, zero (or null)
};
constexpr int LAD_CONSTS = 3;

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

// Bloch matrices of a gate, of |0> -> initial state and of H. Rotations take the sine and cosine of the whole angle
// and the others (H, X, Y, Z, S, S^H and the preparations) their exact entries of 0 and +-1: formed from the 2 x 2 matrix's
// half angles, every entry would carry twice the rounding, and H, at every layer of some circuits, a bias of its own
// (a gradient of 40 qubits and 5,000 words against sums in 80 bits: 2.5e-15 of its norm that way, 3.4e-16 this way).
__device__ __forceinline__ void bloch_exact(const cplx *u, double *o) {
  bloch(u, o);
  for (int i = 0; i < 9; ++i) o[i] = rint(o[i]);
}
__device__ __forceinline__ void bloch_gate(const LadGate &g, const cplx *mats, const double *theta, double *o) {
  if (g.mat >= 0) {
    bloch_exact(mats + g.mat, o);
    return;
  }
  double s, c;
  sincos(g.param >= 0 ? theta[g.param] * g.angle : g.angle, &s, &c);
  const bool x = g.rot == ROT_X, y = g.rot == ROT_Y, z = !x && !y;
  o[0] = x ? 1.0 : c; o[1] = z ? -s : 0.0; o[2] = y ? s : 0.0;
  o[3] = z ? s : 0.0; o[4] = y ? 1.0 : c; o[5] = x ? -s : 0.0;
  o[6] = y ? -s : 0.0; o[7] = x ? s : 0.0; o[8] = z ? 1.0 : c;
}
__device__ __forceinline__ void bloch_hadamard(double *o) {
  for (int i = 0; i < 9; ++i) o[i] = 0.0;
  o[2] = o[6] = 1.0;
  o[4] = -1.0;
}
__device__ __forceinline__ void bloch_left(const double *o, double *m) {    // m <- o m
  double t[9];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) t[3 * r + c] = o[3 * r] * m[c] + o[3 * r + 1] * m[3 + c] + o[3 * r + 2] * m[6 + c];
  for (int i = 0; i < 9; ++i) m[i] = t[i];
}

// ---- a quad's components ------------------------------------------------------
// Lane q of a quad holds the components with digit 4 = q.
//
// Complex amplitudes: x[d1 + 4 d2 + 16 d3], all 64.
//
// Real amplitudes: only components of one Y parity are nonzero, so the lane's class c (parity of
// Y among digits 1-3: the word's parity so far, the other one on lane Y) selects 36 (c = 0) or 28
// (c = 1) of the 64. They are grouped by g = d1 + 4 d2: a group whose own Y parity equals c has
// d3 in {I, X, Z}, the others only d3 = Y. x[g] holds the group's X or Y component, x[16 + 2 m] and
// x[17 + 2 m] the I and Z components of the m-th group of parity c (10 or 6 of them; the rest of the
// 36 slots is zero). With these slots S4 and SF, which mix lanes of different classes, are the same
// instructions for every lane; only S1-S3 are written per class.
constexpr int LAD_XR = 36, LAD_XC = 64;
template <bool REAL> __host__ __device__ constexpr int lad_lane_comps() { return REAL ? LAD_XR : LAD_XC; }

template <int I> struct LadInt { static constexpr int v = I; };
template <int N, typename F>
__device__ __forceinline__ void lad_for(F &&f) {
  if constexpr (N > 0) {
    lad_for<N - 1>(f);
    f(LadInt<N - 1>{});
  }
}
__host__ __device__ constexpr int lad_gpar(int g) { return ((g & 3) == 2) ^ ((g >> 2) == 2) ? 1 : 0; }
__host__ __device__ constexpr int lad_rank(int g, int par) {   // groups of that parity before g
  int m = 0;
  for (int i = 0; i < g; ++i) m += lad_gpar(i) == par;
  return m;
}
// slot of component (d1, d2, d3) in class c (which must contain it)
template <int C, int D1, int D2, int D3>
__device__ constexpr int lad_slot() {
  constexpr int g = D1 + 4 * D2;
  return (D3 == 1 || D3 == 2) ? g : 16 + 2 * lad_rank(g, C) + (D3 == 3 ? 1 : 0);
}

// Environments in memory, offsets between a lane's pairs known to the compiler whatever the batch size:
//   W = 8: [slot][tile of 8 states][digit 4][pair][state][2], a warp's access to a digit is one 128-byte line;
//   W = 1: [slot][state][pair][digit 4: I Z X Y][2], a quad's access is 64 contiguous bytes, and steps that
//          keep only I and Z still move whole sectors.
// Batches of a multiple of 8 take W = 8: others would straddle tiles (45 complex states 110 us with W = 1, 118 with
// W = 8). Against
// 8-byte accesses at a run-time stride: 40 qubits, 5,000 words, B = 256 769 -> 732 us.
constexpr int LAD_TILE = 8;
__host__ __device__ constexpr bool lad_tiled(int B) { return B > 0 && B % LAD_TILE == 0; }
// offset of state b's environment from its slot's start (slots are B x 4 N apart)
template <int W, int N>
__device__ __forceinline__ size_t lad_state(int b) {
  return W == 1 ? (size_t)b * (4 * N) : (size_t)(b / W) * (W * 4 * N) + 2 * (b % W);
}
// this lane's pairs of an environment (at lad_state), lad_stride pairs apart
template <int W, int N>
__device__ __forceinline__ const double2 *lad_at(const double *env, int role) {
  const int place = role == 0 ? 0 : (role == 3 ? 1 : role + 1);
  return reinterpret_cast<const double2 *>(env) + (W == 1 ? place : place * (N / 2) * W);
}
template <int W> __host__ __device__ constexpr int lad_stride() { return W == 1 ? 4 : W; }
// A lane's share of an environment; real environments of class 1 carry zeros in the slots they do not use.
template <int W, int N>
__device__ __forceinline__ void lad_get(double (&x)[N], const double *env, int role) {
  const double2 *src = lad_at<W, N>(env, role);
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const double2 v = src[lad_stride<W>() * i];
    x[2 * i] = v.x;
    x[2 * i + 1] = v.y;
  }
}
template <int W, int N>
__device__ __forceinline__ void lad_put(const double (&x)[N], double *env, int role) {
  double2 *dst = const_cast<double2 *>(lad_at<W, N>(env, role));
#pragma unroll
  for (int i = 0; i < N / 2; ++i) dst[lad_stride<W>() * i] = make_double2(x[2 * i], x[2 * i + 1]);
}
// boundary: prefix |0> in every digit (I = Z = 1), suffix all ones (I = X = 1)
template <bool REAL>
__device__ __forceinline__ void lad_boundary(double (&x)[lad_lane_comps<REAL>()], int role, bool suffix) {
  const int other = suffix ? 1 : 3;
  auto in = [&](int d) { return d == 0 || d == other; };
  lad_for<64>([&](auto J) {
    constexpr int j = decltype(J)::v, d1 = j & 3, d2 = (j >> 2) & 3, d3 = j >> 4;
    const double v = in(d1) && in(d2) && in(d3) && in(role) ? 1.0 : 0.0;
    if constexpr (!REAL) x[j] = v;
    else if constexpr (((d1 == 2) ^ (d2 == 2) ^ (d3 == 2)) == 0) x[lad_slot<0, d1, d2, d3>()] = v;
  });
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
  if (p.consts != nullptr && b == 0) {
    constexpr int NX = lad_lane_comps<REAL>();
    const bool tiled = lad_tiled(B);
    const size_t env = (size_t)(tiled ? LAD_TILE : 1) * (4 * NX);
    if (tid < 4 * LAD_CONSTS) {
      double x[NX];
      lad_boundary<REAL>(x, tid & 3, (tid >> 2) == 1);
      if (tid >= 8)
        for (double &v : x) v = 0.0;
      double *dst = p.consts + (tid >> 2) * env;
      if (tiled) lad_put<LAD_TILE>(x, dst, tid & 3);
      else lad_put<1>(x, dst, tid & 3);
    }
  }
  int bad = 0;
  const int pad = LAD_MAX_LAYERS - p.layers;        // leading layers without a CX
  for (int it = tid; it < p.n * 5; it += 256) {
    const int s = it / 5, k = it % 5, kk = k - pad;
    double o[9] = {1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0}, t[9];
    if (kk >= 0) {
      if (kk == 0) bloch_exact(p.prep, o);
      else if (p.hadamard) bloch_hadamard(o);
      const int g0 = p.off[s * (p.layers + 1) + kk], g1 = p.off[s * (p.layers + 1) + kk + 1];
      for (int g = g0; g < g1; ++g) {
        bloch_gate(p.gates[g], p.mats, th, t);
        bloch_left(t, o);
      }
      if (k < 4 && p.hadamard) {
        bloch_hadamard(t);
        bloch_left(t, o);
      }
    }
    double sum = 0.0;
    for (int i = 0; i < 9; ++i) sum += o[i];
    if (!isfinite(sum)) bad |= (k < 4) ? 1 : 2;
    double *c = p.coef + ((size_t)s * B + b) * NC;
    if (REAL) {
      if (k == 0) {
        c[0] = o[2];
        c[1] = o[8];
      } else {
        double *d = c + 2 + 5 * (k - 1);
        d[0] = o[0]; d[1] = o[2]; d[2] = o[6]; d[3] = o[8]; d[4] = o[4];
      }
    } else {
      if (k == 0) {
        c[0] = o[2]; c[1] = o[5]; c[2] = o[8];
        c[LAD_COEFS - 1] = 0.0;
      } else {
        double *d = c + 3 + 9 * (k - 1);
        for (int i = 0; i < 9; ++i) d[i] = o[i];
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

// Rotations of one site (a row of LadCoefParams::coef in shared memory).
struct LadRot { double xx, xy, xz, yx, yy, yz, zx, zy, zz; };
template <bool REAL>
__device__ __forceinline__ LadRot lad_rot(const double *c, int k, double ysign) {
  LadRot o;
  if constexpr (REAL) {
    const double *d = c + 2 + 5 * k;
    o.xx = d[0]; o.xz = d[1]; o.zx = d[2]; o.zz = d[3]; o.yy = d[4];
    o.xy = o.yx = o.yz = o.zy = 0.0;
  } else {
    const double *d = c + 3 + 9 * k;
    o.xx = d[0]; o.xy = ysign * d[1]; o.xz = d[2];
    o.yx = ysign * d[3]; o.yy = d[4]; o.yz = ysign * d[5];
    o.zx = d[6]; o.zy = ysign * d[7]; o.zz = d[8];
  }
  return o;
}

// ---- S1: I' = I + nx X, X' = X + nx I, Y' = nz Y + ny Z, Z' = nz Z - ny Y -----
// The transposed stage is the same with -ny.
template <int C>
__device__ __forceinline__ void lad_s1r(double (&x)[LAD_XR], double nx, double nz) {
  lad_for<16>([&](auto G) {
    constexpr int d2 = decltype(G)::v & 3, d3 = decltype(G)::v >> 2;
    if constexpr (((d2 == 2) ^ (d3 == 2)) == C) {
      constexpr int i = lad_slot<C, 0, d2, d3>(), a = lad_slot<C, 1, d2, d3>(), z = lad_slot<C, 3, d2, d3>();
      const double vi = x[i], va = x[a];
      x[i] = fma(nx, va, vi);
      x[a] = fma(nx, vi, va);
      x[z] *= nz;
    } else {
      x[lad_slot<C, 2, d2, d3>()] *= nz;
    }
  });
}
__device__ __forceinline__ void lad_s1c(double (&x)[LAD_XC], double nx, double ny, double nz) {
#pragma unroll
  for (int o = 0; o < 64; o += 4) {
    const double i = x[o], a = x[o + 1], y = x[o + 2], z = x[o + 3];
    x[o] = fma(nx, a, i);
    x[o + 1] = fma(nx, i, a);
    x[o + 2] = fma(ny, z, nz * y);
    x[o + 3] = fma(-ny, y, nz * z);
  }
}

// ---- Sk: digits (k - 1: spin -> r_{k-1}) and (k: l_k -> spin), k = 2 and 3 -----
// The transposed stage is the same with the entries odd in y (xy, yx, yz, zy) negated.
template <int C, int K>
__device__ __forceinline__ void lad_skr(double (&x)[LAD_XR], const LadRot &o) {
  lad_for<4>([&](auto Q) {
    constexpr int q = decltype(Q)::v;               // the digit that stands by: 3 (k = 2) or 1 (k = 3)
    constexpr int sub = C ^ (q == 2 ? 1 : 0);       // Y parity of the pair
#define LX(P, Bt) x[K == 2 ? lad_slot<C, P, Bt, q>() : lad_slot<C, q, P, Bt>()]
    if constexpr (sub == 0) {
      const double ii = LX(0, 0), ix = LX(0, 1), iz = LX(0, 3), zi = LX(3, 0), zx = LX(3, 1), zz = LX(3, 3);
      LX(0, 0) = fma(o.xz, zx, ii);
      LX(0, 1) = fma(o.xz, zi, ix);
      LX(0, 3) = o.zz * zz;
      LX(3, 0) = fma(o.xz, ix, zi);
      LX(3, 1) = fma(o.xz, ii, zx);
      LX(3, 3) = o.zz * iz;
      const double xi = LX(1, 0), xx = LX(1, 1), xz = LX(1, 3), yy = LX(2, 2);
      LX(1, 0) = o.xx * xx;
      LX(1, 1) = o.xx * xi;
      LX(1, 3) = fma(-o.yy, yy, o.zx * xz);
      LX(2, 2) = fma(-o.yy, xz, o.zx * yy);
    } else {
      const double iy = LX(0, 2), zy = LX(3, 2);
      LX(0, 2) = o.zz * zy;
      LX(3, 2) = o.zz * iy;
      const double xy = LX(1, 2), yi = LX(2, 0), yx = LX(2, 1), yz = LX(2, 3);
      LX(1, 2) = fma(o.yy, yz, o.zx * xy);
      LX(2, 0) = o.xx * yx;
      LX(2, 1) = o.xx * yi;
      LX(2, 3) = fma(o.yy, xy, o.zx * yz);
    }
#undef LX
  });
}
template <int SP, int SB, int SO>
__device__ __forceinline__ void lad_skc(double (&x)[LAD_XC], const LadRot &o) {
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
      LX(0, 2) = fma(o.yz, zz, o.zz * zy);
      LX(0, 3) = fma(-o.yz, zy, o.zz * zz);
      LX(3, 2) = fma(o.yz, iz, o.zz * iy);
      LX(3, 3) = fma(-o.yz, iy, o.zz * iz);
    }
    {
      const double xi = LX(1, 0), xx = LX(1, 1), xy = LX(1, 2), xz = LX(1, 3);
      const double yi = LX(2, 0), yx = LX(2, 1), yy = LX(2, 2), yz = LX(2, 3);
      LX(1, 0) = fma(o.xy, yx, o.xx * xx);
      LX(1, 1) = fma(o.xy, yi, o.xx * xi);
      LX(1, 2) = fma(o.yx, xz, fma(o.yy, yz, fma(o.zy, yy, o.zx * xy)));
      LX(1, 3) = fma(-o.yx, xy, fma(-o.yy, yy, fma(o.zy, yz, o.zx * xz)));
      LX(2, 0) = fma(-o.xy, xx, o.xx * yx);
      LX(2, 1) = fma(-o.xy, xi, o.xx * yi);
      LX(2, 2) = fma(o.yx, yz, fma(-o.yy, xz, fma(-o.zy, xy, o.zx * yy)));
      LX(2, 3) = fma(-o.yx, yy, fma(o.yy, xy, fma(-o.zy, xz, o.zx * yz)));
    }
#undef LX
  }
}

// ---- S4: digit 3 (registers) spin -> r_3, digit 4 (lanes) l_4 -> spin -----------
// Lanes I and X keep the identity part and send x, lanes Y and Z keep z and send -+ y, to lane
// q ^ 1: kept I = ki I + kz Z, Z = ki Z + kz I, X = kx X + ky Y, Y = kx Y - ky X; sent I = sz Z, Z = sz I,
// X = sx X + sy Y, Y = sx Y - sy X.
constexpr unsigned LAD_FULL = 0xffffffffu;
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
// Real amplitudes: SF and its transpose only scale and exchange whole lanes (W has no x-y or y-z
// entries), so a quad's lanes carry roles instead: role r holds the components with digit 4 = r,
// codes X and Z exchange the roles I and Z, code Y the roles X and Y, and the factor of the code
// (by the role before the exchange) joins the rows of S4. factor I: 1 on I and Z, else 0; X, Z: W_pz on
// I and Z, W_px on X and Y; Y: +-W_yy on X and Y.
__device__ __forceinline__ double lad_factor(const double *c, int code, int role, double tsign) {
  const double *w = c + 17;                          // xx xz zx zz yy
  const bool iz = role == 0 || role == 3;
  if (code == 0) return iz ? 1.0 : 0.0;
  if (code == 2) return iz ? 0.0 : (role == 2 ? tsign * w[4] : -tsign * w[4]);
  const int k = code == 1 ? 0 : 2;
  return iz ? w[k + 1] : w[k];
}
__device__ __forceinline__ int lad_role(int q, int swaps) {       // swaps: bit 0 I <-> Z, bit 1 X <-> Y
  return (q == 0 || q == 3) ? ((swaps & 1) ? 3 - q : q) : ((swaps & 2) ? 3 - q : q);
}

// A group's X or Y component goes to the partner's X or Y component of the same group (roles Y
// and Z are of different classes, where X and Y change places, as the rotation by yy asks). u, up: the
// code's factor of this lane's role and of its partner's. exchange false: roles X and Y hold zeros
// and only I and Z are wanted.
__device__ __forceinline__ void lad_s4r(double (&x)[LAD_XR], const LadS4 &r, int role, int cls, int src, double u,
                                        double up, bool exchange) {
  const double kx = u * r.kx, ki = u * r.ki, kz = u * r.kz;
  if (exchange) {
    const double s0 = role >= 2 ? -up * r.sy : up * r.sx, s1 = role >= 2 ? up * r.sy : up * r.sx;   // sender's X / Y
    const double ce = cls ? s1 : s0, co = cls ? s0 : s1, sz = up * r.sz;   // groups of even / odd Y parity
    lad_for<16>([&](auto G) {
      constexpr int g = decltype(G)::v;
      const double v = __shfl_sync(LAD_FULL, (lad_gpar(g) ? co : ce) * x[g], src);
      x[g] = fma(kx, x[g], v);
    });
#pragma unroll
    for (int m = 16; m < LAD_XR; m += 2) {
      const double vi = x[m], vz = x[m + 1];
      const double wi = __shfl_sync(LAD_FULL, sz * vz, src), wz = __shfl_sync(LAD_FULL, sz * vi, src);
      x[m] = fma(ki, vi, fma(kz, vz, wi));
      x[m + 1] = fma(ki, vz, fma(kz, vi, wz));
    }
  } else {
#pragma unroll
    for (int g = 0; g < 16; ++g) x[g] *= kx;
#pragma unroll
    for (int m = 16; m < LAD_XR; m += 2) {
      const double vi = x[m], vz = x[m + 1];
      x[m] = fma(ki, vi, kz * vz);
      x[m + 1] = fma(ki, vz, kz * vi);
    }
  }
}
// The transposed SF and S4 (roles already exchanged).
__device__ __forceinline__ void lad_s4r_t(double (&x)[LAD_XR], const LadS4 &r, int role, int cls, int src, double u,
                                          double up, bool exchange) {
  const double kx = u * r.kx, ki = u * r.ki, kz = u * r.kz;
  if (exchange) {
    const double s0 = role >= 2 ? -up * r.sy : up * r.sx, s1 = role >= 2 ? up * r.sy : up * r.sx;   // receiver's X / Y
    const double ce = cls ? s1 : s0, co = cls ? s0 : s1, sz = up * r.sz;
    lad_for<16>([&](auto G) {
      constexpr int g = decltype(G)::v;
      const double v = __shfl_sync(LAD_FULL, x[g], src);
      x[g] = fma(kx, x[g], (lad_gpar(g) ? co : ce) * v);
    });
#pragma unroll
    for (int m = 16; m < LAD_XR; m += 2) {
      const double vi = x[m], vz = x[m + 1];
      const double wi = __shfl_sync(LAD_FULL, vi, src), wz = __shfl_sync(LAD_FULL, vz, src);
      x[m] = fma(ki, vi, fma(kz, vz, sz * wz));
      x[m + 1] = fma(ki, vz, fma(kz, vi, sz * wi));
    }
  } else {
#pragma unroll
    for (int g = 0; g < 16; ++g) x[g] *= kx;
#pragma unroll
    for (int m = 16; m < LAD_XR; m += 2) {
      const double vi = x[m], vz = x[m + 1];
      x[m] = fma(ki, vi, kz * vz);
      x[m + 1] = fma(ki, vz, kz * vi);
    }
  }
}
__device__ __forceinline__ void lad_s4c(double (&x)[LAD_XC], const LadS4 &r, bool exchange) {
#pragma unroll
  for (int o = 0; o < 16; ++o) {
    const double vi = x[o], vx = x[o + 16], vy = x[o + 32], vz = x[o + 48];
    x[o] = fma(r.ki, vi, r.kz * vz);
    x[o + 48] = fma(r.ki, vz, r.kz * vi);
    x[o + 16] = fma(r.ky, vy, r.kx * vx);
    x[o + 32] = fma(-r.ky, vx, r.kx * vy);
    if (exchange) {
      x[o] += __shfl_xor_sync(LAD_FULL, r.sz * vz, 1);
      x[o + 48] += __shfl_xor_sync(LAD_FULL, r.sz * vi, 1);
      x[o + 16] += __shfl_xor_sync(LAD_FULL, fma(r.sy, vy, r.sx * vx), 1);
      x[o + 32] += __shfl_xor_sync(LAD_FULL, fma(-r.sy, vx, r.sx * vy), 1);
    }
  }
}
__device__ __forceinline__ void lad_s4c_t(double (&x)[LAD_XC], const LadS4 &r, bool exchange) {
#pragma unroll
  for (int o = 0; o < 16; ++o) {
    const double vi = x[o], vx = x[o + 16], vy = x[o + 32], vz = x[o + 48];
    x[o] = fma(r.ki, vi, r.kz * vz);
    x[o + 48] = fma(r.ki, vz, r.kz * vi);
    x[o + 16] = fma(-r.ky, vy, r.kx * vx);
    x[o + 32] = fma(r.ky, vx, r.kx * vy);
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

// ---- SF and its transpose (tsign -1): value <- u value + v value of lane q ^ 3 (complex amplitudes) --------
struct LadSF { double u, v; };
__device__ __forceinline__ LadSF lad_sf_row(const double *c, int q, int code, double tsign) {
  LadSF r;
  const bool iz = q == 0 || q == 3;
  if (code == 0) {
    r.u = iz ? 1.0 : 0.0;
    r.v = 0.0;
    return r;
  }
  const double *d = c + 30 + 3 * (code - 1);          // row of W for this Pauli, read whole by every lane
  const double x = d[0], y = d[1], z = d[2];
  r.u = iz ? 0.0 : x;
  r.v = iz ? z : (q == 1 ? tsign * y : -tsign * y);
  return r;
}
template <int N>
__device__ __forceinline__ void lad_sf(double (&x)[N], const LadSF &r) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const double w = __shfl_xor_sync(LAD_FULL, x[j], 3);
    x[j] = fma(r.u, x[j], r.v * w);
  }
}

// One task: a walk through a subtree of the prefix trie (sites upwards) or of the suffix trie
// (downwards), depth first. A step word moves the environment over one site:
//   bits 0-1 the Pauli code, bit 2 store the result in the task's next slot,
//   bit 3 (suffix) lanes X and Y of the result are wanted, bit 5 first load the task's next slot,
//   bit 6 odd Y count before the step, bit 7 lanes X, Y of the input are set, bits 16-31 the site.
// A walk that does not begin with a load begins at the chain's boundary. Slots of stores and loads
// are listed per task in the order of use; a task only loads slots that an earlier launch or the
// same task stored.
struct LadTask {
  int32_t step, nsteps, slot;
  int32_t flags;     // bit 1 suffix, bit 3 store the boundary first
};

struct LadPathParams {
  const LadTask *tasks;
  const uint32_t *steps;
  const int32_t *slots;
  const double *coef;
  double *envp, *envs;   // prefix / suffix environments (lad_at)
  int npre, ntasks;      // tasks 0 .. npre - 1 prefix, npre .. ntasks - 1 suffix
  int B;
};

constexpr int LAD_THREADS = 128;
constexpr int LAD_AHEAD = 3;     // steps whose rotations are in flight
__device__ __forceinline__ void lad_cp16(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// Bound: FP64 issue (an identity step of a real environment is 180 FP64 instructions for eight
// environments, another one about 360 and 72 shuffles) and, for small batches, the latency of one
// warp's step (1-2 us). Real environments take 72 registers, so four CTAs of four warps fit an SM;
// complex ones take 128 and two CTAs fit. Measured (B200), whole energy call, gate chain + 16 x 16
// transfer products -> this: 40 qubits, 5,000 words, B = 256: 5,504 -> 732 us (FP64 pipe 40 % busy, issue 53 %);
// B = 3: 1,082 -> 52 us; 96 qubits, 40,000 words, B = 2: 3,039 -> 128 us; complex, 27 qubits, 1,300 words,
// B = 45: 1,191 -> 103 us; error against 64-bit values 1e-13 -> 3e-15 (no SVD in between).
template <bool REAL, int W>
__global__ void __launch_bounds__(LAD_THREADS, REAL ? 4 : 2)
ladder_path_kernel(LadPathParams p) {
  constexpr int NC = REAL ? LAD_REAL_COEFS : LAD_COEFS;
  constexpr int NX = lad_lane_comps<REAL>();
  // rotations of each quad's site, three steps ahead: rows of 176 or 320 bytes, whose 8-byte reads
  // by the eight quads of a warp fall on distinct banks (real) or two to a bank (complex)
  __shared__ __align__(16) double rows[LAD_AHEAD + 1][LAD_THREADS / 4][NC];
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int B = p.B;
  // quads: prefix tasks x states, padded to a whole warp, then suffix tasks x states
  const long long quad = ((long long)blockIdx.x * LAD_THREADS + threadIdx.x) >> 2;
  const long long npre_q = (long long)p.npre * B, pre_pad = (npre_q + 7) & ~7LL;
  const bool suffix = quad >= pre_pad;                       // uniform over the warp
  const long long idx = suffix ? quad - pre_pad + npre_q : quad;
  const bool live = suffix ? idx < (long long)p.ntasks * B : quad < npre_q;
  LadTask task{};
  int b = 0;
  if (live) {
    task = p.tasks[idx / B];
    b = (int)(idx % B);
  }
  const uint32_t *steps = p.steps + task.step;
  const int32_t *slots = p.slots + task.slot;
  auto word = [&](int t) { return t < task.nsteps ? steps[t] : 0u; };
  auto stage = [&](int t, uint32_t w) {                      // rotations of step t, if there is one
    if (t < task.nsteps) {
      const double *src = p.coef + ((size_t)(w >> 16) * B + b) * NC;
      double *dst = rows[t % (LAD_AHEAD + 1)][threadIdx.x >> 2];
#pragma unroll
      for (int i = 0; i < NC / 2; i += 4)
        if (i + q < NC / 2) lad_cp16(dst + 2 * (i + q), src + 2 * (i + q));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  static_assert(LAD_AHEAD == 3, "the words of four steps are kept");
  uint32_t w0 = word(0), w1 = word(1), w2 = word(2), w3 = word(3);
  dependency_wait();                                         // the rotations, and earlier launches' environments
  stage(0, w0);
  stage(1, w1);
  stage(2, w2);
  double *env = (suffix ? p.envs : p.envp) + lad_state<W, NX>(b);
  const size_t slot_size = (size_t)B * (4 * NX);
  double x[NX];
  int swaps = 0;                                             // real: lanes' roles (lad_role)
  int slot = live ? *slots : 0;                              // the next one: read ahead, the lists end with a spare entry
  auto advance = [&] { slot = *++slots; };
  auto store = [&](int role, bool lanes_xy) {
    if (!lanes_xy && role != 0 && role != 3) return;
    lad_put<W>(x, env + slot * slot_size, role);
  };
  lad_boundary<REAL>(x, q, suffix);
  if (live && (task.flags & 8)) {
    store(q, suffix);
    advance();
  }
  int longest = task.nsteps;
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(LAD_FULL, longest, o));
  for (int t = 0; t < longest; ++t) {
    const bool on = t < task.nsteps;
    const uint32_t w = w0;
    w0 = w1;
    w1 = w2;
    w2 = w3;
    w3 = word(t + 4);
    const int code = w & 3;
    int par = (w >> 6) & 1;
    const bool xy = (w & 128) != 0;
    stage(t + 3, w2);
    if (w & 32) {
      swaps = 0;
      if (xy || q == 0 || q == 3) {
        lad_get<W>(x, env + slot * slot_size, q);
      } else {
#pragma unroll
        for (int j = 0; j < NX; ++j) x[j] = 0.0;
      }
      advance();
    }
    asm volatile("cp.async.wait_group 3;\n" ::);
    __syncwarp();
    const double *c = rows[t % (LAD_AHEAD + 1)][threadIdx.x >> 2];
    if constexpr (REAL) {
      if (suffix) {
        // the transposed SF: its factor by the role before the exchange of roles
        swaps ^= code == 0 ? 0 : (code == 2 ? 2 : 1);
        par ^= (code == 2);
        const int role = lad_role(q, swaps), cls = par ^ (role == 2);
        const int prole = role ^ 1;
        // factor of a lane whose role is now k: before the exchange it was 3 - k on the exchanged pair
        auto fac = [&](int k) {
          const bool iz = k == 0 || k == 3;
          return lad_factor(c, code, code == 0 ? k : ((code == 2) != iz ? 3 - k : k), -1.0);
        };
        const int pq = lad_role(prole, swaps);               // lad_role is its own inverse
        const bool next = (w0 & 3) != 0 && !(w0 & 32);
        const bool any = __any_sync(LAD_FULL, on && (code != 0 || next || (w & 8)));
        const LadS4 r4 = lad_s4_rows<true>(lad_rot<true>(c, 2, 1.0), role);
        const bool iz = role == 0 || role == 3;
        lad_s4r_t(x, r4, role, cls, (lane & ~3) | pq, fac(role), fac(prole), any);
        if (any || iz) {
          if (cls == 0) {
            lad_skr<0, 3>(x, lad_rot<true>(c, 1, 1.0));
            lad_skr<0, 2>(x, lad_rot<true>(c, 0, 1.0));
            lad_s1r<0>(x, c[0], c[1]);
          } else {
            lad_skr<1, 3>(x, lad_rot<true>(c, 1, 1.0));
            lad_skr<1, 2>(x, lad_rot<true>(c, 0, 1.0));
            lad_s1r<1>(x, c[0], c[1]);
          }
        }
        __syncwarp();
        if (on && (w & 4)) {
          store(role, (w & 8) != 0);
          advance();
        }
      } else {
        int role = lad_role(q, swaps);
        const int cls = par ^ (role == 2);
        const bool iz = role == 0 || role == 3;
        if (xy || iz) {
          if (cls == 0) {
            lad_s1r<0>(x, c[0], c[1]);
            lad_skr<0, 2>(x, lad_rot<true>(c, 0, 1.0));
            lad_skr<0, 3>(x, lad_rot<true>(c, 1, 1.0));
          } else {
            lad_s1r<1>(x, c[0], c[1]);
            lad_skr<1, 2>(x, lad_rot<true>(c, 0, 1.0));
            lad_skr<1, 3>(x, lad_rot<true>(c, 1, 1.0));
          }
        }
        __syncwarp();
        const LadS4 r4 = lad_s4_rows<true>(lad_rot<true>(c, 2, 1.0), role);
        const bool any = __any_sync(LAD_FULL, on && (code != 0 || xy));
        const int pq = lad_role(role ^ 1, swaps);
        lad_s4r(x, r4, role, cls, (lane & ~3) | pq, lad_factor(c, code, role, 1.0), lad_factor(c, code, role ^ 1, 1.0), any);
        swaps ^= code == 0 ? 0 : (code == 2 ? 2 : 1);
        par ^= (code == 2);
        role = lad_role(q, swaps);
        if (on && (w & 4)) {
          store(role, code != 0);
          advance();
        }
      }
    } else {
      const bool izlane = q == 0 || q == 3;
      if (suffix) {
        if (__any_sync(LAD_FULL, on && code != 0)) {
          lad_sf(x, lad_sf_row(c, q, code, -1.0));
        } else if (!izlane) {
#pragma unroll
          for (int j = 0; j < NX; ++j) x[j] = 0.0;
        }
        LadS4 r4 = lad_s4_rows<false>(lad_rot<false>(c, 2, 1.0), q);
        const bool next = (w0 & 3) != 0 && !(w0 & 32);
        const bool any = __any_sync(LAD_FULL, on && (code != 0 || next || (w & 8)));
        if (!any && !izlane) r4.ki = r4.kz = r4.kx = r4.ky = 0.0;
        lad_s4c_t(x, r4, any);
        lad_skc<4, 16, 1>(x, lad_rot<false>(c, 1, -1.0));
        lad_skc<1, 4, 16>(x, lad_rot<false>(c, 0, -1.0));
        lad_s1c(x, c[0], -c[1], c[2]);
        if (on && (w & 4)) {
          store(q, (w & 8) != 0);
          advance();
        }
      } else {
        lad_s1c(x, c[0], c[1], c[2]);
        lad_skc<1, 4, 16>(x, lad_rot<false>(c, 0, 1.0));
        lad_skc<4, 16, 1>(x, lad_rot<false>(c, 1, 1.0));
        LadS4 r4 = lad_s4_rows<false>(lad_rot<false>(c, 2, 1.0), q);
        const bool any = __any_sync(LAD_FULL, on && (code != 0 || xy));
        if (!any && !izlane) r4.ki = r4.kz = r4.kx = r4.ky = 0.0;
        lad_s4c(x, r4, any);
        if (__any_sync(LAD_FULL, on && code != 0)) {
          lad_sf(x, lad_sf_row(c, q, code, 1.0));
        } else if (!izlane) {
#pragma unroll
          for (int j = 0; j < NX; ++j) x[j] = 0.0;
        }
        if (on && (w & 4)) {
          store(q, code != 0);
          advance();
        }
      }
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Closures: value of a word = sum over components of its prefix and suffix environments, four
// lanes per (word, state) as the paths, every sum in the same order whatever the batch size.
struct LadPair {
  int32_t pslot, sslot, leaf;
  int32_t flags;    // bit 1 lanes X and Y count (prefix ends with X, Y or Z)
};

template <bool REAL, int W>
__global__ void __launch_bounds__(256)
ladder_close_kernel(const double *__restrict__ envp, const double *__restrict__ envs, const LadPair *__restrict__ pairs,
                    int npairs, int B, const int32_t *__restrict__ status, const double *__restrict__ poison,
                    double *__restrict__ leafval, int nleaf) {
  constexpr int NX = lad_lane_comps<REAL>();
  const long long quad = ((long long)blockIdx.x * 256 + threadIdx.x) >> 2;
  const int q = threadIdx.x & 3;
  const bool live = quad < (long long)npairs * B;
  double v = 0.0;
  LadPair pr{};
  int b = 0;
  if (live) {
    pr = pairs[quad / B];
    b = (int)(quad % B);
  }
  dependency_wait();
  if (live) {
    if ((pr.flags & 2) || q == 0 || q == 3) {
      const size_t slot_size = (size_t)B * (4 * NX), at = lad_state<W, NX>(b);
      const double2 *t = lad_at<W, NX>(envp + at + pr.pslot * slot_size, q);
      const double2 *w = lad_at<W, NX>(envs + at + pr.sslot * slot_size, q);
#pragma unroll(REAL ? 18 : 16)
      for (int i = 0; i < NX / 2; ++i) {
        const double2 a = t[lad_stride<W>() * i], c = w[lad_stride<W>() * i];
        v = fma(a.x, c.x, v);
        v = fma(a.y, c.y, v);
      }
    }
  }
  v += __shfl_xor_sync(LAD_FULL, v, 1);
  v += __shfl_xor_sync(LAD_FULL, v, 2);
  if (live && q == 0) leafval[(size_t)b * nleaf + pr.leaf] = status[b] == 0 ? v + poison[b] : 0.0;
}

}  // namespace vqemps
