// Gradient of the energy of a ladder circuit (see ladder.cuh for the stages).
//
// Reference: test/tools/reverse_mps.py:84-99 (ReverseMPS.value_gradient), torch autograd
// through the same exact matrix product state.
//
// Forward: the paths of every task, each step's environment kept (ladder_path_kernel). Backward: a
// prefix task is walked in reverse with the cotangent of its environment, which lives in the dual
// components and moves by the transposed stages; a suffix task, whose environments are dual, with
// a cotangent in the primal components that moves by the stages themselves. In both, a step
// has a primal tensor t on its left and a dual one w on its right, and the derivative of sum w S(t) by
// the entries of each stage's rotation is a sum of products of the stage's input (from t) and the
// pulled-back w at its output: the kernel forms the chain that comes from memory first, keeps its inner
// members in shared memory and then takes the carried tensor through the stages, adding the
// products on the way. Per step and state 16 (33) derivatives remain; they are summed over the
// steps of a site in a fixed order and contracted with the gates' own derivatives.
#pragma once
#include "ladder.cuh"

namespace vqemps {

struct LadBack {
  int32_t in;        // slot of the step's input environment, -1: the boundary
  int32_t cot_add;   // cotangent collected from the step's other children, -1: none
  int32_t cot_out;   // -1: goes on to the previous step, -2: ends at the boundary, else 2 x cotangent + (1: first)
  int32_t close;     // first of the words that close here (up to the next step's)
};

struct LadClose {
  int32_t slot;      // the word's environment in the other half
  int32_t flags;     // bit 1: its lanes X and Y count, bit 2: a sum made ahead, slot counts those
  double coef;
};
struct LadGather {   // a sum of closures made ahead; its slot is its place in the list
  int32_t first, count;
  int32_t half;      // of the step: 0 takes suffix environments, 1 prefix ones
};
constexpr int LAD_CLOSE_MOST = 2, LAD_CLOSE_CHUNK = 16;

constexpr int LAD_GR = 16;   // nx nz | k = 2, 3, 4: xx xz zx zz | W: x z of the step's code
constexpr int LAD_GC = 36;   // nx ny nz | k = 2: O row-major || k = 3 | 3 unused || k = 4 | W: x y z of the step's code
constexpr int LAD_GROUP = 12;   // complex derivatives are summed and stored twelve at a time, so that few are live

struct LadBackParams {
  const LadTask *tasks;
  const uint32_t *steps;
  const LadBack *back;
  const LadClose *closers;
  const double *coef;
  const double *envp, *envs;
  double *gathered;          // sums of closures made ahead, laid out as the environments
  const LadGather *gathers;
  const double *consts;      // boundaries and zero (LadCoefParams)
  double *cotp, *cots;       // cotangents, laid out as the environments
  double *part;              // [step][LAD_GR or LAD_GC][B]
  int npre, ntasks, B;
};

// Sums of products of a stage's output cotangent y and its input v (real amplitudes).
template <int C, class V>
__device__ __forceinline__ void lad_g1r(const double (&y)[LAD_XR], V v, double &nx, double &nz) {
  lad_for<16>([&](auto G) {
    constexpr int d2 = decltype(G)::v & 3, d3 = decltype(G)::v >> 2;
    if constexpr (((d2 == 2) ^ (d3 == 2)) == C) {
      constexpr int i = lad_slot<C, 0, d2, d3>(), a = lad_slot<C, 1, d2, d3>(), z = lad_slot<C, 3, d2, d3>();
      nx = fma(y[i], v(a), fma(y[a], v(i), nx));
      nz = fma(y[z], v(z), nz);
    } else {
      constexpr int k = lad_slot<C, 2, d2, d3>();
      nz = fma(y[k], v(k), nz);
    }
  });
}
template <int C, int K, class V>
__device__ __forceinline__ void lad_gkr(const double (&y)[LAD_XR], V v, double &xx, double &xz, double &zx, double &zz) {
  lad_for<4>([&](auto Q) {
    constexpr int q = decltype(Q)::v;
    constexpr int sub = C ^ (q == 2 ? 1 : 0);
#define LS(P, Bt) (K == 2 ? lad_slot<C, P, Bt, q>() : lad_slot<C, q, P, Bt>())
    if constexpr (sub == 0) {
      const double vii = v(LS(0, 0)), vix = v(LS(0, 1)), vzi = v(LS(3, 0)), vzx = v(LS(3, 1));
      xz = fma(y[LS(0, 0)], vzx, fma(y[LS(0, 1)], vzi, fma(y[LS(3, 0)], vix, fma(y[LS(3, 1)], vii, xz))));
      zz = fma(y[LS(0, 3)], v(LS(3, 3)), fma(y[LS(3, 3)], v(LS(0, 3)), zz));
      xx = fma(y[LS(1, 0)], v(LS(1, 1)), fma(y[LS(1, 1)], v(LS(1, 0)), xx));
      zx = fma(y[LS(1, 3)], v(LS(1, 3)), fma(y[LS(2, 2)], v(LS(2, 2)), zx));
    } else {
      zz = fma(y[LS(0, 2)], v(LS(3, 2)), fma(y[LS(3, 2)], v(LS(0, 2)), zz));
      xx = fma(y[LS(2, 0)], v(LS(2, 1)), fma(y[LS(2, 1)], v(LS(2, 0)), xx));
      zx = fma(y[LS(1, 2)], v(LS(1, 2)), fma(y[LS(2, 3)], v(LS(2, 3)), zx));
    }
#undef LS
  });
}

// The complex stages' sums; w(j) the output cotangent, v(j) the input.
template <class W, class V>
__device__ __forceinline__ void lad_g1c(W w, V v, double *g) {
#pragma unroll
  for (int o = 0; o < 64; o += 4) {
    g[0] = fma(w(o), v(o + 1), fma(w(o + 1), v(o), g[0]));
    g[1] = fma(w(o + 2), v(o + 3), fma(-w(o + 3), v(o + 2), g[1]));
    g[2] = fma(w(o + 2), v(o + 2), fma(w(o + 3), v(o + 3), g[2]));
  }
}
template <int SP, int SB, int SO, class W, class V>
__device__ __forceinline__ void lad_gkc(W w, V v, double *g) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int base = q * SO;
#define LV(P, Bt) v(base + (P) * SP + (Bt) * SB)
#define LW(P, Bt) w(base + (P) * SP + (Bt) * SB)
#pragma unroll
    for (int a = 0; a < 4; a += 3) {                 // spin copies I and Z: input z = Z resp. I
      const int z = 3 - a;
      const double wi = LW(a, 0), wx = LW(a, 1), wy = LW(a, 2), wz = LW(a, 3);
      const double vi = LV(z, 0), vx = LV(z, 1), vy = LV(z, 2), vz = LV(z, 3);
      g[2] = fma(wi, vx, fma(wx, vi, g[2]));
      g[5] = fma(wy, vz, fma(-wz, vy, g[5]));
      g[8] = fma(wy, vy, fma(wz, vz, g[8]));
    }
    const double xi = LV(1, 0), xx = LV(1, 1), xy = LV(1, 2), xz = LV(1, 3);
    const double yi = LV(2, 0), yx = LV(2, 1), yy = LV(2, 2), yz = LV(2, 3);
    {
      const double wi = LW(1, 0), wx = LW(1, 1), wy = LW(1, 2), wz = LW(1, 3);
      g[0] = fma(wi, xx, fma(wx, xi, g[0]));
      g[1] = fma(wi, yx, fma(wx, yi, g[1]));
      g[3] = fma(wy, xz, fma(-wz, xy, g[3]));
      g[4] = fma(wy, yz, fma(-wz, yy, g[4]));
      g[6] = fma(wy, xy, fma(wz, xz, g[6]));
      g[7] = fma(wy, yy, fma(wz, yz, g[7]));
    }
    {                                                // the copy Y: x = Y, y = -X
      const double wi = LW(2, 0), wx = LW(2, 1), wy = LW(2, 2), wz = LW(2, 3);
      g[0] = fma(wi, yx, fma(wx, yi, g[0]));
      g[1] = fma(-wi, xx, fma(-wx, xi, g[1]));
      g[3] = fma(wy, yz, fma(-wz, yy, g[3]));
      g[4] = fma(-wy, xz, fma(wz, xy, g[4]));
      g[6] = fma(wy, yy, fma(wz, yz, g[6]));
      g[7] = fma(-wy, xy, fma(-wz, xz, g[7]));
    }
#undef LV
#undef LW
  }
}

// Sum of N values (a multiple of four) over a quad; lane q keeps values N / 4 * q' .. with
// q' = 2 (q & 1) + (q >> 1), in out[0 .. N / 4).
template <int N>
__device__ __forceinline__ void lad_quad_sums(const double *g, int q, double *out) {
  double h[N / 2];
  const bool up = q & 1, up2 = q >> 1;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const double keep = up ? g[N / 2 + i] : g[i], send = up ? g[i] : g[N / 2 + i];
    h[i] = keep + __shfl_xor_sync(LAD_FULL, send, 1);
  }
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const double keep = up2 ? h[N / 4 + i] : h[i], send = up2 ? h[i] : h[N / 4 + i];
    out[i] = keep + __shfl_xor_sync(LAD_FULL, send, 2);
  }
}

// Sums of many words' closures at one step, which would be one task's serial chain: 12 or 16 lanes per (sum, state), each
// with a third or a quarter of a digit's pairs, so that four words' loads are in flight. Bound: the latency of
// loads that depend on the word's record. With tasks of single nodes, 64 qubits, 20,000 words, B = 1: the gradient 1,346 ->
// 530 us with it (the identity chain's steps close 150 words each), 40 qubits, 5,000 words: 437 -> 295 us.
template <bool REAL, int W>
__global__ void __launch_bounds__(128)
ladder_gather_kernel(LadBackParams p, int first, int count) {
  constexpr int NX = lad_lane_comps<REAL>(), SPLIT = REAL ? 3 : 4, NP = NX / 2 / SPLIT, AHEAD = 4;
  dependency_wait();
  const long long at = ((long long)blockIdx.x * 128 + threadIdx.x) >> 2, item = at / SPLIT;
  if (item >= (long long)count * p.B) return;
  const int q = threadIdx.x & 3, part = (int)(at % SPLIT), b = (int)(item % p.B);
  const int slot = first + (int)(item / p.B);
  const LadGather g = p.gathers[slot];
  const size_t slot_size = (size_t)p.B * (4 * NX), at_b = lad_state<W, NX>(b);
  const double *other = (g.half ? p.envp : p.envs) + at_b;
  constexpr int S = lad_stride<W>();
  double2 x[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) x[i] = make_double2(0.0, 0.0);
  for (int c = 0; c < g.count; c += AHEAD) {
    LadClose cl[AHEAD];
    double2 v[AHEAD][NP];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      cl[k] = p.closers[g.first + min(c + k, g.count - 1)];
      if (c + k >= g.count) cl[k].coef = 0.0;
    }
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const bool use = c + k < g.count && ((cl[k].flags & 2) || q == 0 || q == 3);
      const double2 *src = lad_at<W, NX>(((cl[k].flags & 4) ? p.gathered + at_b : other) + cl[k].slot * slot_size, q) +
                           S * NP * part;
#pragma unroll
      for (int i = 0; i < NP; ++i) v[k][i] = use ? src[S * i] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < AHEAD; ++k)
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        x[i].x = fma(cl[k].coef, v[k][i].x, x[i].x);
        x[i].y = fma(cl[k].coef, v[k][i].y, x[i].y);
      }
  }
  double2 *dst = const_cast<double2 *>(lad_at<W, NX>(p.gathered + at_b + slot * slot_size, q)) + S * NP * part;
#pragma unroll
  for (int i = 0; i < NP; ++i) dst[S * i] = x[i];
}

constexpr int LAD_BACK = 32;         // threads: one warp, so that shared memory holds as many as it can
template <bool REAL> __host__ __device__ constexpr int lad_back_arrays() { return REAL ? 3 * LAD_XR : 5 * LAD_XC; }
template <bool REAL> __host__ __device__ constexpr size_t lad_back_smem() {
  return (size_t)(lad_back_arrays<REAL>() * LAD_BACK + 2 * (LAD_BACK / 4) * (REAL ? LAD_REAL_COEFS : LAD_COEFS)) *
         sizeof(double);
}

// Bound: FP64 issue, shared memory and the latencies that seven warps an SM leave (64 qubits, B = 16: FP64 pipe
// 25 % busy, shared-memory pipe 57 %). Real: the carried and the worked-on tensor in registers; the
// step's input, which arrives by cp.async one step ahead, and one chain member in shared memory (30 KB a
// warp); the other member is formed again, which is cheaper than the place that would cost two warps an SM.
// What the two classes of lanes share, loads and stores, stands outside their branches: the loop has
// to stay in the instruction cache. Complex: the carried tensor and four members in shared memory (82 KB a
// warp, two an SM), rotations read where they are used: held for the step they spilled 5 KB a thread.
// Measured (B200), whole gradient call, 16 x 16 transfer products -> this: 64 qubits, 20,000 words, B = 32:
// 20,850 -> 3,450 us; 40 qubits, 5,000 words, B = 1: 1,488 -> 346 us; complex, 21 qubits, 790 words, B = 7:
// 876 -> 292 us.
template <bool REAL, int W>
__global__ void __launch_bounds__(LAD_BACK, REAL ? 7 : 2)
ladder_back_kernel(LadBackParams p) {
  constexpr int NC = REAL ? LAD_REAL_COEFS : LAD_COEFS;
  constexpr int NX = lad_lane_comps<REAL>();
  constexpr int NT = LAD_BACK;
  constexpr int NG = REAL ? LAD_GR : LAD_GC;
  extern __shared__ __align__(16) double lad_smem[];
  double *rows = lad_smem + (size_t)lad_back_arrays<REAL>() * NT;      // [2][NT / 4][NC]
  const int tid = threadIdx.x, lane = tid & 31, q = lane & 3;
  auto keep = [&](int arr, int j) -> double & { return lad_smem[(size_t)(arr * NX + j) * NT + tid]; };   // complex
  auto keep2 = [&](int arr, int i) -> double2 & {                                                    // real: pairs
    return reinterpret_cast<double2 *>(lad_smem)[(size_t)(arr * (NX / 2) + i) * NT + tid];
  };
  const int B = p.B;
  const long long quad = ((long long)blockIdx.x * NT + tid) >> 2;
  const long long npre_q = (long long)p.npre * B, pre_pad = (npre_q + 7) & ~7LL;
  const bool suffix = quad >= pre_pad;
  const long long idx = suffix ? quad - pre_pad + npre_q : quad;
  const bool live = suffix ? idx < (long long)p.ntasks * B : quad < npre_q;
  LadTask task{};
  int b = 0;
  if (live) {
    task = p.tasks[idx / B];
    b = (int)(idx % B);
  }
  constexpr int ENV = W * 4 * NX;                    // of the constants
  const size_t slot_size = (size_t)B * (4 * NX), at_b = lad_state<W, NX>(b);
  const double *own = (suffix ? p.envs : p.envp) + at_b, *other = (suffix ? p.envp : p.envs) + at_b;
  double *cots = (suffix ? p.cots : p.cotp) + at_b;
  int longest = task.nsteps;
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(LAD_FULL, longest, o));
  auto word = [&](int i) { return i >= 0 && i < task.nsteps ? p.steps[task.step + i] : 0u; };
  auto record = [&](int i) {
    int4 v = make_int4(-1, -1, -2, 0);
    if (i >= 0 && i < task.nsteps) v = *reinterpret_cast<const int4 *>(p.back + task.step + i);
    return LadBack{v.x, v.y, v.z, v.w};
  };
  auto flips = [](uint32_t w) { const int code = w & 3; return code == 0 ? 0 : (code == 2 ? 2 : 1); };
  // the input environment of a step, for this lane's role at that end
  auto input_at = [&](const LadBack &rec, uint32_t w, int r) {
    if (!((w & 128) || r == 0 || r == 3)) return p.consts + 2 * ENV;
    return rec.in < 0 ? p.consts + (suffix ? ENV : 0) : own + rec.in * slot_size;
  };
  // rotations (and real inputs) of iteration t's step
  auto stage = [&](int t, uint32_t w, const LadBack &rec, int r) {
    if (t < task.nsteps) {
      const double *src = p.coef + ((size_t)(w >> 16) * B + b) * NC;
      double *dst = rows + (size_t)((t & 1) * (NT / 4) + (tid >> 2)) * NC;
#pragma unroll
      for (int i = 0; i < NC / 2; i += 4)
        if (i + q < NC / 2) lad_cp16(dst + 2 * (i + q), src + 2 * (i + q));
      if constexpr (REAL) {
        const double2 *in = lad_at<W, NX>(input_at(rec, w, r), r);
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) lad_cp16(&keep2(1 + (t & 1), i), in + lad_stride<W>() * i);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  uint32_t w_now = word(task.nsteps - 1), w_next = word(task.nsteps - 2);
  LadBack rec_now{}, rec_next{};       // real: read ahead (complex steps have no registers for it)
  if (REAL) {
    rec_now = record(task.nsteps - 1);
    rec_next = record(task.nsteps - 2);
  }
  int close_end = live ? p.back[task.step + task.nsteps].close : 0;
  dependency_wait();
  stage(0, w_now, rec_now, lad_role(q, flips(w_now)));
  double y[NX];                        // the carried cotangent (right end of the step for prefix, left end for suffix)
#pragma unroll
  for (int j = 0; j < NX; ++j) y[j] = 0.0;
  int swaps = 0;                       // real: roles of the lanes of y
  bool fresh = true;                   // y starts from zero at this step
  for (int t = 0; t < longest; ++t) {
    const int i = task.nsteps - 1 - t;
    const bool on = i >= 0;
    const uint32_t w = w_now;
    const LadBack rec = REAL ? rec_now : record(i);
    w_now = w_next;
    w_next = word(i - 2);
    if (REAL) {
      rec_now = rec_next;
      rec_next = record(i - 2);
    }
    const int code = w & 3, flip = flips(w);
    if (fresh) swaps = 0;
    stage(t + 1, w_now, rec_now, lad_role(q, (rec.cot_out != -1 ? 0 : swaps ^ flip) ^ flips(w_now)));
    const int par = (w >> 6) & 1;                    // before the task's own step: left end (prefix), right end (suffix)
    const bool xy = (w & 128) != 0;                  // lanes X, Y of the step's input environment
    const int end_par = par ^ (code == 2);           // at the step's result
    // ---- y: carried, collected and the words that close here
    if (fresh) {
#pragma unroll
      for (int j = 0; j < NX; ++j) y[j] = 0.0;
    }
    int role = REAL ? lad_role(q, swaps) : q;
    {
      const bool iz = role == 0 || role == 3;
      if (rec.cot_add >= 0) {
        const double2 *src = lad_at<W, NX>(cots + rec.cot_add * slot_size, role);
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) {
          const double2 v = src[lad_stride<W>() * i];
          y[2 * i] += v.x;
          y[2 * i + 1] += v.y;
        }
      }
      if (on)
      for (int c = rec.close; c < close_end; ++c) {
        const LadClose cl = p.closers[c];
        if (!(cl.flags & 2) && !iz) continue;
        const double2 *src = lad_at<W, NX>(((cl.flags & 4) ? p.gathered + at_b : other) + cl.slot * slot_size, role);
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) {
          const double2 v = src[lad_stride<W>() * i];
          y[2 * i] = fma(cl.coef, v.x, y[2 * i]);
          y[2 * i + 1] = fma(cl.coef, v.y, y[2 * i + 1]);
        }
      }
    }
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncwarp();
    const double *c = rows + (size_t)((t & 1) * (NT / 4) + (tid >> 2)) * NC;
    double g[REAL ? NG : LAD_GROUP];
    auto clear = [&] {
#pragma unroll
      for (double &v : g) v = 0.0;
    };
    clear();
    // derivatives first .. of this step, summed over the quad
    auto flush = [&](int first) {
      constexpr int N = REAL ? NG : LAD_GROUP;
      double sums[N / 4];
      lad_quad_sums<N>(g, q, sums);
      if (on) {
        double *dst = p.part + ((size_t)(task.step + i) * NG + first + (N / 4) * (2 * (q & 1) + (q >> 1))) * B + b;
#pragma unroll
        for (int j = 0; j < N / 4; ++j) dst[(size_t)j * B] = sums[j];
      }
    };
    if (on) close_end = rec.close;
    if constexpr (REAL) {
      double x[NX];
      // roles at the left end; SF and its transpose scale a lane by the same factor, set by its role there
      const int lswaps = suffix ? swaps : swaps ^ flip;
      const int lrole = lad_role(q, lswaps), prole = lrole ^ 1;
      const int lpar = suffix ? end_par : par;
      const int cls = lpar ^ (lrole == 2);
      const bool iz = lrole == 0 || lrole == 3;
      const int src = (lane & ~3) | lad_role(prole, lswaps);
      const double u = lad_factor(c, code, lrole, 1.0), up = lad_factor(c, code, prole, 1.0);
      const LadS4 r4 = lad_s4_rows<true>(lad_rot<true>(c, 2, 1.0), lrole);
      const bool hi = lrole >= 2;
      const bool left_xy = suffix ? (w & 8) != 0 : xy;                 // lanes X, Y at the left end count
      const bool any = __any_sync(LAD_FULL, on && (code != 0 || left_xy));
      const bool busy = any || iz;
      const double s0 = hi ? -r4.sy : r4.sx, s1 = hi ? r4.sy : r4.sx;
      const double ce = cls ? s1 : s0, co = cls ? s0 : s1;
      double ga = 0.0, gb = 0.0, gw = 0.0;
      auto put = [&] {
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) keep2(0, i) = make_double2(x[2 * i], x[2 * i + 1]);
      };
      auto get = [&](int arr) {
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) {
          const double2 v = keep2(arr, i);
          x[2 * i] = v.x;
          x[2 * i + 1] = v.y;
        }
      };
      if (!suffix) {
        // t -> T1, T2 (kept), T3
        get(1 + (t & 1));
        if (busy) {
          const LadRot o2 = lad_rot<true>(c, 0, 1.0);
          if (cls == 0) {
            lad_s1r<0>(x, c[0], c[1]);
            lad_skr<0, 2>(x, o2);
          } else {
            lad_s1r<1>(x, c[0], c[1]);
            lad_skr<1, 2>(x, o2);
          }
          put();
          const LadRot o3 = lad_rot<true>(c, 1, 1.0);
          if (cls == 0) lad_skr<0, 3>(x, o3);
          else lad_skr<1, 3>(x, o3);
        }
        __syncwarp();
        // W: products of y with T4 (S4 without the code's factor); S4 and its transpose with their products
        if (any) {
          lad_for<16>([&](auto G) {
            constexpr int k = decltype(G)::v;
            const double cc = lad_gpar(k) ? co : ce;
            const double tv = __shfl_sync(LAD_FULL, cc * x[k], src), r = __shfl_sync(LAD_FULL, y[k], src);
            gw = fma(y[k], fma(r4.kx, x[k], tv), gw);
            gb = fma(hi ? y[k] : r, x[k], gb);
            // the transposed exchange multiplies at the receiver
            y[k] = fma(u * r4.kx, y[k], (up * cc) * r);
          });
#pragma unroll
          for (int m = 16; m < NX; m += 2) {
            const double vi = x[m], vz = x[m + 1], yi = y[m], yz = y[m + 1];
            const double ti = __shfl_sync(LAD_FULL, r4.sz * vz, src), tz = __shfl_sync(LAD_FULL, r4.sz * vi, src);
            const double ri = __shfl_sync(LAD_FULL, yi, src), rz = __shfl_sync(LAD_FULL, yz, src);
            gw = fma(yi, fma(r4.ki, vi, fma(r4.kz, vz, ti)), gw);
            gw = fma(yz, fma(r4.ki, vz, fma(r4.kz, vi, tz)), gw);
            ga = fma(hi ? yi : ri, vz, fma(hi ? yz : rz, vi, ga));
            y[m] = fma(u * r4.ki, yi, fma(u * r4.kz, yz, (up * r4.sz) * rz));
            y[m + 1] = fma(u * r4.ki, yz, fma(u * r4.kz, yi, (up * r4.sz) * ri));
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            gb = fma(hi ? y[k] : 0.0, x[k], gb);
            y[k] *= u * r4.kx;
          }
#pragma unroll
          for (int m = 16; m < NX; m += 2) {
            const double yi = y[m], yz = y[m + 1];
            ga = fma(hi ? yi : 0.0, x[m + 1], fma(hi ? yz : 0.0, x[m], ga));
            y[m] = fma(u * r4.ki, yi, u * r4.kz * yz);
            y[m + 1] = fma(u * r4.ki, yz, u * r4.kz * yi);
          }
        }
        ga *= hi ? u : up;
        gb *= hi ? u : up;
        if (busy) {
          get(0);
          const LadRot p3 = lad_rot<true>(c, 1, 1.0);
          if (cls == 0) {
            lad_gkr<0, 3>(y, [&](int j) { return x[j]; }, g[6], g[7], g[8], g[9]);
            lad_skr<0, 3>(y, p3);
          } else {
            lad_gkr<1, 3>(y, [&](int j) { return x[j]; }, g[6], g[7], g[8], g[9]);
            lad_skr<1, 3>(y, p3);
          }
          get(1 + (t & 1));                          // T1 once more: cheaper than a place to keep it
          const LadRot p2 = lad_rot<true>(c, 0, 1.0);
          if (cls == 0) {
            lad_s1r<0>(x, c[0], c[1]);
            lad_gkr<0, 2>(y, [&](int j) { return x[j]; }, g[2], g[3], g[4], g[5]);
            lad_skr<0, 2>(y, p2);
          } else {
            lad_s1r<1>(x, c[0], c[1]);
            lad_gkr<1, 2>(y, [&](int j) { return x[j]; }, g[2], g[3], g[4], g[5]);
            lad_skr<1, 2>(y, p2);
          }
          get(1 + (t & 1));
          if (cls == 0) {
            lad_g1r<0>(y, [&](int j) { return x[j]; }, g[0], g[1]);
            lad_s1r<0>(y, c[0], c[1]);
          } else {
            lad_g1r<1>(y, [&](int j) { return x[j]; }, g[0], g[1]);
            lad_s1r<1>(y, c[0], c[1]);
          }
        }
        __syncwarp();
        swaps = lswaps;
      } else {
        // w -> (transposed SF, S4) kept, S3, S2: the cotangent at S1's output
        get(1 + (t & 1));
        lad_s4r_t(x, r4, lrole, cls, src, u, up, any);
        if (busy) {
          put();
          const LadRot o3 = lad_rot<true>(c, 1, 1.0), o2 = lad_rot<true>(c, 0, 1.0);
          if (cls == 0) {
            lad_skr<0, 3>(x, o3);
            lad_skr<0, 2>(x, o2);
            lad_g1r<0>(x, [&](int j) { return y[j]; }, g[0], g[1]);
            lad_s1r<0>(y, c[0], c[1]);
          } else {
            lad_skr<1, 3>(x, o3);
            lad_skr<1, 2>(x, o2);
            lad_g1r<1>(x, [&](int j) { return y[j]; }, g[0], g[1]);
            lad_s1r<1>(y, c[0], c[1]);
          }
          get(0);
          const LadRot q3 = lad_rot<true>(c, 1, 1.0), p2 = lad_rot<true>(c, 0, 1.0);
          if (cls == 0) {
            lad_skr<0, 3>(x, q3);
            lad_gkr<0, 2>(y, [&](int j) { return x[j]; }, g[2], g[3], g[4], g[5]);
            lad_skr<0, 2>(y, p2);
          } else {
            lad_skr<1, 3>(x, q3);
            lad_gkr<1, 2>(y, [&](int j) { return x[j]; }, g[2], g[3], g[4], g[5]);
            lad_skr<1, 2>(y, p2);
          }
          get(0);
          const LadRot p3 = lad_rot<true>(c, 1, 1.0);
          if (cls == 0) {
            lad_gkr<0, 3>(y, [&](int j) { return x[j]; }, g[6], g[7], g[8], g[9]);
            lad_skr<0, 3>(y, p3);
          } else {
            lad_gkr<1, 3>(y, [&](int j) { return x[j]; }, g[6], g[7], g[8], g[9]);
            lad_skr<1, 3>(y, p3);
          }
        }
        __syncwarp();
        // T3 = y; w again; S4 forwards with its products, W, SF
        get(1 + (t & 1));
        if (any) {
          lad_for<16>([&](auto G) {
            constexpr int k = decltype(G)::v;
            const double cc = lad_gpar(k) ? co : ce;
            const double tv = __shfl_sync(LAD_FULL, cc * y[k], src), r = __shfl_sync(LAD_FULL, y[k], src);
            gb = fma(x[k], hi ? y[k] : r, gb);
            const double t4 = fma(r4.kx, y[k], tv);
            gw = fma(x[k], t4, gw);
            y[k] = u * t4;
          });
#pragma unroll
          for (int m = 16; m < NX; m += 2) {
            const double vi = y[m], vz = y[m + 1];
            const double ri = __shfl_sync(LAD_FULL, vi, src), rz = __shfl_sync(LAD_FULL, vz, src);
            ga = fma(x[m], hi ? vz : rz, fma(x[m + 1], hi ? vi : ri, ga));
            const double ti = fma(r4.ki, vi, fma(r4.kz, vz, r4.sz * rz)), tz = fma(r4.ki, vz, fma(r4.kz, vi, r4.sz * ri));
            gw = fma(x[m], ti, fma(x[m + 1], tz, gw));
            y[m] = u * ti;
            y[m + 1] = u * tz;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            gb = fma(x[k], hi ? y[k] : 0.0, gb);
            y[k] *= u * r4.kx;
          }
#pragma unroll
          for (int m = 16; m < NX; m += 2) {
            const double vi = y[m], vz = y[m + 1];
            ga = fma(x[m], hi ? vz : 0.0, fma(x[m + 1], hi ? vi : 0.0, ga));
            y[m] = u * fma(r4.ki, vi, r4.kz * vz);
            y[m + 1] = u * fma(r4.ki, vz, r4.kz * vi);
          }
        }
        ga *= u;
        gb *= u;
        swaps = lswaps ^ flip;
      }
      gw = (code == 1 || code == 3) ? gw : 0.0;
      g[10] = hi ? 0.0 : gb;           // lanes I and X: the rows they send, lanes Y and Z: those they keep
      g[11] = hi ? 0.0 : ga;
      g[12] = hi ? gb : 0.0;
      g[13] = hi ? ga : 0.0;
      g[14] = iz ? 0.0 : gw;
      g[15] = iz ? gw : 0.0;
      flush(0);
    } else {
      double x[NX];
      const bool iz = q == 0 || q == 3;
      const bool hi = q >= 2;
      const double *in = input_at(rec, on ? w : 0, q);
      auto rot = [&](int k, double ysign) { return lad_rot<false>(c, k, ysign); };   // read where it is used
      auto r4 = [&] { return lad_s4_rows<false>(rot(2, 1.0), q); };
      auto sf = [&](double tsign) { return lad_sf_row(c, q, code, tsign); };
      const double psign = q == 3 ? -1.0 : 1.0;      // lane Z receives -y of lane Y; lane Y +y of lane Z
      // products of S4's output cotangent w4 (own) with its input T3 (own, and the partner's)
      auto g4 = [&](auto w4, auto t3own, auto t3other) {
        double kz = 0, kx = 0, ky = 0, rz = 0, rx = 0, ry = 0;
#pragma unroll
        for (int o = 0; o < 16; ++o) {
          const double wi = w4(o), wx = w4(o + 16), wy = w4(o + 32), wz = w4(o + 48);
          const double vi = t3own(o), vx = t3own(o + 16), vy = t3own(o + 32), vz = t3own(o + 48);
          const double pi = t3other(o, vi), px = t3other(o + 16, vx), py = t3other(o + 32, vy), pz = t3other(o + 48, vz);
          kz = fma(wi, vz, fma(wz, vi, kz));
          kx = fma(wx, vx, fma(wy, vy, kx));
          ky = fma(wx, vy, fma(-wy, vx, ky));
          rz = fma(wi, pz, fma(wz, pi, rz));
          rx = fma(wx, px, fma(wy, py, rx));
          ry = fma(wx, py, fma(-wy, px, ry));
        }
        // kept row z (lanes Y, Z); received row x (lanes I, X) or +-y
        if (hi) {
          g[6] = kx; g[7] = ky; g[8] = kz;
          g[3] = psign * rx; g[4] = psign * ry; g[5] = psign * rz;
        } else {
          g[0] = rx; g[1] = ry; g[2] = rz;
        }
      };
      // products of the result's cotangent w5 with T4 for this code's row of W
      auto gw = [&](auto w5, auto t4) {
        double a = 0.0, d = 0.0;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const double v = t4(j), r = __shfl_xor_sync(LAD_FULL, v, 3), wv = w5(j);
          a = fma(wv, iz ? r : v, a);
          d = fma(wv, r, d);
        }
        if (code != 0) {
          if (iz) g[11] = a;
          else {
            g[9] = a;
            g[10] = q == 1 ? d : -d;
          }
        }
      };
      auto other3 = [&](int, double v) { return __shfl_xor_sync(LAD_FULL, v, 1); };
      auto at = [&](int arr) { return [&keep, arr](int j) { return keep(arr, j); }; };
      auto put = [&](int arr) {
#pragma unroll
        for (int j = 0; j < NX; ++j) keep(arr, j) = x[j];
      };
      if (!suffix) {
        // y parked; t -> T1, T2, T3 kept, T4
#pragma unroll
        for (int j = 0; j < NX; ++j) keep(4, j) = y[j];
        lad_get<W>(x, in, q);
        put(0);
        lad_s1c(x, c[0], c[1], c[2]);
        put(1);
        lad_skc<1, 4, 16>(x, rot(0, 1.0));
        put(2);
        lad_skc<4, 16, 1>(x, rot(1, 1.0));
        put(3);
        lad_s4c(x, r4(), true);
        gw(at(4), [&](int j) { return x[j]; });
#pragma unroll
        for (int j = 0; j < NX; ++j) x[j] = keep(4, j);
        lad_sf(x, sf(-1.0));
        g4([&](int j) { return x[j]; }, at(3), other3);
        flush(2 * LAD_GROUP);
        clear();
        lad_s4c_t(x, r4(), true);
        lad_gkc<4, 16, 1>([&](int j) { return x[j]; }, at(2), g);
        flush(LAD_GROUP);
        clear();
        lad_skc<4, 16, 1>(x, rot(1, -1.0));
        lad_gkc<1, 4, 16>([&](int j) { return x[j]; }, at(1), g + 3);
        lad_skc<1, 4, 16>(x, rot(0, -1.0));
        lad_g1c([&](int j) { return x[j]; }, at(0), g);
        flush(0);
        lad_s1c(x, c[0], -c[1], c[2]);
      } else {
        // y parked; w, then S4's, S3's and S2's output cotangents kept
#pragma unroll
        for (int j = 0; j < NX; ++j) keep(4, j) = y[j];
        lad_get<W>(x, in, q);
        lad_sf(x, sf(-1.0));
        put(3);
        lad_s4c_t(x, r4(), true);
        put(2);
        lad_skc<4, 16, 1>(x, rot(1, -1.0));
        put(1);
        lad_skc<1, 4, 16>(x, rot(0, -1.0));
        lad_g1c([&](int j) { return x[j]; }, at(4), g);
#pragma unroll
        for (int j = 0; j < NX; ++j) x[j] = keep(4, j);
        lad_s1c(x, c[0], c[1], c[2]);
        lad_gkc<1, 4, 16>(at(1), [&](int j) { return x[j]; }, g + 3);
        flush(0);
        clear();
        lad_skc<1, 4, 16>(x, rot(0, 1.0));
        lad_gkc<4, 16, 1>(at(2), [&](int j) { return x[j]; }, g);
        flush(LAD_GROUP);
        clear();
        lad_skc<4, 16, 1>(x, rot(1, 1.0));
        g4(at(3), [&](int j) { return x[j]; }, other3);
        lad_s4c(x, r4(), true);
        put(0);
        lad_get<W>(x, in, q);
        gw([&](int j) { return x[j]; }, at(0));
        flush(2 * LAD_GROUP);
#pragma unroll
        for (int j = 0; j < NX; ++j) x[j] = keep(0, j);
        lad_sf(x, sf(1.0));
      }
#pragma unroll
      for (int j = 0; j < NX; ++j) y[j] = x[j];
    }
    // ---- where the cotangent goes
    fresh = rec.cot_out != -1;
    if (on && rec.cot_out >= 0) {
      role = REAL ? lad_role(q, swaps) : q;
      double *dst = cots + (rec.cot_out >> 1) * slot_size;
      if (!(rec.cot_out & 1)) {
        const double2 *src = lad_at<W, NX>(dst, role);
#pragma unroll
        for (int i = 0; i < NX / 2; ++i) {
          const double2 v = src[lad_stride<W>() * i];
          y[2 * i] += v.x;
          y[2 * i + 1] += v.y;
        }
      }
      lad_put<W>(y, dst, role);
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Sums over the steps of a site in a fixed order: 32 partial sums (step i of the list into sum i mod 32), then
// those in order. site_off: 4 x site + code. Outputs [site][39 or 18][B]: the stage derivatives over all codes,
// then the rows of W (real: X and Z rows' x and z entries).
template <bool REAL>
__global__ void __launch_bounds__(256)
ladder_site_sum_kernel(const double *__restrict__ part, const int32_t *__restrict__ site_off,
                       const int32_t *__restrict__ steps, int B, double *__restrict__ out) {
  constexpr int NG = REAL ? LAD_GR : LAD_GC, STAGE = REAL ? 14 : 30, NW = REAL ? 2 : 3;
  constexpr int NO = REAL ? 18 : 39;
  __shared__ double red[32][33];
  dependency_wait();
  const int site = blockIdx.x, o = blockIdx.y;
  int g = !REAL && o >= 21 ? o + 3 : o, lo = site_off[4 * site], hi = site_off[4 * site + 4];
  if (o >= STAGE) {
    const int row = (o - STAGE) / NW, code = REAL ? (row == 0 ? 1 : 3) : row + 1;
    g = (REAL ? STAGE : STAGE + 3) + (o - STAGE) % NW;
    lo = site_off[4 * site + code];
    hi = site_off[4 * site + code + 1];
  }
  // threads: bt states x 256 / bt partial sums at a time
  int bt = 1;
  while (bt < 32 && bt < B) bt <<= 1;
  const int lb = threadIdx.x % bt, sub0 = threadIdx.x / bt, nsub = min(32, 256 / bt);
  const int b = blockIdx.z * bt + lb;
  if (sub0 < nsub)
    for (int sub = sub0; sub < 32; sub += nsub) {
      double acc = 0.0;
      if (b < B)
        for (int i = lo + sub; i < hi; i += 32) acc += part[((size_t)steps[i] * NG + g) * B + b];
      red[sub][lb] = acc;
    }
  __syncthreads();
  if (threadIdx.x < bt && b < B) {
    double acc = 0.0;
    for (int sub = 0; sub < 32; ++sub) acc += red[sub][threadIdx.x];
    out[((size_t)site * NO + o) * B + b] = acc;
  }
}

struct LadAngleParams {
  const LadGate *gates;
  const int32_t *off;
  const cplx *mats;
  const double *theta;
  const double *sums;       // [site][18 or 39][B]
  const double *poison;     // B
  double *stage;            // B x nslots: derivative of every gate's angle parameter
  int n, P, layers, hadamard, nslots, B;
  cplx prep[4];
};

// Derivatives by the gates' angles: with O = A G_j B (Bloch matrices), dO / dangle_j = A K_j G_j B, K_j the
// generator of the rotation. One thread per (state, site, layer).
template <bool REAL>
__global__ void __launch_bounds__(128)
ladder_angle_kernel(LadAngleParams p) {
  constexpr int NO = REAL ? 18 : 39;
  dependency_wait();
  const int item = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  if (item >= p.n * (p.layers + 1)) return;
  const int s = item / (p.layers + 1), kk = item % (p.layers + 1);
  const int g0 = p.off[item], g1 = p.off[item + 1];
  if (g0 == g1) return;
  const int k = kk + (LAD_MAX_LAYERS - p.layers);             // 0: n, 1 .. 3: S2 .. S4, 4: W
  const double *sum = p.sums + (size_t)s * NO * p.B + b;
  auto at = [&](int i) { return sum[(size_t)i * p.B]; };
  double a[9];                                                // derivative by O, then by A's right end
  for (int i = 0; i < 9; ++i) a[i] = 0.0;
  if (REAL) {
    if (k == 0) {
      a[2] = at(0); a[8] = at(1);
    } else if (k < 4) {
      const int o = 2 + 4 * (k - 1);
      a[0] = at(o); a[2] = at(o + 1); a[6] = at(o + 2); a[8] = at(o + 3);
    } else {
      a[0] = at(14); a[2] = at(15); a[6] = at(16); a[8] = at(17);
    }
  } else if (k == 0) {
    a[2] = at(0); a[5] = at(1); a[8] = at(2);
  } else {
    const int o = 3 + 9 * (k - 1);
    for (int i = 0; i < 9; ++i) a[i] = at(o + i);
  }
  const double *th = p.theta + (size_t)b * p.P;
  auto left_t = [&](const double *o, double *m) {             // m <- o^T m
    double t[9];
    for (int r = 0; r < 3; ++r)
      for (int cc = 0; cc < 3; ++cc) t[3 * r + cc] = o[r] * m[cc] + o[3 + r] * m[3 + cc] + o[6 + r] * m[6 + cc];
    for (int i = 0; i < 9; ++i) m[i] = t[i];
  };
  double o[9];
  if (k < 4 && p.hadamard) {
    bloch_hadamard(o);
    left_t(o, a);
  }
  for (int g = g1 - 1; g >= g0; --g) {
    const LadGate lg = p.gates[g];
    if (lg.slot >= 0) {
      double m[9];
      if (kk == 0) bloch_exact(p.prep, m);
      else if (p.hadamard) bloch_hadamard(m);
      else
        for (int i = 0; i < 9; ++i) m[i] = (i % 4 == 0) ? 1.0 : 0.0;
      for (int h = g0; h <= g; ++h) {
        bloch_gate(p.gates[h], p.mats, th, o);
        bloch_left(o, m);
      }
      // axis x v for every column of m: rows r1, r2 of the plane, d r1 = -r2, d r2 = r1 (cyclic after the axis)
      const int r1 = lg.rot == ROT_X ? 1 : lg.rot == ROT_Y ? 2 : 0, r2i = lg.rot == ROT_X ? 2 : lg.rot == ROT_Y ? 0 : 1;
      double d = 0.0;
      for (int cc = 0; cc < 3; ++cc) d += a[3 * r2i + cc] * m[3 * r1 + cc] - a[3 * r1 + cc] * m[3 * r2i + cc];
      p.stage[(size_t)b * p.nslots + lg.slot] = d * lg.angle + p.poison[b];
    }
    bloch_gate(lg, p.mats, th, o);
    left_t(o, a);
  }
}

}  // namespace vqemps
