// Perfect (Ferris-Vidal) bitstring sampling and shot estimates of Z words.
//
// Reference algorithm (test/backend/source/sharded_mps.cuh):
//   prepareSamplingRightEnvironments / k_rightStage / k_rightFinish  :814-836, 61-90
//   sampleBitsFromPreparedRight / k_sampleW / k_sampleProbabilities /
//   k_chooseSample / sampleHash                                      :838-877, 103-188
//   sampleZExpectationsGpu / k_zSampleSums                           :906-935, 193-214
//   sampleZExpectationsIndependentGpu (one stream per Z word)       :942-982
//
// B200 design: one THREAD per shot walks the sites in one launch (the reference
// launches three kernels per site). A CTA owns SAMPLE_THREADS shots of one
// state; at each site it stages the site tensor and the two branch matrices
// M_i[a,a'] = sum conj(A[a,i,c]) R_{s+1}[c,c'] A[a',i,c'] in shared memory (the
// right-environment sweep produces them: R_s = M_0 + M_1), and every thread
// reads them with warp-uniform addresses (broadcast). A shot keeps only its
// left vector v in registers. Bits are packed into 64-bit words in QUBIT order;
// Z-word parities are popcounts over 32 shots at a time.
//
// The walk is bound by FP64 multiply-adds, a quadratic form and a vector-matrix product per shot and
// site, so it takes as few as it can:
//  - M_i is Hermitian: half of it is read, 16 + 4 x 120 products a branch instead of 4 x 256;
//  - circuits of real gates (REAL) carry real vectors: a quarter of the rest;
//  - the first sites of all shots of a state share their vectors: there are only 2^s of them at site s, so
//    they are walked once (sample_kernel<2>, thread = prefix) into a table of thresholds and
//    vectors, and a shot's own walk starts where the table ends. The same operations in
//    the same order on the same numbers: the same bits as a walk from site 0.
// 22 qubits, two states, some 370 Z words of 1,000 shots each: 4,635 -> 678 us (table 155); 64 states of
// 8-48 qubits (real), 1,000 shots: 1,051 -> 267 us (table 15).
#pragma once
#include <type_traits>
#include "common.cuh"

namespace vqemps {

__host__ __device__ __forceinline__ uint64_t splitmix_hash(uint64_t x) {
  // SplitMix64 finaliser (Steele, Lea, Flood 2014), as sampleHash.
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}

__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
  // Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11).
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c[0];
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * c[2];
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0;
    const uint32_t n1 = (uint32_t)p1;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1;
    const uint32_t n3 = (uint32_t)p0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

// Uniform in [0, 1) for (seed, site, shot).
__device__ __forceinline__ double draw_uniform(int rng, uint64_t seed, int site, int shot) {
  if (rng == 0) {
    // reference: ((u64)seed << 32) ^ ((u64)site << 20) ^ shot, seed a 32-bit unsigned
    const uint64_t raw = splitmix_hash(((seed & 0xffffffffULL) << 32) ^
                                       ((uint64_t)site << 20) ^ (uint64_t)shot);
    return (double)(raw >> 11) * 0x1.0p-53;
  }
  uint32_t c[4] = {(uint32_t)shot, (uint32_t)site, 0u, 0u};
  philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const uint64_t bits53 = (((uint64_t)c[0] << 21) ^ ((uint64_t)c[1] >> 11)) & ((1ULL << 53) - 1);
  return (double)bits53 * 0x1.0p-53;
}

constexpr int SAMPLE_THREADS = 128;
constexpr int MAX_WORDS64 = 4;   // up to 256 qubits
constexpr int SAMPLE_MAX_DEPTH = 16;

struct SampleParams {
  const cplx *sites;        // B x n x SITE_ELEMS
  const cplx *branch;       // B x n x 2 x ENV_ELEMS: M_i of every site (right_env_kernel)
  const int32_t *status;    // B
  int n, shots, W;
  int site_order;           // 0: site = qubit, 1: site = n-1-qubit
  int rng;
  // shared mode: one seed per state (seeds[b]); per-word mode: seeds[b * nwords + listed word]
  const uint64_t *seeds;
  uint64_t *bits;           // shared mode: B x shots x W
  // per-word mode
  const uint64_t *zmask;    // T x W (qubit order)
  const int32_t *words;     // list of word indices to sample
  const int32_t *last_site; // per listed word: last site to sample (inclusive)
  int nwords;
  int32_t *sums;            // B x nwords
  // partition sets (null: uniform batch): width part_n[st_part[b]], stride n
  const int32_t *st_part;
  const int32_t *part_n;
  // prefixes walked before: p_0 / (p_0 + p_1) after the first s < depth draws x (x = the draws, the first one
  // highest) at thr[b][(1 << s) + x], the left vector after depth draws at vecs[b][x]. A state narrower than
  // depth stops at its width. Table mode extends them to depth_out, vecs_out.
  double *thr;              // B x 2^SAMPLE_MAX_DEPTH's used part (thr_stride)
  int thr_stride;
  const double *vecs;       // B x 2^depth x CHI (real or complex)
  int depth;
  double *vecs_out;
  int depth_out;
};

__device__ __forceinline__ void sample_copy16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void sample_copy8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__device__ __forceinline__ double sc_zero(double) { return 0.0; }
__device__ __forceinline__ cplx sc_zero(cplx) { return cmake(0, 0); }
__device__ __forceinline__ void sc_fma(double &o, double a, double b) { o = fma(a, b, o); }
__device__ __forceinline__ void sc_fma(cplx &o, cplx a, cplx b) { cfma(o, a, b); }
__device__ __forceinline__ double sc_scale(double a, double k) { return a * k; }
__device__ __forceinline__ cplx sc_scale(cplx a, double k) { return cscale(a, k); }
__device__ __forceinline__ double sc_norm(double a) { return a * a; }
__device__ __forceinline__ double sc_norm(cplx a) { return cabs2(a); }
__device__ __forceinline__ double sc_re(double a) { return a; }
__device__ __forceinline__ double sc_re(cplx a) { return a.x; }
__device__ __forceinline__ double sc_dot(double a, double b, double o) { return fma(a, b, o); }              // o + Re(conj(a) b)
__device__ __forceinline__ double sc_dot(cplx a, cplx b, double o) { return fma(a.x, b.x, fma(a.y, b.y, o)); }

// A site's operands; the rows of the two physical indices lie 16 bytes apart modulo the banks, for
// a warp's shots read either.
template <typename T>
struct SampleStage {
  static constexpr int AS = CHI + 16 / sizeof(T);
  T A[2 * CHI * AS];
  T M[2 * ENV_ELEMS];
};

template <typename T>
__device__ __forceinline__ void sample_stage(SampleStage<T> &d, const cplx *A, const cplx *M) {
  for (int e = threadIdx.x; e < SITE_ELEMS; e += SAMPLE_THREADS) {
    T *a = &d.A[(e >> 4) * SampleStage<T>::AS + (e & 15)];
    if constexpr (sizeof(T) == 16) {
      sample_copy16(a, A + e);
      sample_copy16(&d.M[e], M + e);
    } else {
      sample_copy8(a, A + e);
      sample_copy8(&d.M[e], M + e);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Re v^H M v from the upper half of M
template <typename T>
__device__ __forceinline__ double sample_form(const T *M, const T (&v)[CHI]) {
  double diag = 0.0, off = 0.0;
#pragma unroll
  for (int a = 0; a < CHI; ++a) {
    diag = fma(sc_re(M[a * CHI + a]), sc_norm(v[a]), diag);
    T y = sc_zero(T{});
#pragma unroll
    for (int ap = a + 1; ap < CHI; ++ap) sc_fma(y, M[a * CHI + ap], v[ap]);
    off = sc_dot(v[a], y, off);
  }
  return fma(2.0, off, diag);
}

// One thread = one shot. MODE 0: shared sample set, writes packed bits.
// MODE 1: independent stream per listed Z word, accumulates parity sums.
// MODE 2: thread = prefix of depth_out draws, writes the table.
template <int MODE, bool REAL>
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(SampleParams p) {
  using T = typename std::conditional<REAL, double, cplx>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SampleStage<T> *stage = reinterpret_cast<SampleStage<T> *>(smem_raw);
  __shared__ int red[SAMPLE_THREADS / 32];
  const int b = MODE == 1 ? blockIdx.z : blockIdx.y;
  const int widx = MODE == 1 ? blockIdx.y : 0;
  const int shot = blockIdx.x * SAMPLE_THREADS + threadIdx.x;
  const int nb = p.st_part ? p.part_n[p.st_part[b]] : p.n;
  const int depth = min(p.depth, nb);
  const int depth_out = MODE == 2 ? min(p.depth_out, nb) : 0;
  const bool live = MODE == 2 ? (shot >> depth_out) == 0 : shot < p.shots && p.status[b] == 0;
  const uint64_t seed = MODE == 2 ? 0 : (MODE == 0 ? p.seeds[b] : p.seeds[(size_t)b * p.nwords + widx]);
  const int last = MODE == 2 ? depth_out - 1 : (MODE == 0 ? nb - 1 : p.last_site[widx]);
  if (MODE == 2 && ((int)(blockIdx.x * SAMPLE_THREADS) >> depth_out) != 0) return;
  const cplx *sb = p.sites + (size_t)b * p.n * SITE_ELEMS;
  const cplx *mb = p.branch + (size_t)b * p.n * 2 * ENV_ELEMS;
  double *thr = p.thr + (size_t)b * p.thr_stride;

  if (depth <= last) sample_stage(stage[depth & 1], sb + (size_t)depth * SITE_ELEMS, mb + (size_t)depth * 2 * ENV_ELEMS);
  uint64_t word[MAX_WORDS64] = {0, 0, 0, 0};
  int x = 0;
  if (MODE == 2) {
    x = live ? shot >> (depth_out - depth) : 0;
  } else {
    for (int s = 0; s < depth && s <= last; ++s) {
      const double u = draw_uniform(p.rng, seed, s, shot);
      const int sel = u < thr[(1 << s) + x] ? 0 : 1;
      x = 2 * x + sel;
      const int q = p.site_order == 1 ? nb - 1 - s : s;
      if (sel) word[q >> 6] |= (1ULL << (q & 63));
    }
  }
  T v[CHI];
  if (depth > 0 && depth <= last) {
    const T *src = reinterpret_cast<const T *>(p.vecs) + (((size_t)b << p.depth) + x) * CHI;
#pragma unroll
    for (int a = 0; a < CHI; ++a) v[a] = src[a];
  } else {
#pragma unroll
    for (int a = 0; a < CHI; ++a) v[a] = sc_zero(T{});
    if constexpr (REAL) v[0] = 1.0;
    else v[0] = cmake(1.0, 0.0);
  }

  for (int s = depth; s <= last; ++s) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();   // this site's operands have arrived, the other buffer's are read
    if (s < last)
      sample_stage(stage[(s + 1) & 1], sb + (size_t)(s + 1) * SITE_ELEMS, mb + (size_t)(s + 1) * 2 * ENV_ELEMS);
    const SampleStage<T> &st = stage[s & 1];
    // p_i = Re v^H M_i v, the same number as Re(w_i^H R w_i), w_i = v A_i (k_sampleProbabilities)
    double p0 = sample_form<T>(st.M, v), p1 = sample_form<T>(st.M + ENV_ELEMS, v);
    p0 = p0 > 0.0 ? p0 : 0.0;
    p1 = p1 > 0.0 ? p1 : 0.0;
    double tot = p0 + p1;
    if (tot <= 0.0) { p0 = p1 = 0.5; tot = 1.0; }
    // k_chooseSample
    int sel;
    if (MODE == 2) {
      const int below = depth_out - 1 - s;
      sel = (shot >> below) & 1;
      if (live && (shot & ((2 << below) - 1)) == 0) thr[(1 << s) + (shot >> (below + 1))] = p0 / tot;
    } else {
      sel = draw_uniform(p.rng, seed, s, shot) < p0 / tot ? 0 : 1;
      const int q = p.site_order == 1 ? nb - 1 - s : s;
      if (sel) word[q >> 6] |= (1ULL << (q & 63));
    }
    const double ps = sel ? p1 : p0;
    const double inv = ps > 0.0 ? 1.0 / sqrt(ps) : 1.0;
    // v <- (v A_sel) / sqrt(p_sel)
    T w[CHI];
#pragma unroll
    for (int c = 0; c < CHI; ++c) w[c] = sc_zero(T{});
#pragma unroll
    for (int a = 0; a < CHI; ++a)
#pragma unroll
      for (int c = 0; c < CHI; ++c) sc_fma(w[c], v[a], st.A[(a * 2 + sel) * SampleStage<T>::AS + c]);
#pragma unroll
    for (int c = 0; c < CHI; ++c) v[c] = sc_scale(w[c], inv);
  }
  if (MODE == 2) {
    if (live) {
      T *dst = reinterpret_cast<T *>(p.vecs_out) + (((size_t)b << p.depth_out) + shot) * CHI;
#pragma unroll
      for (int a = 0; a < CHI; ++a) dst[a] = v[a];
    }
  } else if (MODE == 0) {
    if (live) {
      uint64_t *dst = p.bits + ((size_t)b * p.shots + shot) * p.W;
      for (int w = 0; w < p.W; ++w) dst[w] = word[w];
    }
  } else {
    int parity = 0;
    const uint64_t *mask = p.zmask + (size_t)p.words[widx] * p.W;
    for (int w = 0; w < p.W; ++w) parity ^= __popcll(word[w] & mask[w]) & 1;
    int val = live ? (parity ? -1 : 1) : 0;
    for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = val;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < SAMPLE_THREADS / 32; ++w) t += red[w];
      atomicAdd(p.sums + (size_t)b * p.nwords + widx, t);
    }
  }
}

// sums[b, t] = sum over shots of (-1)^popc(bits & zmask[t]) for every word t, one thread per word. The shots
// are turned into columns first (bit j of col[q][g]: qubit q of shot 32 g + j, one ballot each), so a word's
// parities of 32 shots are as many XORs as it has Z's and one popcount, instead of an AND, a
// popcount and an add per shot: 64 partitions, 1,000 shots, 200-3,000 words each 267 -> 23 us.
// st_part (partition sets, or null): state b uses the part_T[k] masks of partition k = st_part[b]
// (rows k * term_stride ..) and writes sums[b * term_stride + t].
constexpr int ZSUM_THREADS = 256;
constexpr int ZSUM_COLS = 16;              // columns words of a chunk: 512 shots
constexpr int ZSUM_STRIDE = ZSUM_COLS + 4; // 16-byte pieces of neighbouring qubits on different banks
__global__ void __launch_bounds__(ZSUM_THREADS)
zsum_kernel(const uint64_t *__restrict__ bits, int shots, int W, const uint64_t *__restrict__ zmask, int term_stride,
            const int32_t *__restrict__ st_part, const int32_t *__restrict__ part_T, int32_t *__restrict__ sums) {
  __shared__ __align__(16) uint32_t col[64 * MAX_WORDS64 * ZSUM_STRIDE];
  const int b = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = st_part ? st_part[b] : 0;
  const int T = st_part ? part_T[k] : term_stride;
  if (blockIdx.x * ZSUM_THREADS >= T) return;
  const int t = blockIdx.x * ZSUM_THREADS + threadIdx.x;
  uint64_t m[MAX_WORDS64] = {0, 0, 0, 0};
  if (t < T)
    for (int w = 0; w < W; ++w) m[w] = zmask[((size_t)k * term_stride + t) * W + w];
  int odd = 0;
  const uint64_t *bb = bits + (size_t)b * shots * W;
  for (int base = 0; base < shots; base += 32 * ZSUM_COLS) {
    __syncthreads();
    for (int it = warp; it < ZSUM_COLS * W; it += ZSUM_THREADS / 32) {
      const int g = it % ZSUM_COLS, w = it / ZSUM_COLS, shot = base + 32 * g + lane;
      const uint64_t v = shot < shots ? bb[(size_t)shot * W + w] : 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t half = (uint32_t)(v >> (32 * h));
        uint32_t mine = 0;
#pragma unroll
        for (int q = 0; q < 32; ++q) {
          const uint32_t c = __ballot_sync(0xffffffffu, (half >> q) & 1);
          if (lane == q) mine = c;
        }
        col[(64 * w + 32 * h + lane) * ZSUM_STRIDE + g] = mine;
      }
    }
    __syncthreads();
    uint4 x[ZSUM_COLS / 4];
#pragma unroll
    for (int i = 0; i < ZSUM_COLS / 4; ++i) x[i] = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int w = 0; w < MAX_WORDS64; ++w) {
      for (uint64_t left = m[w]; left; left &= left - 1) {
        const uint4 *c = reinterpret_cast<const uint4 *>(col + (64 * w + __ffsll((long long)left) - 1) * ZSUM_STRIDE);
#pragma unroll
        for (int i = 0; i < ZSUM_COLS / 4; ++i) {
          const uint4 v = c[i];
          x[i].x ^= v.x; x[i].y ^= v.y; x[i].z ^= v.z; x[i].w ^= v.w;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < ZSUM_COLS / 4; ++i) odd += __popc(x[i].x) + __popc(x[i].y) + __popc(x[i].z) + __popc(x[i].w);
  }
  if (t < T) sums[(size_t)b * term_stride + t] = shots - 2 * odd;
}

// Shot-estimated energies: value_t = sums[t] / shots for sampled words, the
// analytic per-term value for the others; fixed-order reduction per state.
__device__ __forceinline__ void sampled_energy_body(const int32_t *__restrict__ sums,
                                                    const int32_t *__restrict__ sum_index,
                                                    const double *__restrict__ analytic,
                                                    const double *__restrict__ coeffs, int T, int shots, bool ok,
                                                    double *__restrict__ energy, double *__restrict__ per_term) {
  __shared__ double part[REDUCE_THREADS];
  const int tid = threadIdx.x;
  double acc = 0.0;
  for (int t = tid; t < T; t += REDUCE_THREADS) {
    const int si = sum_index[t];
    // si >= 0: sampled word; -2: identity word (+1 on every shot); -1: analytic (X/Y)
    const double v = si >= 0 ? (double)sums[si] / shots : (si == -2 ? 1.0 : analytic[t]);
    if (per_term) per_term[t] = ok ? v : __longlong_as_double(0x7ff8000000000000LL);
    acc = fma(coeffs[t], v, acc);
  }
  part[tid] = acc;
  __syncthreads();
  for (int w = REDUCE_THREADS / 2; w > 0; w >>= 1) {
    if (tid < w) part[tid] += part[tid + w];
    __syncthreads();
  }
  if (tid == 0) *energy = ok ? part[0] : __longlong_as_double(0x7ff8000000000000LL);
}

__global__ void __launch_bounds__(REDUCE_THREADS)
sampled_energy_kernel(const int32_t *__restrict__ sums, int sums_stride, const int32_t *__restrict__ sum_index,
                      const double *__restrict__ analytic, const double *__restrict__ coeffs, int T, int shots,
                      const int32_t *__restrict__ status, double *__restrict__ energies,
                      double *__restrict__ per_term) {
  const int b = blockIdx.x;
  sampled_energy_body(sums + (size_t)b * sums_stride, sum_index, analytic ? analytic + (size_t)b * T : nullptr,
                      coeffs, T, shots, status[b] == 0, energies + b,
                      per_term ? per_term + (size_t)b * T : nullptr);
}

// Partition sets: every array is strided by term_stride, per partition
// (sum_index, coeffs) or per state (sums, analytic, per_term).
__global__ void __launch_bounds__(REDUCE_THREADS)
sampled_energy_multi_kernel(const int32_t *__restrict__ sums, const int32_t *__restrict__ sum_index,
                            const double *__restrict__ analytic, const double *__restrict__ coeffs,
                            int term_stride, const int32_t *__restrict__ st_part,
                            const int32_t *__restrict__ part_T, int shots, const int32_t *__restrict__ status,
                            double *__restrict__ energies, double *__restrict__ per_term) {
  const int b = blockIdx.x;
  const int k = st_part[b];
  const size_t so = (size_t)b * term_stride, po = (size_t)k * term_stride;
  sampled_energy_body(sums + so, sum_index + po, analytic ? analytic + so : nullptr, coeffs + po, part_T[k],
                      shots, status[b] == 0, energies + b, per_term ? per_term + so : nullptr);
}

}  // namespace vqemps
