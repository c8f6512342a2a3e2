// The 2-D DCT family and the Poisson solve on power-of-two grids, by fast
// transforms in shared memory (fp32).
//
// A dense cosine-matrix product spends O(n) operations per element and
// re-reads both operands from L2 for every tile; a fast transform spends
// O(log n) and reads and writes each element once per axis, so the solve
// becomes three passes over the maps:
//   1. rows:    T = rho C_N^T                    (two real rows per complex transform)
//   2. columns: a = 4/(M N) C_M T, the spectral weights, the energy, and both
//               inverse column transforms Sh_M (a wx), Ch_M (a wy) -- the
//               columns stay in shared memory between the three transforms
//   3. rows:    Ex = 4 (.) Ch_N^T, Ey = 4 (.) Sh_N^T, one complex transform per row
// against operand preparation and 4 GEMM launches of the dense form.  One solve,
// us, split-BF16 products -> fast transforms (replayed graph): 64^2 27 -> 11,
// 256^2 36 -> 13, 512^2 46 -> 15, 1024^2 68 -> 25, 2048^2 389 -> 65, 4096^2
// 2420 -> 243; relative error of the field (2-norm) at 1024^2 against fp64 4e-7
// to 5e-7 on GP states, the products' 2e-5 to 4e-5.  Up to 512^2 the three
// launches bound it, from 2048^2 issue and the exchanges (57% issue, 128 MB of
// rows in 38 us = 3.4 TB/s at 4096^2); at 1024^2 the column pass's 128 blocks.
//
// The 1-D transforms are Makhoul's (IEEE Trans. ASSP 28(1), 1980): with
// v[n] = x[2n], v[N-1-n] = x[2n+1] and V = FFT(v), w_k = exp(-i pi k / 2N),
//   DCT:    X[k] = Re(w_k V[k]),  and Im(w_k V[k]) = -X[N-k]
//   IDCT:   V[k] = conj(w_k) (a[k] - i a[N-k]), a[N] = 0;  Ch a = IFFT(V) / 2
//           (unnormalised inverse), read back through the same permutation
//   IDXST:  sin(pi p (u+1/2)/N) with p = N - q is (-1)^u cos(pi q (u+1/2)/N),
//           so Sh a = (-1)^u Ch a' with a'[q] = a[N-q], a'[0] = 0
// Two real transforms share one complex one: z = x1 + i x2 forward (separated
// by Z[k] +- conj Z[N-k]), V1 + i V2 inverse.  The complex transform is a
// Stockham autosort of radix 8 or 16 (Govindaraju et al., SC 2008), E points
// per thread in registers, exchanged through shared memory.
#include "epilogue.cuh"

namespace dpb {

constexpr int kFftMinLog = 6, kFftMaxLog = 12;  // sides 64 .. 4096

__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * w, or a * conj(w)
template <bool kConj>
__device__ __forceinline__ float2 c_mul(float2 a, float2 w) {
  return kConj ? make_float2(fmaf(a.x, w.x, a.y * w.y), fmaf(a.y, w.x, -a.x * w.y))
               : make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.y, w.x, a.x * w.y));
}
// a * (-i) forward, a * i inverse
template <bool kInv>
__device__ __forceinline__ float2 c_rot(float2 a) {
  return kInv ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool kInv>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
  const float2 t0 = c_add(a, c), t1 = c_sub(a, c), t2 = c_add(b, d), t3 = c_rot<kInv>(c_sub(b, d));
  a = c_add(t0, t2);
  b = c_add(t1, t3);
  c = c_sub(t0, t2);
  d = c_sub(t1, t3);
}

// in-place DFT of R points, natural order in and out
template <int R, bool kInv>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = c_add(a, b);
    v[1] = c_sub(a, b);
  } else if constexpr (R == 4) {
    dft4<kInv>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    constexpr float h = 0.70710678118654752f;
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4<kInv>(e[0], e[1], e[2], e[3]);
    dft4<kInv>(o[0], o[1], o[2], o[3]);
    const float2 w1 = make_float2(h, -h), w3 = make_float2(-h, -h);
    o[1] = c_mul<kInv>(o[1], w1);
    o[2] = c_rot<kInv>(o[2]);
    o[3] = c_mul<kInv>(o[3], w3);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = c_add(e[k], o[k]);
      v[k + 4] = c_sub(e[k], o[k]);
    }
  } else {
    static_assert(R == 16, "radix 2, 4, 8 or 16");
    // 4 x 4: X[k1 + 4 k2] = sum_n2 W16^(n2 k1) W4^(n2 k2) sum_n1 v[4 n1 + n2] W4^(n1 k1)
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
    const float2 w[10] = {{1.f, 0.f}, {c1, -s1}, {h, -h}, {s1, -c1}, {0.f, -1.f},
                          {-s1, -c1}, {-h, -h}, {-c1, -s1}, {-1.f, 0.f}, {-c1, s1}};
    float2 g[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      float2 a = v[n2], b = v[n2 + 4], c = v[n2 + 8], d = v[n2 + 12];
      dft4<kInv>(a, b, c, d);
      g[n2][0] = a;
      g[n2][1] = n2 ? c_mul<kInv>(b, w[n2]) : b;
      g[n2][2] = n2 ? (n2 == 2 ? c_rot<kInv>(c) : c_mul<kInv>(c, w[2 * n2])) : c;
      g[n2][3] = n2 ? c_mul<kInv>(d, w[3 * n2]) : d;
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      float2 a = g[0][k1], b = g[1][k1], c = g[2][k1], d = g[3][k1];
      dft4<kInv>(a, b, c, d);
      v[k1] = a;
      v[k1 + 4] = b;
      v[k1 + 8] = c;
      v[k1 + 12] = d;
    }
  }
}

// One transform's shape: N points, E per thread, N / E threads.
template <int LOGN>
struct FftShape {
  static constexpr int LOGE = LOGN >= 10 ? 4 : 3;
  static constexpr int N = 1 << LOGN, E = 1 << LOGE, T = N / E;
  // shared-memory pitch of a transform (float2): one pad per 16, and 4 mod 16
  // so that the four interleaved transforms of a column block fall on
  // different banks
  static constexpr int PITCH = (N + N / 16 + 15) / 16 * 16 + 4;
};

__device__ __forceinline__ constexpr int fft_pad(int i) { return i + (i >> 4); }

// register r (0..E) after the last pass holds point fft_out_base + fft_out_step:
// t + (r / RL) T + (r % RL) N / RL, RL the radix of the last pass
template <int LOGN>
__device__ __forceinline__ constexpr int fft_out_step(int r) {
  using S = FftShape<LOGN>;
  constexpr int RL = 1 << (LOGN % S::LOGE ? LOGN % S::LOGE : S::LOGE);
  return (r / RL) * S::T + (r % RL) * (S::N / RL);
}

// padded offset of adding the constant `step` to an index below 16 * (step's
// granularity): the pad of a sum is the sum of the pads when one of the two is
// a multiple of 16, or when no carry leaves the low four bits
template <int LOGN>
__device__ __forceinline__ int fft_at(int t, int step) {
  // steps are multiples of T; below 16 threads a transform's T does not clear
  // the low four bits and the pad is formed from the sum
  if constexpr (FftShape<LOGN>::T >= 16) return fft_pad(t) + step + step / 16;
  return fft_pad(t + step);
}

// v[m R + r] *= W^r, the powers formed from the one loaded root (each at most
// log2 r products deep: a few 2^-24; the loads of all R - 1 roots, strided
// across the warp, took longer than the products)
template <int R, bool kInv>
__device__ __forceinline__ void twiddle(float2* v, float2 w1) {
  float2 p[R];
  p[1] = w1;
  v[1] = c_mul<kInv>(v[1], w1);
#pragma unroll
  for (int r = 2; r < R; ++r) {
    p[r] = c_mul<false>(p[r / 2], p[r - r / 2]);
    v[r] = c_mul<kInv>(v[r], p[r]);
  }
}

// the passes after the first: exchange, twiddle, butterfly
template <int LOGN, int LOGNS, bool kInv>
__device__ __forceinline__ void fft_rest(float2* v, float2* s, const float2* __restrict__ W, int t) {
  using S = FftShape<LOGN>;
  if constexpr (LOGNS < LOGN) {
    constexpr int LOGR = LOGN - LOGNS < S::LOGE ? LOGN - LOGNS : S::LOGE;
    constexpr int R = 1 << LOGR, NB = S::E / R, LOGP = LOGNS - S::LOGE;  // LOGP: the previous pass's span
    // output r of the previous pass goes to (t >> LOGP << LOGNS) + (t mod 2^LOGP) + r 2^LOGP.
    // The pad of the sum is the sum of the pads: no carry leaves the low four
    // bits (a multiple of 16 is added, or r 2^LOGP fills the bits above base's)
    const int base = fft_pad(((t >> LOGP) << LOGNS) + (t & ((1 << LOGP) - 1)));
#pragma unroll
    for (int r = 0; r < S::E; ++r) s[base + fft_pad(r << LOGP)] = v[r];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      const int k = (t + m * S::T) & ((1 << LOGNS) - 1);
      const float2 w1 = __ldg(W + (k << (LOGN - LOGNS - LOGR)));
#pragma unroll
      for (int r = 0; r < R; ++r) v[m * R + r] = s[fft_at<LOGN>(t, m * S::T + r * (S::N / R))];
      twiddle<R, kInv>(v + m * R, w1);
      dft<R, kInv>(v + m * R);
    }
    __syncthreads();  // the buffer may be overwritten
    fft_rest<LOGN, LOGNS + LOGR, kInv>(v, s, W, t);
  }
}

// complex transform of the E points t + r T of each thread (natural order);
// the result sits in registers at fft_out_index.  The buffer s must be free on
// entry and is free on return.
template <int LOGN, bool kInv>
__device__ __forceinline__ void fft_run(float2* v, float2* s, const float2* __restrict__ W, int t) {
  dft<FftShape<LOGN>::E, kInv>(v);
  fft_rest<LOGN, FftShape<LOGN>::LOGE, kInv>(v, s, W, t);
}

// real index of permuted position n
template <int LOGN>
__device__ __forceinline__ int dct_src(int n) {
  constexpr int N = 1 << LOGN;
  return n < N / 2 ? 2 * n : 2 * N - 1 - 2 * n;
}

// (X1[k], X2[k]) of two packed real transforms from Z[k], Z[N-k]
__device__ __forceinline__ float2 dct_unpack(float2 zk, float2 zn, float2 w) {
  const float v1x = 0.5f * (zk.x + zn.x), v1y = 0.5f * (zk.y - zn.y);
  const float v2x = 0.5f * (zk.y + zn.y), v2y = 0.5f * (zn.x - zk.x);
  return make_float2(fmaf(v1x, w.x, -v1y * w.y), fmaf(v2x, w.x, -v2y * w.y));
}

// packed spectrum V1 + i V2 at k of two inverse transforms (IDCT, or IDXST
// where kSin): ak = (a1[k], a2[k]), an = (a1[N-k], a2[N-k])
template <bool kSin1, bool kSin2>
__device__ __forceinline__ float2 idct_pack(int k, float2 ak, float2 an, float2 w) {
  const float p1 = kSin1 ? an.x : ak.x, p2 = kSin2 ? an.y : ak.y;
  const float q1 = kSin1 ? ak.x : an.x, q2 = kSin2 ? ak.y : an.y;
  // k = 0: a[N] = 0 for the IDCT, both terms zero for the IDXST
  if (k == 0) return make_float2(kSin1 ? 0.f : ak.x, kSin2 ? 0.f : ak.y);
  return c_mul<true>(make_float2(p1 + q2, p2 - q1), w);
}

// ---------------------------------------------------------------- row staging
// A transform's two rows (or its row of pairs) are 8 N contiguous bytes: one
// thread copies them into the exchange buffers with bulk asynchronous copies,
// so each row is read once in full lines whatever order the permutation asks
// for.  The wait for the copies is bounded like the tensor-core GEMM's
// (dp_tc_set_wait_budget): on expiry status 2 is recorded (dp_tc_status) and
// the block returns, once its copies have landed (a second wait, bounded by
// kFftDrainCycles whatever the budget): a block that is gone must not have its
// shared memory written.
__device__ int g_fft_status = 0;
__device__ long long g_fft_wait_budget = 4000000000ll;  // ~2 s at 2 GHz
__device__ int g_fft_skip_loads = 0;                    // test hook (dp_tc_set_skip_loads)

__device__ __forceinline__ uint32_t fft_smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool fft_try_wait(uint64_t* bar) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(fft_smem_addr(bar))
      : "memory");
  return ok != 0;
}

__device__ __noinline__ bool fft_bounded_wait(uint64_t* bar) {
  const long long budget = g_fft_wait_budget, start = clock64();
  while (!fft_try_wait(bar))
    if (clock64() - start > budget) {
      atomicCAS(&g_fft_status, 0, 2);
      return false;
    }
  return true;
}

constexpr long long kFftDrainCycles = 4000000000ll;  // ~2 s at 2 GHz

__device__ __noinline__ void fft_drain(uint64_t* bar) {
  const long long start = clock64();
  while (!fft_try_wait(bar) && clock64() - start <= kFftDrainCycles) {
  }
}

enum { kRowDct = 0, kRowInv = 1, kRowInvPairs = 2 };

// transforms per block: at least 128 threads
template <int LOGN>
struct RowBlock {
  using S = FftShape<LOGN>;
  static constexpr int F = S::T >= 128 ? 1 : 128 / S::T;
  static constexpr int kThreads = F * S::T;
  static constexpr int kSmem = F * S::PITCH * (int)sizeof(float2);
};

struct RowArgs {
  const float* src;  // transform i: 2 N floats from src + 2 N i (rows 2i and 2i + 1, or row i of pairs)
  float* dst1;       // planar results: row 1 to dst1 + i dst_pitch, row 2 to dst2 + i dst_pitch
  float* dst2;
  float2* dst_pair;  // inverse: interleaved results instead, or nullptr
  int dst_pitch;
  int count;         // transforms
  float scale;
  const float2* tw;  // [N] exp(-i pi k / 2N), [N] exp(-2 pi i k / N)
  double* zero;      // set to 0 by the first thread (the energy that a later pass sums), or nullptr
  const int* gate;
};

// One complex transform per pair of real rows: the DCT of both, or the two
// inverses (IDXST of row 1 / 2 where kSin1 / kSin2) of planar rows or of a row
// of pairs.  Bound by instruction issue and the exchanges at 1024 points.
template <int LOGN, int kMode, bool kSin1, bool kSin2>
__global__ void __launch_bounds__(RowBlock<LOGN>::kThreads) fft_rows_kernel(RowArgs a) {
  using S = FftShape<LOGN>;
  using B = RowBlock<LOGN>;
  extern __shared__ __align__(16) float2 fft_smem[];
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(fft_smem_addr(&bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  grid_dep_sync();
  if (gate_closed(a.gate)) return;
  const int f = threadIdx.x / S::T, t = threadIdx.x % S::T;
  const int first = blockIdx.x * B::F;
  const int here = min(B::F, a.count - first);
  int skip = 0;
  if (threadIdx.x == 0) {
    if (a.zero && blockIdx.x == 0) *a.zero = 0.0;
    skip = g_fft_skip_loads;
    constexpr uint32_t kBytes = 2 * S::N * sizeof(float);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fft_smem_addr(&bar)),
                 "r"(kBytes * here)
                 : "memory");
    for (int i = 0; i < here && !skip; ++i)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              fft_smem_addr(fft_smem + i * S::PITCH)),
          "l"(a.src + (size_t)(first + i) * 2 * S::N), "r"(kBytes), "r"(fft_smem_addr(&bar))
          : "memory");
  }
  __syncthreads();
  if (!__syncthreads_and(fft_try_wait(&bar) || fft_bounded_wait(&bar))) {
    if (threadIdx.x == 0 && !skip) fft_drain(&bar);  // the block lives until its last thread returns
    return;
  }
  float2* s = fft_smem + f * S::PITCH;
  const float2* W = a.tw + S::N;
  const bool live = f < here;  // every thread takes part in the barriers
  const size_t dof = (size_t)(first + f) * a.dst_pitch;
  const float* x1 = reinterpret_cast<const float*>(s);
  const float* x2 = x1 + S::N;
  float2 v[S::E];
  if (kMode == kRowDct) {
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int i = r < S::E / 2 ? 2 * (t + r * S::T) : 2 * S::N - 1 - 2 * (t + r * S::T);  // dct_src
      v[r] = make_float2(x1[i], x2[i]);
    }
    __syncthreads();  // the rows are in registers: the buffer serves the exchanges
    fft_run<LOGN, false>(v, s, W, t);
#pragma unroll
    for (int r = 0; r < S::E; ++r) s[fft_at<LOGN>(t, fft_out_step<LOGN>(r))] = v[r];
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int k = t + r * S::T;
      const float2 X = dct_unpack(s[fft_at<LOGN>(t, r * S::T)], s[fft_pad((S::N - k) & (S::N - 1))], __ldg(a.tw + k));
      a.dst1[dof + k] = X.x * a.scale;
      a.dst2[dof + k] = X.y * a.scale;
    }
  } else {
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int k = t + r * S::T, kn = (S::N - k) & (S::N - 1);
      const float2 ak = kMode == kRowInvPairs ? s[k] : make_float2(x1[k], x2[k]);
      const float2 an = kMode == kRowInvPairs ? s[kn] : make_float2(x1[kn], x2[kn]);
      v[r] = idct_pack<kSin1, kSin2>(k, ak, an, __ldg(a.tw + k));
    }
    __syncthreads();
    fft_run<LOGN, true>(v, s, W, t);
#pragma unroll
    for (int r = 0; r < S::E; ++r) s[fft_at<LOGN>(t, fft_out_step<LOGN>(r))] = v[r];
    __syncthreads();
    if (!live) return;
    const float h = 0.5f * a.scale;
    // outputs u = t + r T: T is even, so u has t's parity; u / 2 and N - 1 - u / 2
    const bool odd = t & 1;
    const float h1 = kSin1 && odd ? -h : h, h2 = kSin2 && odd ? -h : h;
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int u = t + r * S::T;
      const float2 z = s[fft_pad(odd ? S::N - 1 - (u >> 1) : u >> 1)];
      if (a.dst_pair) {
        a.dst_pair[dof + u] = make_float2(z.x * h1, z.y * h2);
      } else {
        a.dst1[dof + u] = z.x * h1;
        a.dst2[dof + u] = z.y * h2;
      }
    }
  }
}

enum { kColDct = 0, kColIdct = 1, kColIdxst = 2, kColSpectral = 3 };

// Column pairs per block.  A block takes 2 F neighbouring columns, transform f
// the columns c0 + f and c0 + F + f: 8 columns are a full 32-byte sector of
// each row read, and 4 neighbouring pairs of the spectral pass's output a full
// sector written.  (4096-point columns two pairs to a block, 512 threads of
// 128 registers instead of 1024 of 64: a solve 315 us instead of 236.)
template <int LOGM>
struct ColBlock {
  using S = FftShape<LOGM>;
  static constexpr int F = 4;
  static constexpr int kThreads = F * S::T;
  static constexpr int kSmem = F * S::PITCH * (int)sizeof(float2);
};

struct ColArgs {
  const float* src;  // [M, N]
  float* dst;        // [M, N]; kColSpectral: [M, N] pairs (x field, y field)
  int N;
  float scale;
  const float2* tw;  // of M
  EpiParams epi;     // kColSpectral: weights (M, N, wv_scale, two_pi_over_m / _n) and energy
  const int* gate;
};

// One column's coefficients a[k] (register r: k = t + r T) through the spectral
// weights and both inverse transforms, Sh_M (a wx) and Ch_M (a wy) sharing one
// complex transform, to pairs in dst.  Returns the column's energy terms
// w_u winv a^2 (w_0 = 1/2) summed over the thread's k.  The buffer must be free.
template <int LOGM>
__device__ __forceinline__ double spectral_column(const ColArgs& a, const float* coef, int col, float2* s,
                                                  const float2* __restrict__ W, int t) {
  using S = FftShape<LOGM>;
  float2 v[S::E];
  double e = 0.0;
#pragma unroll
  for (int r = 0; r < S::E; ++r) {
    const int k = t + r * S::T;
    float wx, wy, winv;
    spectral_weights(a.epi, k, col, wx, wy, winv);
    if (a.epi.energy) {
      const double c = (double)coef[r], wc = (double)winv * c;
      e = fma(k == 0 ? 0.5 * wc : wc, c, e);
    }
    v[r] = make_float2(__fmul_rn(coef[r], wx), __fmul_rn(coef[r], wy));
    s[fft_at<LOGM>(t, r * S::T)] = v[r];
  }
  if (col == 0) e *= 0.5;
  if (!a.dst) return e;  // the energy only (uniform)
  __syncthreads();
#pragma unroll
  for (int r = 0; r < S::E; ++r) {
    const int k = t + r * S::T;  // the mirrored coefficient is another thread's
    v[r] = idct_pack<true, false>(k, v[r], s[fft_pad((S::N - k) & (S::N - 1))], __ldg(a.tw + k));
  }
  __syncthreads();
  fft_run<LOGM, true>(v, s, W, t);
#pragma unroll
  for (int r = 0; r < S::E; ++r) {
    const int n = t + fft_out_step<LOGM>(r);
    const float g = n >= S::N / 2 ? -0.5f : 0.5f;
    reinterpret_cast<float2*>(a.dst)[(size_t)dct_src<LOGM>(n) * a.N + col] = make_float2(v[r].x * g, v[r].y * 0.5f);
  }
  return e;
}

template <int LOGM, int kMode>
__global__ void __launch_bounds__(ColBlock<LOGM>::kThreads) fft_cols_kernel(const __grid_constant__ ColArgs a) {
  grid_dep_sync();
  if (gate_closed(a.gate)) return;
  using S = FftShape<LOGM>;
  constexpr int F = ColBlock<LOGM>::F;
  extern __shared__ __align__(16) float2 fft_smem[];
  const int f = threadIdx.x % F, t = threadIdx.x / F;  // neighbouring threads hold neighbouring columns
  float2* s = fft_smem + f * S::PITCH;
  const float2* W = a.tw + S::N;
  const int c0 = blockIdx.x * 2 * F + f, c1 = c0 + F;  // N is a multiple of 2 F
  float2 v[S::E];
  if (kMode == kColDct || kMode == kColSpectral) {
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const float* row = a.src + (size_t)dct_src<LOGM>(t + r * S::T) * a.N;
      v[r] = make_float2(__ldg(row + c0), __ldg(row + c1));
    }
    fft_run<LOGM, false>(v, s, W, t);
#pragma unroll
    for (int r = 0; r < S::E; ++r) s[fft_at<LOGM>(t, fft_out_step<LOGM>(r))] = v[r];
    __syncthreads();
    float a0[S::E], a1[S::E];
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int k = t + r * S::T;
      const float2 X = dct_unpack(s[fft_at<LOGM>(t, r * S::T)], s[fft_pad((S::N - k) & (S::N - 1))], __ldg(a.tw + k));
      a0[r] = X.x * a.scale;
      a1[r] = X.y * a.scale;
      if (kMode == kColDct) {
        a.dst[(size_t)k * a.N + c0] = a0[r];
        a.dst[(size_t)k * a.N + c1] = a1[r];
      }
    }
    if (kMode == kColDct) return;
    __syncthreads();
    double e = spectral_column<LOGM>(a, a0, c0, s, W, t);
    e += spectral_column<LOGM>(a, a1, c1, s, W, t);
    if (a.epi.energy) {
      // sum_xy rho IDCT2(a winv) = M N sum w_u w_v winv a^2 (spectral_energy)
      e *= (double)a.epi.M * (double)a.epi.N;
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      __syncthreads();  // the buffer is free once every transform is done
      double* red = reinterpret_cast<double*>(fft_smem);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < ColBlock<LOGM>::kThreads / 32; ++w) e += red[w];
        atomicAdd(a.epi.energy, e);
      }
    }
  } else {
    constexpr bool kSin = kMode == kColIdxst;
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int k = t + r * S::T;
      const float* row = a.src + (size_t)k * a.N;
      const float* mir = a.src + (size_t)((S::N - k) & (S::N - 1)) * a.N;
      v[r] = idct_pack<kSin, kSin>(k, make_float2(__ldg(row + c0), __ldg(row + c1)),
                                   make_float2(__ldg(mir + c0), __ldg(mir + c1)), __ldg(a.tw + k));
    }
    fft_run<LOGM, true>(v, s, W, t);
    const float h = 0.5f * a.scale;
#pragma unroll
    for (int r = 0; r < S::E; ++r) {
      const int n = t + fft_out_step<LOGM>(r);
      const float g = kSin && n >= S::N / 2 ? -h : h;
      float* row = a.dst + (size_t)dct_src<LOGM>(n) * a.N;
      row[c0] = v[r].x * g;
      row[c1] = v[r].y * g;
    }
  }
}

int fft_take_status(int* out) {
  int v = 0;
  const int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_fft_status, sizeof(int));
  if (e == cudaSuccess && v) e = cudaMemcpyToSymbol(g_fft_status, &zero, sizeof(int));
  if (v) *out = v;
  return (int)e;
}
int fft_set_wait_budget(long long cycles) { return (int)cudaMemcpyToSymbol(g_fft_wait_budget, &cycles, sizeof(cycles)); }
int fft_set_skip_loads(int skip) { return (int)cudaMemcpyToSymbol(g_fft_skip_loads, &skip, sizeof(skip)); }

static int log2_side(int n) {
  for (int l = kFftMinLog; l <= kFftMaxLog; ++l)
    if (n == (1 << l)) return l;
  return -1;
}

template <int LOGN, int kMode, bool kSin1, bool kSin2>
static int run_rows(const RowArgs& a, cudaStream_t s, const char* who) {
  using B = RowBlock<LOGN>;
  auto kern = fft_rows_kernel<LOGN, kMode, kSin1, kSin2>;
  int rc = opt_in_smem(kern, B::kSmem, who);
  if (rc) return rc;
  launch_kernel(kern, ceil_div(a.count, B::F), B::kThreads, B::kSmem, s, a);
  return check_launch(who);
}

template <int kMode, bool kSin1, bool kSin2>
static int rows(int N, const RowArgs& a, cudaStream_t s, const char* who) {
  switch (log2_side(N)) {
    case 6: return run_rows<6, kMode, kSin1, kSin2>(a, s, who);
    case 7: return run_rows<7, kMode, kSin1, kSin2>(a, s, who);
    case 8: return run_rows<8, kMode, kSin1, kSin2>(a, s, who);
    case 9: return run_rows<9, kMode, kSin1, kSin2>(a, s, who);
    case 10: return run_rows<10, kMode, kSin1, kSin2>(a, s, who);
    case 11: return run_rows<11, kMode, kSin1, kSin2>(a, s, who);
    case 12: return run_rows<12, kMode, kSin1, kSin2>(a, s, who);
  }
  set_error("%s: unsupported side %d", who, N);
  return DP_ERR_UNSUPPORTED;
}

template <int LOGM, int kMode>
static int run_cols(const ColArgs& a, cudaStream_t s, const char* who) {
  using B = ColBlock<LOGM>;
  auto kern = fft_cols_kernel<LOGM, kMode>;
  int rc = opt_in_smem(kern, B::kSmem, who);
  if (rc) return rc;
  launch_kernel(kern, a.N / (2 * B::F), B::kThreads, B::kSmem, s, a);
  return check_launch(who);
}

template <int kMode>
static int cols(int M, const ColArgs& a, cudaStream_t s, const char* who) {
  switch (log2_side(M)) {
    case 6: return run_cols<6, kMode>(a, s, who);
    case 7: return run_cols<7, kMode>(a, s, who);
    case 8: return run_cols<8, kMode>(a, s, who);
    case 9: return run_cols<9, kMode>(a, s, who);
    case 10: return run_cols<10, kMode>(a, s, who);
    case 11: return run_cols<11, kMode>(a, s, who);
    case 12: return run_cols<12, kMode>(a, s, who);
  }
  set_error("%s: unsupported side %d", who, M);
  return DP_ERR_UNSUPPORTED;
}

}  // namespace dpb

using namespace dpb;

extern "C" int dp_fft_supported(int M, int N) { return log2_side(M) > 0 && log2_side(N) > 0 ? 1 : 0; }

extern "C" int dp_fft_twiddles(int n, float* out_host) {
  DP_REQUIRE(log2_side(n) > 0 && out_host, "dp_fft_twiddles: bad arguments (n = %d)", n);
  for (int k = 0; k < n; ++k) {
    out_host[2 * k] = (float)cos(M_PI * k / (2.0 * n));
    out_host[2 * k + 1] = (float)-sin(M_PI * k / (2.0 * n));
    out_host[2 * (n + k)] = (float)cos(2.0 * M_PI * k / n);
    out_host[2 * (n + k) + 1] = (float)-sin(2.0 * M_PI * k / n);
  }
  return DP_OK;
}

// a, b, c: optional maps; the tables and the work map are required
static int require_maps(const char* who, int M, int N, const float* tw_m, const float* tw_n, const void* work,
                        const void* a, const void* b, const void* c) {
  DP_REQUIRE(dp_fft_supported(M, N), "%s: sides must be powers of two in 64 .. 4096, got %d x %d", who, M, N);
  DP_REQUIRE(tw_m && tw_n && work, "%s: null pointer argument", who);
  DP_REQUIRE((((uintptr_t)tw_m | (uintptr_t)tw_n | (uintptr_t)work | (uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0,
             "%s: maps and twiddle tables must be 16-byte aligned", who);
  return DP_OK;
}

extern "C" int dp_transform_fft(int kind, const float* x, int M, int N, const float* tw_m, const float* tw_n,
                                float* work, float* out, dp_stream_t stream) {
  const char* who = "dp_transform_fft";
  int rc = require_maps(who, M, N, tw_m, tw_n, work, x, out, nullptr);
  if (rc) return rc;
  DP_REQUIRE(x && out && work != x && work != out,
             "dp_transform_fft: null map, or work shared with the input or output");
  cudaStream_t s = as_stream(stream);
  RowArgs r;
  memset(&r, 0, sizeof(r));
  r.src = x;
  r.dst1 = work;
  r.dst2 = work + N;
  r.dst_pitch = 2 * N;
  r.count = M / 2;
  r.scale = 1.f;
  r.tw = reinterpret_cast<const float2*>(tw_n);
  r.gate = trial_gate();
  ColArgs c;
  memset(&c, 0, sizeof(c));
  c.src = work;
  c.dst = out;
  c.N = N;
  c.tw = reinterpret_cast<const float2*>(tw_m);
  c.gate = trial_gate();
  switch (kind) {
    case DP_FFT_DCT2:
      c.scale = 4.0f / ((float)M * (float)N);
      rc = rows<kRowDct, false, false>(N, r, s, who);
      return rc ? rc : cols<kColDct>(M, c, s, who);
    case DP_FFT_IDCT2:
      c.scale = 4.f;
      rc = rows<kRowInv, false, false>(N, r, s, who);
      return rc ? rc : cols<kColIdct>(M, c, s, who);
    case DP_FFT_IDCT_IDXST:
      c.scale = 4.f;
      rc = rows<kRowInv, true, true>(N, r, s, who);
      return rc ? rc : cols<kColIdct>(M, c, s, who);
    case DP_FFT_IDXST_IDCT:
      c.scale = 4.f;
      rc = rows<kRowInv, false, false>(N, r, s, who);
      return rc ? rc : cols<kColIdxst>(M, c, s, who);
  }
  set_error("dp_transform_fft: unknown kind %d", kind);
  return DP_ERR_INVALID_ARGUMENT;
}

extern "C" int dp_poisson_fft(const float* rho, int M, int N, float rho_scale, float wv_scale, const float* tw_m,
                              const float* tw_n, float* work, float* ex, float* ey, float* exy, double* energy,
                              int want_energy, dp_stream_t stream) {
  const char* who = "dp_poisson_fft";
  int rc = require_maps(who, M, N, tw_m, tw_n, work, exy, exy ? nullptr : ex, exy ? nullptr : ey);
  if (rc) return rc;
  DP_REQUIRE(rho && energy, "dp_poisson_fft: null pointer argument");
  DP_REQUIRE(exy || (!ex == !ey), "dp_poisson_fft: ex and ey come together");
  DP_REQUIRE(((uintptr_t)rho & 15) == 0, "dp_poisson_fft: rho must be 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  const size_t mn = (size_t)M * N;
  const bool fields = exy || ex;
  RowArgs r;
  memset(&r, 0, sizeof(r));
  r.src = rho;
  r.dst1 = work;
  r.dst2 = work + N;
  r.dst_pitch = 2 * N;
  r.count = M / 2;
  r.scale = rho_scale;
  r.tw = reinterpret_cast<const float2*>(tw_n);
  r.zero = energy;
  r.gate = trial_gate();
  rc = rows<kRowDct, false, false>(N, r, s, who);
  if (rc) return rc;
  ColArgs c;
  memset(&c, 0, sizeof(c));
  c.src = work;
  c.dst = fields ? work + mn : nullptr;
  c.N = N;
  c.scale = (float)(4.0 / ((double)M * (double)N));
  c.tw = reinterpret_cast<const float2*>(tw_m);
  c.epi.M = M;
  c.epi.N = N;
  c.epi.wv_scale = wv_scale;
  c.epi.two_pi_over_m = (float)(2.0 * M_PI / M);
  c.epi.two_pi_over_n = (float)(2.0 * M_PI / N);
  c.epi.energy = want_energy ? energy : nullptr;
  c.gate = trial_gate();
  rc = cols<kColSpectral>(M, c, s, who);
  if (rc || !fields) return rc;
  r.src = work + mn;
  r.dst1 = ex;
  r.dst2 = ey;
  r.dst_pair = reinterpret_cast<float2*>(exy);
  r.dst_pitch = N;
  r.count = M;
  r.scale = 4.f;
  r.zero = nullptr;
  return rows<kRowInvPairs, false, true>(N, r, s, who);
}
