// kernels.cuh -- the interpreter engine's evaluation kernels, the sums of partials,
// the end of a step (step_kernel), exchanges, the two-stage loop, and helper
// kernels (data layout, points, draws layout).
//
// The evaluation body here is the register-stack interpreter (interp.cuh):
// the bytecode is whatever the session compiled, read from the constant bank.
#pragma once
#include "common.cuh"
#include "interp.cuh"

namespace gpum {

// G values per thread: G chains (O = 1), or G/2 chains at two observations of a
// lane at once (O = 2).  Either way a lane's observations are added in the same
// order.
template <int G, int D, int O>
struct InterpBody {
  static constexpr bool kChainLanes = false;
  static constexpr int kObsPerEval = 1;
  static constexpr int kRounds = O;
  static constexpr int kChains = G / O;
  const EvalProg& pg;
  const float* pc0;
  int CG;
  float* hsm;
  float2 s[D][G / 2];  // chain pairs
  Comp acc[kChains];
  __device__ InterpBody(const EvalProg& p, float* h) : pg(p), pc0(nullptr), CG(0), hsm(h) {}
  __device__ __forceinline__ void begin(const float* p0, int cg) {
    pc0 = p0;
    CG = cg;
#pragma unroll
    for (int g = 0; g < kChains; ++g) acc[g].init();
  }
  __device__ __forceinline__ void add(int round) {
#pragma unroll
    for (int h = 0; h < kChains / 2; ++h) {
      acc[2 * h].add(s[0][round * (kChains / 2) + h].x);
      acc[2 * h + 1].add(s[0][round * (kChains / 2) + h].y);
    }
  }
  __device__ __forceinline__ void eval(const float* xo, int T, bool valid) {
    interp_run<G, D, O>(pg, s, xo, 0, T, pc0, CG, hsm);
    if (valid) add(0);
  }
  // The observations at xo and xo + xs.
  __device__ __forceinline__ void eval_rounds(const float* xo, int xs, int T, bool v0, bool v1) {
    interp_run<G, D, O>(pg, s, xo, xs, T, pc0, CG, hsm);
    if (v0) add(0);
    if (v1) add(O - 1);
  }
  __device__ __forceinline__ float last(int g, int round = 0) const {
    const float2 v = s[0][round * (kChains / 2) + (g >> 1)];
    return (g & 1) ? v.y : v.x;
  }
  __device__ __forceinline__ void end() {}
  __device__ __forceinline__ double total(int g, int) const { return acc[g].total(); }
};

// f64 prior interpreted from the source bytecode; its gradient (MALA on the
// interpreter engine) by the reverse-mode tape over chain c's scratch.
struct InterpPrior {
  __device__ static double value(const ChainArgs& A, int, const double* p) {
    return prior_interp(A.prior_code, A.n_prior, A.prior_consts, p);
  }
  __device__ static double value_grad(const ChainArgs& A, int c, const double* p, double* g) {
    const size_t n = (size_t)(A.n_prior > 0 ? A.n_prior : 1);
    double* tv = A.ptape + (size_t)c * 2 * n;
    uint32_t* ti = A.ptape_i + (size_t)c * 2 * n;
    return prior_value_grad_tape(A.prior_code, A.n_prior, A.prior_consts, p, g, tv, tv + n, ti,
                                 ti + n);
  }
};

// The widest variants (sixteen chains per thread over a six-deep stack, eight
// over eight: 96 and 64 stack registers) keep their stacks in registers at one
// CTA per SM; the others fit two.
template <int G, int D, int O = 1>
__global__ void __launch_bounds__(kThreads, (G >= 8 ? 1 : 2))
iter_kernel(const __grid_constant__ EvalProg prog, const __grid_constant__ TmapDesc tmap,
            EvalArgs E, ChainArgs A, int phase) {
  static_assert(kThreads == kInterpThreads, "the operand scratch is laid out per thread");
  __shared__ float hsm[2 * G * kInterpThreads];
  InterpBody<G, D, O> body(prog, hsm + threadIdx.x);
  run_iteration<G / O, 1, InterpBody<G, D, O>, InterpPrior>(&tmap, E, A, phase, body);
}

// ------------------------------------------------------- failure self-test
// The device-failure path end to end: an mbarrier that expects one arrival
// and gets none, polled by every thread at most `polls` times and for at
// most `max_ns` nanoseconds; the wait runs out, thread 0 sets the error word
// the host reads after every run, and the kernel returns (no copy or MMA is
// in flight, nothing hangs).
static __global__ void selftest_wait_kernel(uint32_t* err, uint32_t polls, uint64_t max_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const uint64_t t0 = gm_globaltimer();
  bool done = false;
  for (uint32_t i = 0; i < polls && !done; ++i) {
    done = mbar_try_wait(&bar, 0u);
    if (gm_globaltimer() - t0 > max_ns) break;
  }
  if (__syncthreads_or(done ? 0 : 1) && threadIdx.x == 0) atomicOr(err, DEV_ERR_WAIT_SELFTEST);
}

// ------------------------------------------ gradient in the interpreter engine
// The node program of compile_grad_program (program.hpp) in the constant bank.
struct __align__(16) GradProg {
  uint32_t n_nodes, root, has_root, np;
  uint32_t node[kMaxGradNodes];
  float cst[kMaxConsts];
};

// Value and parameter gradient per observation by a reverse sweep over a tape
// of the observation's node values (cpu_native.rs:148-279 in FP32, with the
// compiled engine's local derivatives: POW's exponent term only where the
// base is positive, LGAMMA's the digamma, an exponent of constant 2 as a
// square).  One chain per thread, lanes over observations (G = 1); the tape
// and the adjoints live in the thread's local memory.  W = 1 + the largest
// parameter count the instantiation serves; entries past np stay 0.
template <int W>
struct InterpGradBody {
  static constexpr bool kChainLanes = false;
  static constexpr int kObsPerEval = 1;
  static constexpr int kRounds = 1;
  static constexpr int kNp = W - 1;
  const GradProg& pg;
  const float* pc0;
  int CG;
  float vals[kMaxGradNodes];
  float adj[kMaxGradNodes];
  float gp[kNp];
  double gpd[kNp];
  double s;
  float part, lastv;
  int cnt;
  __device__ explicit InterpGradBody(const GradProg& p) : pg(p), pc0(nullptr), CG(0) {}

  __device__ __forceinline__ void begin(const float* p0, int cg) {
    pc0 = p0;
    CG = cg;
    for (int j = 0; j < kNp; ++j) {
      gp[j] = 0.0f;
      gpd[j] = 0.0;
    }
    s = 0.0;
    part = 0.0f;
    lastv = 0.0f;
    cnt = 0;
  }
  __device__ __forceinline__ float fetch(uint32_t r, const float* xo, int T) const {
    const uint32_t t = r & 3u, i = r >> 2;
    return t == GREF_NODE ? vals[i]
         : t == GREF_CONST ? pg.cst[i]
         : t == GREF_PARAM ? pc0[(size_t)i * CG]
                           : xo[(size_t)i * T];
  }
  __device__ __forceinline__ void sink(uint32_t r, float x) {
    const uint32_t t = r & 3u, i = r >> 2;
    if (t == GREF_NODE) adj[i] += x;
    else if (t == GREF_PARAM) gp[i] += x;
  }
  __device__ __forceinline__ void flush() {
    s += (double)part;
    part = 0.0f;
    for (uint32_t j = 0; j < pg.np; ++j) {
      gpd[j] += (double)gp[j];
      gp[j] = 0.0f;
    }
    cnt = 0;
  }
  __device__ void eval(const float* xo, int T, bool valid) {
    if (!valid) {  // padding rows add neither value nor gradient
      lastv = 0.0f;
      return;
    }
    const uint32_t n = pg.n_nodes;
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t w = pg.node[i], op = w & 15u;
      const uint32_t ra = (w >> 4) & 0x3FFFu, rb = w >> 18;
      const float a = fetch(ra, xo, T);
      float v;
      if (op == 7) v = -a;
      else if (op == 8) v = expf(a);
      else if (op == 9) v = logf(a);
      else if (op == 10) v = sqrtf(a);
      else if (op == 12) v = lgammaf(a);
      else {
        const float b = fetch(rb, xo, T);
        if (op == 3) v = a + b;
        else if (op == 4) v = a - b;
        else if (op == 5) v = a * b;
        else if (op == 6) v = a / b;
        else v = ((rb & 3u) == GREF_CONST && b == 2.0f) ? a * a : powf(a, b);
      }
      vals[i] = v;
    }
    const float val = pg.has_root ? fetch(pg.root, xo, T) : 0.0f;
    lastv = val;
    part += val;
    if (pg.has_root) {
      if ((pg.root & 3u) == GREF_NODE) {
        for (uint32_t i = 0; i < n; ++i) adj[i] = 0.0f;
        adj[pg.root >> 2] = 1.0f;
        for (int i = (int)n - 1; i >= 0; --i) {
          const float g = adj[i];
          if (g == 0.0f) continue;
          const uint32_t w = pg.node[i], op = w & 15u;
          const uint32_t ra = (w >> 4) & 0x3FFFu, rb = w >> 18;
          const float a = fetch(ra, xo, T), v = vals[i];
          switch (op) {
            case 3: sink(ra, g); sink(rb, g); break;
            case 4: sink(ra, g); sink(rb, -g); break;
            case 5: {
              const float b = fetch(rb, xo, T);
              sink(ra, g * b);
              sink(rb, g * a);
              break;
            }
            case 6: {
              const float b = fetch(rb, xo, T);
              sink(ra, g / b);
              sink(rb, -g * v / b);
              break;
            }
            case 7: sink(ra, -g); break;
            case 8: sink(ra, g * v); break;
            case 9: sink(ra, g / a); break;
            case 10: sink(ra, g * 0.5f / v); break;
            case 12: sink(ra, g * gm_digammaf(a)); break;
            default: {
              const float b = fetch(rb, xo, T);
              if ((rb & 3u) == GREF_CONST && b == 2.0f) {
                sink(ra, g * 2.0f * a);
              } else {
                sink(ra, g * b * powf(a, b - 1.0f));
                sink(rb, a > 0.0f ? g * v * logf(a) : 0.0f);
              }
              break;
            }
          }
        }
      } else if ((pg.root & 3u) == GREF_PARAM) {
        gp[pg.root >> 2] += 1.0f;
      }
    }
    if (++cnt == 8) flush();
  }
  __device__ __forceinline__ float last(int) const { return lastv; }
  __device__ __forceinline__ void end() { flush(); }
  __device__ __forceinline__ double total(int, int w) const {
    if (w == 0) return s + (double)part;
    return w - 1 < (int)pg.np ? gpd[w - 1] : 0.0;
  }
};

template <int W>
__global__ void __launch_bounds__(kThreads, 1)
iter_kernel_grad(const __grid_constant__ GradProg prog, const __grid_constant__ TmapDesc tmap,
                 EvalArgs E, ChainArgs A, int phase) {
  InterpGradBody<W> body(prog);
  run_iteration<1, W, InterpGradBody<W>, InterpPrior>(&tmap, E, A, phase, body);
}

// -------------------------------------------------------------- MALA helpers
// out = f * (1/2) M g, M = Ls Ls' (or diag sd^2), the whitened drift capped at
// 2 sqrt(d) (MALTA; cpu_native.rs:617-651).
__device__ inline void half_m_times(int np, const double* sd, const double* L, const double* g,
                                    double* out, double* tmp) {
  const double dmax = 2.0 * sqrt((double)np);
  if (!L) {
    for (int j = 0; j < np; ++j) tmp[j] = 0.5 * sd[j] * g[j];
  } else {
    for (int j = 0; j < np; ++j) {
      double acc = 0.0;
      for (int k = j; k < np; ++k) acc += L[(size_t)k * np + j] * g[k];
      tmp[j] = 0.5 * acc;
    }
  }
  double ss = 0.0;
  for (int j = 0; j < np; ++j) ss += tmp[j] * tmp[j];
  const double norm = sqrt(ss);
  const double f = norm > dmax ? dmax / norm : 1.0;
  if (!L) {
    for (int j = 0; j < np; ++j) out[j] = f * sd[j] * tmp[j];
  } else {
    for (int k = 0; k < np; ++k) {
      double acc = 0.0;
      for (int j = 0; j <= k; ++j) acc += L[(size_t)k * np + j] * tmp[j];
      out[k] = f * acc;
    }
  }
}

// -1/2 |Ls^{-1}(v - m)|^2 by forward substitution (cpu_native.rs:655-673).
__device__ inline double log_q(int np, const double* sd, const double* L, const double* v,
                               const double* m, double* tmp) {
  double q = 0.0;
  if (!L) {
    for (int j = 0; j < np; ++j) {
      const double r = (v[j] - m[j]) / sd[j];
      q -= 0.5 * r * r;
    }
  } else {
    for (int k = 0; k < np; ++k) {
      double acc = v[k] - m[k];
      for (int j = 0; j < k; ++j) acc -= L[(size_t)k * np + j] * tmp[j];
      tmp[k] = acc / L[(size_t)k * np + k];
      q -= 0.5 * tmp[k] * tmp[k];
    }
  }
  return q;
}

// ------------------------------------------------------------- proposals
// Next proposal of chain c into prop (f64) and params (f32).
// Diagonal RWM chain_kernel.rs:212-223 / cpu_native.rs:726-735; Cholesky
// RWM :224-249 / :736-753; DE on the frozen snapshot :250-295 / :754-784;
// MALA :681-703 (mean from the cached gradient, then L z or sd * z).
__device__ inline void propose(const ChainArgs& A, int c, Stream& rs, float* params, int C_pad) {
  const int np = A.np;
  const double* x = A.state + (size_t)c * np;
  double* y = A.prop + (size_t)c * np;
  const double* sd = A.sd + (size_t)c * np;
  const double* L = A.L ? A.L + (size_t)c * np * np : nullptr;
  if (A.mode == MODE_RWM) {
    for (int j = 0; j < np; ++j) y[j] = x[j] + sd[j] * rs.normal();
  } else if (A.mode == MODE_CHOL || A.mode == MODE_MALA) {
    double* z = A.zbuf + (size_t)c * np;
    const double* base = x;
    if (A.mode == MODE_MALA) {
      double* mx = A.mx + (size_t)c * np;
      half_m_times(np, sd, L, A.gx + (size_t)c * np, mx, A.vbuf + (size_t)c * np);
      for (int j = 0; j < np; ++j) mx[j] += x[j];
      base = mx;
    }
    for (int j = 0; j < np; ++j) z[j] = rs.normal();
    if (L) {
      for (int k = 0; k < np; ++k) {
        double acc = base[k];
        for (int j = 0; j <= k; ++j) acc += L[(size_t)k * np + j] * z[j];
        y[k] = acc;
      }
    } else {
      for (int j = 0; j < np; ++j) y[j] = base[j] + sd[j] * z[j];
    }
  } else {
    const int n = A.n_chains;
    int a = (int)(rs.next() * (double)n);
    if (a >= n) a = n - 1;
    int b = (int)(rs.next() * (double)n);
    if (b >= n) b = n - 1;
    if (b == a) b = (b + 1) % n;
    const double g = rs.next() < 0.1 ? 1.0 : A.gamma;
    const double* pa = A.snap + (size_t)a * np;
    const double* pb = A.snap + (size_t)b * np;
    for (int j = 0; j < np; ++j) {
      const double z = rs.normal();
      const double diff = pa[j] - pb[j];
      y[j] = x[j] + g * diff + A.de_noise * sd[j] * z;
    }
  }
  for (int j = 0; j < np; ++j) params[(size_t)j * C_pad + c] = (float)y[j];
}

// Synchronous per-generation DE (path B, cpu_native.rs:400-506): the
// difference vector comes from the current population, so this runs in its
// own kernel after every chain's previous accept.  Partners a != c and
// b != c, a (cpu_native.rs:430-440); g = 1 with probability 0.1, else gamma.
__device__ inline void propose_desync(const ChainArgs& A, int c, Stream& rs, float* params,
                                      int C_pad) {
  const int n = A.n_chains, np = A.np;
  int a = (int)(rs.next() * (double)n);
  if (a >= n) a = n - 1;
  if (a == c) a = (a + 1) % n;
  int b = (int)(rs.next() * (double)n);
  if (b >= n) b = n - 1;
  while (b == c || b == a) b = (b + 1) % n;  // n >= 3 is checked by the host
  const double g = rs.next() < 0.1 ? 1.0 : A.gamma;
  const double* x = A.state + (size_t)c * np;
  const double* pa = A.state + (size_t)a * np;
  const double* pb = A.state + (size_t)b * np;
  const double* sd = A.sd + (size_t)c * np;
  double* y = A.prop + (size_t)c * np;
  for (int j = 0; j < np; ++j) {
    const double z = rs.normal();
    y[j] = x[j] + g * (pa[j] - pb[j]) + A.de_noise * sd[j] * z;
    params[(size_t)j * C_pad + c] = (float)y[j];
  }
}

// ------------------------------------------------- one chain, one warp
__device__ __forceinline__ double warp_sum64(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// half_m_times by the lanes of a warp, added to `at`: out = at + f (1/2) M g.
// L has leading dimension ldL (shared or global memory); tmp: np doubles of
// shared memory.
__device__ __forceinline__ void half_m_warp(int np, const double* sd, const double* L, int ldL,
                                            const double* g, const double* at, double* out,
                                            double* tmp, int lane) {
  double ss = 0.0;
  for (int j = lane; j < np; j += 32) {
    double v;
    if (!L) {
      v = 0.5 * sd[j] * g[j];
    } else {
      double acc = 0.0;
      for (int k = j; k < np; ++k) acc += L[(size_t)k * ldL + j] * g[k];
      v = 0.5 * acc;
    }
    tmp[j] = v;
    ss += v * v;
  }
  const double norm = sqrt(warp_sum64(ss)), dmax = 2.0 * sqrt((double)np);
  const double f = norm > dmax ? dmax / norm : 1.0;
  __syncwarp();
  for (int k = lane; k < np; k += 32) {
    double v;
    if (!L) {
      v = f * sd[k] * tmp[k];
    } else {
      double acc = 0.0;
      for (int j = 0; j <= k; ++j) acc += L[(size_t)k * ldL + j] * tmp[j];
      v = f * acc;
    }
    out[k] = v + at[k];
  }
  __syncwarp();
}

// log_q(x | mx') - log_q(y | my'), the MALA proposal ratio, by the lanes of a
// warp: r1 = x - my and r2 = y - mx through one forward substitution, column
// by column (each row subtracts its terms in the serial order), so its serial
// chain is np divisions long instead of np^2 products.  r1, r2: np doubles of
// shared memory each.
__device__ __forceinline__ double log_q_ratio_warp(int np, const double* sd, const double* L,
                                                   int ldL, const double* x, const double* my,
                                                   const double* y, const double* mx, double* r1,
                                                   double* r2, int lane) {
  double q = 0.0;
  if (!L) {
    for (int j = lane; j < np; j += 32) {
      const double a = (x[j] - my[j]) / sd[j], b = (y[j] - mx[j]) / sd[j];
      q += 0.5 * b * b - 0.5 * a * a;
    }
    return warp_sum64(q);
  }
  for (int j = lane; j < np; j += 32) {
    r1[j] = x[j] - my[j];
    r2[j] = y[j] - mx[j];
  }
  __syncwarp();
  for (int j = 0; j < np; ++j) {
    const double d = L[(size_t)j * ldL + j];
    const double t1 = r1[j] / d, t2 = r2[j] / d;
    for (int k = j + 1 + lane; k < np; k += 32) {
      const double l = L[(size_t)k * ldL + j];
      r1[k] -= l * t1;
      r2[k] -= l * t2;
    }
    q += 0.5 * t2 * t2 - 0.5 * t1 * t1;
    __syncwarp();
  }
  return q;
}

// propose() for chain c by the 32 lanes of a warp: the same draws, one
// coordinate per lane.  L: the chain's factor with leading dimension ldL
// (global or staged in shared memory), or nullptr; `sm` is this warp's
// scratch of 2 np doubles.  Returns the stream advanced past the draws.
__device__ inline Stream propose_warp(const ChainArgs& A, int c, Stream rs, float* params,
                                      int C_pad, int lane, double* sm, const double* L, int ldL) {
  const int np = A.np;
  const double* x = A.state + (size_t)c * np;
  double* y = A.prop + (size_t)c * np;
  const double* sd = A.sd + (size_t)c * np;
  uint32_t used = 2u * (uint32_t)np;
  float* out = params + c;
  if (A.mode == MODE_CHOL || A.mode == MODE_MALA) {
    double* z = sm;
    const double* base = x;
    if (A.mode == MODE_MALA) {  // mean = x + f (1/2) M g (cpu_native.rs:617-651)
      double* mx = A.mx + (size_t)c * np;
      half_m_warp(np, sd, L, ldL, A.gx + (size_t)c * np, x, mx, z, lane);
      base = mx;
    }
    for (int j = lane; j < np; j += 32) z[j] = stream_normal_at(rs, 0, j);
    __syncwarp();
    for (int k = lane; k < np; k += 32) {
      double v;
      if (L) {
        v = base[k];
        for (int j = 0; j <= k; ++j) v += L[(size_t)k * ldL + j] * z[j];
      } else {
        v = base[k] + sd[k] * z[k];
      }
      y[k] = v;
      out[(size_t)k * C_pad] = (float)v;
    }
  } else {
    const double *pa = x, *pb = x;
    double g = 0.0, noise = 1.0;
    uint32_t i0 = 0;
    if (A.mode == MODE_DE) {  // the pair of the snapshot
      const int n = A.n_chains;
      int a = (int)(stream_at(rs, 1) * (double)n);
      if (a >= n) a = n - 1;
      int b = (int)(stream_at(rs, 2) * (double)n);
      if (b >= n) b = n - 1;
      if (b == a) b = (b + 1) % n;
      g = stream_at(rs, 3) < 0.1 ? 1.0 : A.gamma;
      pa = A.snap + (size_t)a * np;
      pb = A.snap + (size_t)b * np;
      noise = A.de_noise;
      i0 = 3;
    }
    for (int j = lane; j < np; j += 32) {
      const double z = stream_normal_at(rs, i0, j);
      const double v = i0 ? x[j] + g * (pa[j] - pb[j]) + noise * sd[j] * z : x[j] + sd[j] * z;
      y[j] = v;
      out[(size_t)j * C_pad] = (float)v;
    }
    used += i0;
  }
  __syncwarp();
  if (rs.kind == RNG_TRIPLE32) rs.ctr += used;
  else rs.k += used;
  return rs;
}

// ------------------------------------------------------------ partial sums
// The sums over the observation blocks of chain c's first W of Ws values,
// partials [nob][C_pad][Ws], by the `wpc` warps of a group (wi: this warp's
// number in it); red: [wpc][W] doubles of shared memory.  With one value the
// threads take the blocks, with several the lanes take the values (coalesced)
// and the warps the blocks, up to 16 values 32 / W blocks at a time: a gradient
// call of 250 points x 300,001 observations x 1 parameter (two values, 1,172
// blocks) took 90 us with a block per warp at a time, 60 so.
__device__ __forceinline__ void group_partials(const double* __restrict__ partials, int nob,
                                               int C_pad, int Ws, int W, int c, int wi,
                                               int wpc, double* red, int lane) {
  if (W == 1) {
    double v = 0.0;
#pragma unroll 4
    for (int o = wi * 32 + lane; o < nob; o += 32 * wpc)
      v += __ldcg(&partials[((size_t)o * C_pad + c) * Ws]);
    v = warp_sum64(v);
    if (lane == 0) red[wi] = v;
  } else if (W <= 16) {  // 32 / W observation blocks at a time
    const int per = 32 / W, w = lane % W, j = lane / W;
    const double* p = partials + (size_t)c * Ws + w;
    const size_t st = (size_t)C_pad * Ws;
    double v = 0.0;
    if (j < per) {
#pragma unroll 8
      for (int o = wi * per + j; o < nob; o += per * wpc) v += __ldcg(&p[(size_t)o * st]);
    }
    double t = v;
    for (int i = 1; i < per; ++i) t += __shfl_sync(0xffffffffu, v, (lane + i * W) & 31);
    if (lane < W) red[(size_t)wi * W + lane] = t;
  } else {
    for (int w = lane; w < W; w += 32) {
      const double* p = partials + (size_t)c * Ws + w;
      const size_t st = (size_t)C_pad * Ws;
      double v = 0.0;
#pragma unroll 8
      for (int o = wi; o < nob; o += wpc) v += __ldcg(&p[(size_t)o * st]);
      red[(size_t)wi * W + w] = v;
    }
  }
}
__device__ __forceinline__ double group_total(const double* red, int W, int w, int wpc) {
  double v = red[w];
  for (int i = 1; i < wpc; ++i) v += red[(size_t)i * W + w];
  return v;
}

// Sums of each point's values w0 .. W - 1 into out[point][W - w0]: one group of
// wpc warps per point.  A single thread per value over all observation blocks
// took 25 us for 250 points of 18 values.
// out and err_out may be pinned host memory; err_out, when given, receives
// the session's device error word.
static __global__ void __launch_bounds__(kThreads)
reduce_partials_kernel(const double* __restrict__ partials, double* __restrict__ out, int nob,
                       int C_pad, int Ws, int n, int W, int w0, int wpc,
                       const uint32_t* __restrict__ err, uint32_t* __restrict__ err_out) {
  extern __shared__ double rsm[];  // [8][W]
  pdl_wait();
  if (err_out && blockIdx.x == 0 && threadIdx.x == 0) *err_out = __ldcg(err);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wi = warp % wpc, c = (int)blockIdx.x * (kWarps / wpc) + warp / wpc;
  double* red = rsm + (size_t)(warp / wpc) * wpc * W;
  if (c < n) group_partials(partials, nob, C_pad, Ws, W, c, wi, wpc, red, lane);
  __syncthreads();
  if (wi != 0 || c >= n) return;
  for (int w = w0 + lane; w < W; w += 32)
    out[(size_t)c * (W - w0) + w - w0] = group_total(red, W, w, wpc);
}

// ------------------------------------------------------------- a step's end
// What a Metropolis step does after the evaluation of its proposals: the
// partial sums added up, the f64 prior, the accept decision on the f64 totals
// (MALA with the proposal ratio), the draw, the next proposal.  `wpc` warps per
// chain: all of them add the chain's partials, the first one does the rest, a
// coordinate per lane; the step's draws come from the evaluation's side rows or
// are made first.
//
// It is bound by latency (dependent loads, with MALA np steps of the
// substitution), not by any rate.  Run by one thread per chain in the last CTA
// of each chain block it took 30 us at 1,024 chains x 17 parameters, 144 us at
// 2,048 x 65 (DE) and 620 us at 2,048 x 24 (MALA with a factor) of every
// iteration, on at most a few SMs.  Up to 32 parameters lane j keeps coordinate
// j in registers, loaded while the partials are; MALA's factor is staged in
// shared memory before the wait for the evaluation, when it fits.
// Per iteration: 8 Gaussian chains on 20,000 observations 10.0 us with the
// last-CTA end, 6.2 with this kernel drawing for itself, 4.5 with the side
// rows' draws; MALA with a factor, 2,048 x 24 on 256 observations, 620 us to 78.
struct StepArgs {
  const double* partials;    // [nob][C_pad][Ws], W values of each used
  int nob, C_pad, Ws, W;
  const double* prior;       // [C], or nullptr: no prior
  const double* prior_grad;  // [C][np] (MALA), or nullptr
  const double* lu;          // [C] logs of the acceptance uniforms
  const double* z;           // [C][np] normals of the next proposal, or nullptr:
                             // all three drawn here
  const double* inc;         // [C][np] L z, or DE differences
  float* params;             // [np][C_pad] evaluation points of the next step
  int phase;                 // PH_INIT or PH_STEP
  int wpc;                   // warps per chain: 1, 2, 4 or 8
  int wpb;                   // warps per block
  int stage_L;               // 1: factors staged in shared memory
};
// Doubles of shared memory per chain: partial sums, 4 np scratch (the factor's
// leading dimension is odd, so a column of it spreads over the banks).
__host__ __device__ inline int step_ld(int np) { return np | 1; }
__host__ __device__ inline size_t step_smem_doubles(int np, int W, int wpc, bool stage_L) {
  return (size_t)wpc * W + 4 * (size_t)np + (stage_L ? (size_t)np * step_ld(np) : 0);
}

// The next proposal's coordinate from its mean: RWM and diagonal MALA mean + sd
// z, with a factor mean + L z, DE (x + g (x_a - x_b)) + noise sd z.
__device__ __forceinline__ double next_point(const ChainArgs& A, double mean, double sd, double z,
                                             double inc) {
  if (A.L) return mean + inc;
  if (A.mode == MODE_DE) return (mean + inc) + (A.de_noise * sd) * z;
  return mean + sd * z;
}
// Draws of a step from the triple32 counter: the uniform and the proposal's.
__device__ __forceinline__ uint32_t draws_used(const ChainArgs& A, bool step, bool more) {
  return (step ? 1u : 0u) +
         (more ? 2u * (uint32_t)A.np + (A.mode == MODE_DE ? 3u : 0u) : 0u);
}

// The draws of chain c's step by its first warp: the log of the acceptance
// uniform, and into z and inc (np doubles of shared memory each) the next
// proposal's normals and L z or the DE differences.
__device__ __forceinline__ double draw_warp(const ChainArgs& A, int c, bool step, uint32_t t,
                                            const double* L, int ldL, double* z, double* inc,
                                            int lane) {
  const int np = A.np;
  const double lu = step ? log(stream_at(accept_stream(A, c, t), 1u)) : 0.0;
  if (A.mode == MODE_DESYNC || (step ? t + 1 : 0u) >= A.n_iter) return lu;
  const Stream rs = propose_stream(A, c, step, t);
  const bool de = A.mode == MODE_DE;
  for (int j = lane; j < np; j += 32) {
    z[j] = stream_normal_at(rs, de ? 3u : 0u, j);
    if (de) inc[j] = de_difference(A, rs, j);
  }
  __syncwarp();
  if (L)
    for (int k = lane; k < np; k += 32) {
      double acc = 0.0;
      for (int j = 0; j <= k; ++j) acc += L[(size_t)k * ldL + j] * z[j];
      inc[k] = acc;
    }
  __syncwarp();
  return lu;
}

// The drift at `at` for up to 32 parameters, this lane's coordinate of the mean
// at + f (1/2) M g (M = L L' or diag sd^2, the whitened drift capped at 2
// sqrt(np): MALTA; cpu_native.rs:617-651).  sg, st: np doubles of shared memory.
__device__ __forceinline__ double mean_lane(int np, double sd, const double* L, int ldL, double g,
                                            double at, double* sg, double* st, int lane) {
  const bool on = lane < np;
  if (on) sg[lane] = g;
  __syncwarp();
  double v = 0.0;
  if (on) {
    if (!L) {
      v = 0.5 * sd * g;
    } else {
      for (int k = lane; k < np; ++k) v += L[(size_t)k * ldL + lane] * sg[k];
      v *= 0.5;
    }
    st[lane] = v;
  }
  const double norm = sqrt(warp_sum64(v * v)), dmax = 2.0 * sqrt((double)np);
  const double f = norm > dmax ? dmax / norm : 1.0;
  __syncwarp();
  double d = 0.0;
  if (on) {
    if (!L) {
      d = f * sd * v;
    } else {
      for (int j = 0; j <= lane; ++j) d += L[(size_t)lane * ldL + j] * st[j];
      d *= f;
    }
  }
  return d + at;
}

// A chain's state as lane `lane` of its first warp holds it, np <= 32.
struct LaneState {
  double x, y, sd, mx, z, inc, cur, temp, prior, lu;
  uint32_t t, ctr;
};
__device__ __forceinline__ LaneState load_lane(const ChainArgs& A, const StepArgs& S, int c,
                                               int lane) {
  const size_t o = (size_t)c * A.np + lane;
  const bool on = lane < A.np, step = S.phase == PH_STEP;
  LaneState P;
  P.t = A.iter[c];
  P.ctr = A.ctr[c];
  P.temp = A.temp[c];
  P.cur = step ? A.cur[c] : 0.0;
  P.lu = step && S.z ? S.lu[c] : 0.0;
  P.prior = S.prior ? S.prior[c] : 0.0;
  P.x = on ? A.state[o] : 0.0;
  P.y = on && step ? A.prop[o] : 0.0;
  P.sd = on ? A.sd[o] : 1.0;
  P.z = on && S.z ? S.z[o] : 0.0;
  P.inc = on && S.inc ? S.inc[o] : 0.0;
  P.mx = on && step && A.mode == MODE_MALA ? A.mx[o] : 0.0;
  return P;
}

__device__ __forceinline__ void finish_lane(const ChainArgs& A, const StepArgs& S, int c,
                                            int lane, const double* L, int ldL,
                                            const LaneState& P, const double* red, double* sg,
                                            double* st) {
  const int np = A.np;
  const size_t o = (size_t)c * np + lane;
  const bool on = lane < np, step = S.phase == PH_STEP, mala = A.mode == MODE_MALA;
  const double b = A.beta ? A.beta[c] : 1.0;  // likelihood power
  const double ll = group_total(red, S.W, 0, S.wpc);
  const double lp = (A.beta ? b * ll : ll) + P.prior;
  double g = 0.0, mean = 0.0;
  if (mala) {
    if (on) {
      g = b * group_total(red, S.W, 1 + lane, S.wpc);
      if (S.prior_grad) g += S.prior_grad[o];
    }
    mean = mean_lane(np, P.sd, L, ldL, g, step ? P.y : P.x, sg, st, lane);
  }
  bool take = true;  // the start: the mean is the state's
  double xn = P.x;
  if (step) {
    double lqd = 0.0;
    if (mala) {
      // q(x | y) - q(y | x) with the truncated drift at y (cpu_native.rs:704-710):
      // both residuals through one forward substitution, column by column
      double r1 = P.x - mean, r2 = P.y - P.mx;
      if (!L) {
        const double u1 = r1 / P.sd, u2 = r2 / P.sd;
        lqd = warp_sum64(on ? 0.5 * u2 * u2 - 0.5 * u1 * u1 : 0.0);
      } else {
        for (int j = 0; j < np; ++j) {
          const double d = L[(size_t)j * ldL + j];
          const double t1 = __shfl_sync(0xffffffffu, r1, j) / d;
          const double t2 = __shfl_sync(0xffffffffu, r2, j) / d;
          if (on && lane > j) {
            const double l = L[(size_t)lane * ldL + j];
            r1 -= l * t1;
            r2 -= l * t2;
          }
          lqd += 0.5 * t2 * t2 - 0.5 * t1 * t1;
        }
      }
    }
    // Tempered acceptance on the f64 totals (chain_kernel.rs:334,
    // cpu_native.rs:792); MALA adds the proposal ratio and requires a
    // finite proposal log density (cpu_native.rs:713-714).
    take = mala ? (isfinite(lp) && P.lu < (lp - P.cur) / P.temp + lqd)
                : (P.lu < (lp - P.cur) / P.temp);
    if (take) xn = P.y;
  }
  const bool more = A.mode != MODE_DESYNC && (step ? P.t + 1 : 0u) < A.n_iter;
  if (more && on) {
    // a rejected proposal leaves the state, and with it its drift, as it was
    const double y = next_point(A, mala ? (take ? mean : P.mx) : xn, P.sd, P.z, P.inc);
    S.params[(size_t)lane * S.C_pad + c] = (float)y;
    A.prop[o] = y;
  }
  if (step && on) {
    if (take) A.state[o] = xn;
    if (P.t < A.n_iter) A.draws[((size_t)P.t * np + lane) * S.C_pad + c] = (float)xn;
  }
  if (step && A.rec_ll) {
    const uint64_t slot = A.rec_base + (uint64_t)P.t * A.n_chains + c;
    if (slot < A.rec_cap) {
      if (on) A.rec_theta[slot * np + lane] = (float)P.y;
      if (lane == 0) A.rec_ll[slot] = ll;
    }
  }
  if (mala && take && on) {
    A.gx[o] = g;  // a replica exchange moves it with the state
    A.mx[o] = mean;
  }
  if (lane == 0) {
    A.last_eval[c] = lp;
    if (take) A.cur[c] = lp;
    if (step) {
      if (take) A.accepts[c] += 1;
      A.iter[c] = P.t + 1;
    }
    A.ctr[c] = P.ctr + (A.rng == RNG_TRIPLE32 ? draws_used(A, step, more) : 0u);
  }
}

// The same for any number of parameters, lane j taking j, j + 32, ...
__device__ inline void finish_wide(const ChainArgs& A, const StepArgs& S, int c, int lane,
                                   const double* L, int ldL, double lu, const double* z,
                                   const double* inc, const double* red, double* tmp) {
  const int np = A.np;
  const size_t o = (size_t)c * np;
  const bool step = S.phase == PH_STEP, mala = A.mode == MODE_MALA;
  double* x = A.state + o;
  double* y = A.prop + o;
  const double* sd = A.sd + o;
  const uint32_t t = A.iter[c];
  const double b = A.beta ? A.beta[c] : 1.0;  // likelihood power
  const double ll = group_total(red, S.W, 0, S.wpc);
  const double lp = (A.beta ? b * ll : ll) + (S.prior ? S.prior[c] : 0.0);
  double* gy = mala ? A.gy + o : nullptr;
  double* my = mala ? A.my + o : nullptr;
  if (mala) {
    for (int j = lane; j < np; j += 32) {
      const double v = b * group_total(red, S.W, 1 + j, S.wpc);
      gy[j] = S.prior_grad ? v + S.prior_grad[o + j] : v;
    }
    __syncwarp();
    half_m_warp(np, sd, L, ldL, gy, step ? y : x, my, tmp, lane);
  }
  bool take = true;  // the start: the mean is the state's
  if (step) {
    const double lqd =
        mala ? log_q_ratio_warp(np, sd, L, ldL, x, my, y, A.mx + o, tmp, tmp + np, lane) : 0.0;
    const double cur = A.cur[c], temp = A.temp[c];
    take = mala ? (isfinite(lp) && lu < (lp - cur) / temp + lqd) : (lu < (lp - cur) / temp);
  }
  const bool more = A.mode != MODE_DESYNC && (step ? t + 1 : 0u) < A.n_iter;
  const uint64_t slot = A.rec_base + (uint64_t)t * A.n_chains + c;
  const bool rec = step && A.rec_ll && slot < A.rec_cap;
  for (int j = lane; j < np; j += 32) {
    const double yj = step ? y[j] : 0.0;
    const double xn = step && take ? yj : x[j];
    if (step) {
      if (take) x[j] = xn;
      if (t < A.n_iter) A.draws[((size_t)t * np + j) * S.C_pad + c] = (float)xn;
      if (rec) A.rec_theta[slot * np + j] = (float)yj;
    }
    if (mala && take) {
      A.gx[o + j] = gy[j];
      A.mx[o + j] = my[j];
    }
    if (more) {
      const double v =
          next_point(A, mala ? (take ? my[j] : A.mx[o + j]) : xn, sd[j], z[j], inc[j]);
      y[j] = v;
      S.params[(size_t)j * S.C_pad + c] = (float)v;
    }
  }
  if (lane == 0) {
    A.last_eval[c] = lp;
    if (take) A.cur[c] = lp;
    if (rec) A.rec_ll[slot] = ll;
    if (step) {
      if (take) A.accepts[c] += 1;
      A.iter[c] = t + 1;
    }
    if (A.rng == RNG_TRIPLE32) A.ctr[c] += draws_used(A, step, more);
  }
}

// kDraw: the step's draws are made here (many chains: 80 registers, three CTAs
// per SM), else by the side rows (few: no spills on the way of each iteration).
template <bool kDraw>
static __global__ void __launch_bounds__(kThreads, kDraw ? 3 : 2)
step_kernel(ChainArgs A, StepArgs S) {
  extern __shared__ double ssm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpc = S.wpc, wi = warp % wpc, grp = warp / wpc;
  const int c = (int)blockIdx.x * (S.wpb / wpc) + grp;
  const int np = A.np;
  double* red = ssm + (size_t)grp * step_smem_doubles(np, S.W, wpc, S.stage_L != 0);
  double* tmp = red + (size_t)wpc * S.W;  // [4][np]
  const bool live = c < A.n_chains;
  const double* L = A.L && live ? A.L + (size_t)c * np * np : nullptr;
  int ldL = np;
  if (L && S.stage_L) {  // set by the host before the run: no wait needed
    double* Ls = tmp + 4 * np;
    ldL = step_ld(np);
    for (int i = wi * 32 + lane; i < np * np; i += 32 * wpc)
      Ls[(i / np) * ldL + i % np] = L[i];
    L = Ls;
  }
  load_vars(A);  // as the factors
  pdl_wait();
  pdl_trigger();
  LaneState P;
  const bool narrow = np <= 32, step = S.phase == PH_STEP, first = wi == 0 && live;
  if (narrow && first) P = load_lane(A, S, c, lane);
  double lu = 0.0;
  const double *z = tmp + 2 * np, *inc = tmp + 3 * np;
  if constexpr (kDraw) {
    // The factors are staged.  A.L, not L: groups past the last chain have none,
    // and every warp of the block takes the same barriers.
    if (A.L && S.stage_L) __syncthreads();
    if (first) lu = draw_warp(A, c, step, A.iter[c], L, ldL, tmp + 2 * np, tmp + 3 * np, lane);
  } else if (first && !narrow) {
    const size_t o = (size_t)c * np;
    lu = S.lu[c];
    z = S.z + o;
    inc = S.inc ? S.inc + o : z;  // unused without differences
  }
  if (live) group_partials(S.partials, S.nob, S.C_pad, S.Ws, S.W, c, wi, wpc, red, lane);
  __syncthreads();
  if (!first) return;
  if (narrow) {
    if constexpr (kDraw) {
      P.lu = lu;
      P.z = lane < np ? z[lane] : 0.0;
      P.inc = lane < np ? inc[lane] : 0.0;
    }
    finish_lane(A, S, c, lane, L, ldL, P, red, tmp, tmp + np);
  } else {
    finish_wide(A, S, c, lane, L, ldL, lu, z, inc, red, tmp);
  }
}

// ------------------------------------------------------------- helpers
// Row-major f64 rows [r0, r0+nr) -> column-major f32 [ncols][ld].
static __global__ void convert_rows_kernel(const double* __restrict__ src, float* __restrict__ dst,
                                    int ncols, int64_t ld, int64_t r0, int64_t nr) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nr * ncols) return;
  const int64_t r = i / ncols, j = i % ncols;
  dst[(int64_t)j * ld + r0 + r] = (float)src[i];
}

// f64 chain-major points [C][np] -> f32 [np][C_pad]; pad chains copy chain 0.
// pts may be pinned host memory.
static __global__ void points_to_params_kernel(const double* __restrict__ pts,
                                        float* __restrict__ params, int n, int np, int C_pad) {
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np * C_pad) return;
  const int j = i / C_pad, c = i % C_pad;
  const int src = c < n ? c : 0;
  params[i] = (float)pts[(size_t)src * np + j];
}

// The start of a run in one launch: states, DE snapshot, proposal scales,
// temperatures, evaluation points, counters and the run's values.  init, sd
// and temp may be pinned host memory or the state arrays themselves.
struct RunInit {
  const double *init, *sd, *temp;
  RunVars vars;
  RunVars* d_vars;
  uint32_t *pt_att, *pt_acc, *pt_n;  // or nullptr
};
static __global__ void run_init_kernel(ChainArgs A, RunInit R, float* __restrict__ params,
                                       double* snap, double* sd, double* temp, int C_pad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int np = A.np;
  if (i >= np * C_pad) return;
  const int j = i / C_pad, c = i % C_pad;
  const bool live = c < A.n_chains;
  const double x = R.init[(size_t)(live ? c : 0) * np + j];
  params[i] = (float)x;
  if (!live) return;
  const size_t o = (size_t)c * np + j;
  const double s = R.sd[o];
  A.state[o] = x;
  snap[o] = x;
  sd[o] = s;
  if (j != 0) return;
  temp[c] = R.temp[c];
  A.ctr[c] = 0;
  A.accepts[c] = 0;
  A.iter[c] = 0;
  if (R.pt_att) {
    R.pt_att[c] = 0;
    R.pt_acc[c] = 0;
  }
  if (c == 0) {
    *R.d_vars = R.vars;
    if (R.pt_n) R.pt_n[0] = 0;
  }
}

// Internal draws [n_iter][np][C_pad] -> the reference layout, column-major
// (n_iter, C, np): out[t + n_iter*(c + C*j)] (chain_kernel.rs:345).
static __global__ void draws_layout_kernel(const float* __restrict__ in, float* __restrict__ out,
                                    int n_iter, int np, int C, int C_pad) {
  __shared__ float tile[32][33];
  const int j = blockIdx.z;
  const int c0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int t = t0 + r, c = c0 + threadIdx.x;
    if (t < n_iter && c < C) tile[r][threadIdx.x] = in[((size_t)t * np + j) * C_pad + c];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int c = c0 + r, t = t0 + threadIdx.x;
    if (t < n_iter && c < C)
      out[(size_t)t + (size_t)n_iter * ((size_t)c + (size_t)C * j)] = tile[threadIdx.x][r];
  }
}

}  // namespace gpum

// ===================================================== delayed acceptance
// Two-stage Metropolis-Hastings (Christen & Fox 2005) with the surrogate
// log-likelihood s() as stage 1 and the exact log-likelihood l() as stage 2:
//   stage 1: accept y with min(1, exp([s(y)+p(y) - s(x)-p(x)] / T) q(x|y)/q(y|x))
//   stage 2: accept with min(1, exp([(l(y)-l(x)) - (s(y)-s(x))] / T))
// (p = prior, which cancels in stage 2, as does the proposal ratio: the
// stage-1 acceptance of the reverse move carries its inverse).  The product
// of the two acceptance probabilities satisfies detailed balance for the
// exact tempered posterior, so the target is unchanged; only stage-1
// survivors are evaluated exactly.  The proposal is the random walk, DE, or
// a Langevin move whose drift is the surrogate log-posterior gradient (so no
// exact gradient is ever needed).
namespace gpum {

// ------------------------------------------------- draw moments (adaptation)
// Moments of the draws of iterations [t0, t0 + n) in the internal layout
// [n_iter][np][C_pad], all in f64 and in a fixed order: per chain and
// parameter the mean and the sum of squared deviations (two passes), the
// pooled mean per parameter, and the pooled sums of cross deviations.
static __global__ void moments_chain_kernel(const float* __restrict__ draws, int np, int C,
                                            int C_pad, int t0, int n, double* __restrict__ mean,
                                            double* __restrict__ m2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np * C) return;
  const int j = i / C, c = i % C;  // consecutive threads: consecutive chains
  double sm = 0.0;
  for (int t = 0; t < n; ++t) sm += (double)draws[((size_t)(t0 + t) * np + j) * C_pad + c];
  const double mu = sm / n;
  double q = 0.0;
  for (int t = 0; t < n; ++t) {
    const double dv = (double)draws[((size_t)(t0 + t) * np + j) * C_pad + c] - mu;
    q += dv * dv;
  }
  mean[(size_t)c * np + j] = mu;
  m2[(size_t)c * np + j] = q;
}

// One block per parameter: pooled mean of the n x C values (fixed-order
// strided sums, then a fixed shared-memory tree).
static __global__ void moments_pool_mean_kernel(const float* __restrict__ draws, int np, int C,
                                                int C_pad, int t0, int n,
                                                double* __restrict__ pmean) {
  __shared__ double red[256];
  const int j = blockIdx.x;
  const size_t total = (size_t)n * C;
  double sm = 0.0;
  for (size_t k = threadIdx.x; k < total; k += blockDim.x) {
    const size_t t = k / C, c = k % C;
    sm += (double)draws[((t0 + t) * np + j) * C_pad + c];
  }
  red[threadIdx.x] = sm;
  __syncthreads();
  for (int off = 128; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) pmean[j] = red[0] / (double)total;
}

// One block per (j, k >= j): pooled sum of (x_j - m_j)(x_k - m_k).
static __global__ void moments_pool_m2_kernel(const float* __restrict__ draws, int np, int C,
                                              int C_pad, int t0, int n,
                                              const double* __restrict__ pmean,
                                              double* __restrict__ pm2) {
  __shared__ double red[256];
  const int j = blockIdx.x / np, k = blockIdx.x % np;
  if (k < j) return;  // uniform per block
  const size_t total = (size_t)n * C;
  const double mj = pmean[j], mk = pmean[k];
  double sm = 0.0;
  for (size_t q = threadIdx.x; q < total; q += blockDim.x) {
    const size_t t = q / C, c = q % C;
    const double a = (double)draws[((t0 + t) * np + j) * C_pad + c] - mj;
    const double b = (double)draws[((t0 + t) * np + k) * C_pad + c] - mk;
    sm += a * b;
  }
  red[threadIdx.x] = sm;
  __syncthreads();
  for (int off = 128; off > 0; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    pm2[(size_t)j * np + k] = red[0];
    pm2[(size_t)k * np + j] = red[0];
  }
}

// ------------------------------------------------------ parallel tempering
// Replica exchange on the device (the reference swaps on the host between
// batches, R/adaptive.R:272-413): after every `every`-th iteration, the
// adjacent pairs (i, i + 1) of each ladder -- contiguous groups of K chains
// with the temperatures along the group -- of one parity (alternating from
// exchange to exchange, starting with the even pairs) exchange states with
// probability min(1, exp(delta)), delta = (lp[i+1] - lp[i]) (1/T[i] - 1/T[i+1])
// on the untempered log posteriors.  The proposals already drawn for the
// next iteration were centred on the old states, so both chains of an
// exchanged pair draw new ones.  Uniforms: Philox keyed by (seed, exchange,
// pair).  One thread per pair; the pairs of one parity are disjoint.
struct PtArgs {
  int K;               // ladder length
  int every;           // iterations between exchanges
  const uint32_t* iter;  // [1] iterations done (the step's or the DA loop's counter)
  double* sll_x;       // [C] delayed acceptance: surrogate value at the state, or null
  double* prior_x;     // [C] delayed acceptance: prior at the state, or null
  uint32_t* n_swaps;   // [1] exchanges done
  uint32_t* att;       // [C] attempts of pair (c, c + 1)
  uint32_t* acc;       // [C] accepted exchanges of pair (c, c + 1)
  float* params;       // [np][C_pad] evaluation points of the next iteration
  int C_pad;
};

static __global__ void pt_exchange_kernel(ChainArgs A, PtArgs P) {
  load_vars(A);
  const uint32_t t = P.iter[0];  // iterations done (all chain blocks agree here)
  if (t == 0 || t % (uint32_t)P.every != 0 || t >= A.n_iter) return;
  const uint32_t s = t / (uint32_t)P.every;  // exchange number, from 1
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int C = A.n_chains, np = A.np;
  if (i == 0) P.n_swaps[0] = s;
  if (i + 1 >= C || (i % P.K) == P.K - 1) return;     // not a pair of one ladder
  if (((i % P.K) & 1) != (int)((s + 1) & 1)) return;  // odd exchanges: even pairs
  const double lpa = A.cur[i], lpb = A.cur[i + 1];
  const double delta = (lpb - lpa) * (1.0 / A.temp[i] - 1.0 / A.temp[i + 1]);
  const U4 r = philox4x32_10(U4{(uint32_t)i, s, 0x50545357u, 0u}, A.seed, 0x3C6EF372u);
  const double u = u53(r.x, r.y);
  P.att[i] += 1;
  if (!(isfinite(delta) && log(u) < delta)) return;
  P.acc[i] += 1;
  double* xa = A.state + (size_t)i * np;
  double* xb = A.state + (size_t)(i + 1) * np;
  for (int j = 0; j < np; ++j) {
    const double tmp = xa[j];
    xa[j] = xb[j];
    xb[j] = tmp;
  }
  A.cur[i] = lpb;
  A.cur[i + 1] = lpa;
  if (P.sll_x) {  // the two-stage loop's cached values follow their states
    const double s0 = P.sll_x[i], p0 = P.prior_x[i];
    P.sll_x[i] = P.sll_x[i + 1];
    P.prior_x[i] = P.prior_x[i + 1];
    P.sll_x[i + 1] = s0;
    P.prior_x[i + 1] = p0;
  }
  if (A.mode == MODE_MALA) {  // the cached gradients belong to the states
    double* ga = A.gx + (size_t)i * np;
    double* gb = A.gx + (size_t)(i + 1) * np;
    for (int j = 0; j < np; ++j) {
      const double tmp = ga[j];
      ga[j] = gb[j];
      gb[j] = tmp;
    }
  }
  for (int c = i; c <= i + 1; ++c) {
    Stream rs = make_stream(A, c);
    rs.it = t;
    rs.k = 0x40000000u;  // counters apart from the iteration's own proposal
    propose(A, c, rs, P.params, P.C_pad);
    A.ctr[c] = rs.ctr;
  }
}

// Path-B DE proposals of generation A.iter[0] for every chain (one thread per
// chain), between the previous generation's accepts and this generation's
// evaluation.  All chain blocks have the same iteration count here.
static __global__ void desync_propose_kernel(ChainArgs A, float* params, int C_pad) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= A.n_chains) return;
  load_vars(A);
  const uint32_t t = A.iter[0];
  if (t >= A.n_iter) return;
  Stream rs = make_stream(A, c);
  rs.it = t;
  rs.k = 0;
  propose_desync(A, c, rs, params, C_pad);
  A.ctr[c] = rs.ctr;
}

struct DaArgs {
  double* sll_x;     // [C] surrogate log-likelihood at the state
  double* sll_y;     // [C] surrogate log-likelihood at the proposal
  double* prior_x;   // [C] prior at the state
  double* prior_y;   // [C] prior at the proposal
  uint32_t* flag;    // [C] stage 1 accepted this iteration
  uint32_t* slot;    // [C] position in the compacted evaluation
  uint32_t* active;  // [1] stage-1 acceptances this iteration
  uint32_t* stage1;  // [C] stage-1 acceptance counts
  float* params;     // [np][C_pad] compacted evaluation points
  float* full;       // [np][C_pad] scratch for propose()
  int C_pad;
  // Langevin proposal (MALA): the surrogate's data-term gradient at the
  // proposals (at the states during set-up), and the prior tape's scratch
  double* gs;        // [C][np]
  double* tvals;     // [C][n_prior]
  double* tadj;      // [C][n_prior]
  uint32_t* tlhs;    // [C][n_prior]
  uint32_t* trhs;    // [C][n_prior]
  // 1: the compiled engine's prior kernel has already written prior_x (set-up)
  // or prior_y (each iteration) and, with the Langevin proposal, added the
  // prior's gradient into gs; 0: the kernels interpret the prior themselves
  int prior_ready;
};

// Surrogate log-posterior gradient at theta: the surrogate's data-term
// gradient gs plus the f64 prior's gradient (tape); returns the prior.
__device__ __forceinline__ double da_post_grad(const ChainArgs& A, const DaArgs& D, int c,
                                               const double* theta, const double* gs,
                                               double* g) {
  const int np = A.np, n = A.n_prior;
  for (int j = 0; j < np; ++j) g[j] = gs[j];
  const size_t o = (size_t)c * (size_t)(n > 0 ? n : 1);
  return prior_value_grad_tape(A.prior_code, n, A.prior_consts, theta, g, D.tvals + o,
                               D.tadj + o, D.tlhs + o, D.trhs + o);
}

__device__ __forceinline__ double da_uniform(Stream& rs, uint32_t t, uint32_t k) {
  if (rs.kind == RNG_TRIPLE32) return rs.next();
  rs.it = t;
  rs.k = k;
  return rs.next();
}

// After the exact start (PH_INIT): the prior at each state, zero counters.
// With the Langevin proposal (A.mode == MODE_MALA; the start ran with a
// symmetric mode) also the surrogate log-posterior gradient at each state
// (D.gs holds the surrogate's data-term gradient there), and every chain
// draws its first proposal again, now with that drift.
static __global__ void da_setup_kernel(ChainArgs A, DaArgs D) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= A.n_chains) return;
  const double* x = A.state + (size_t)c * A.np;
  if (A.mode == MODE_MALA) {
    if (D.prior_ready) {
      for (int j = 0; j < A.np; ++j) A.gx[(size_t)c * A.np + j] = D.gs[(size_t)c * A.np + j];
    } else {
      D.prior_x[c] =
          da_post_grad(A, D, c, x, D.gs + (size_t)c * A.np, A.gx + (size_t)c * A.np);
    }
    if (A.n_iter > 0) {
      Stream rs = make_stream(A, c);
      rs.it = 0;
      rs.k = 0x20000000u;  // counters apart from the start's own proposal
      propose(A, c, rs, D.full, D.C_pad);
      A.ctr[c] = rs.ctr;
    }
  } else if (!D.prior_ready) {
    D.prior_x[c] = InterpPrior::value(A, c, x);
  }
  D.stage1[c] = 0;
}

// Stage 1 on the surrogate.  With the Langevin proposal the ratio carries
// q(x | y) / q(y | x) of the surrogate-driven drift (the reverse drift from
// the surrogate log-posterior gradient at y, capped as the forward one;
// cpu_native.rs:704-710 for the exact-gradient form), and the surrogate
// log posterior at y must be finite (cpu_native.rs:713-714).
static __global__ void da_stage1_kernel(ChainArgs A, DaArgs D) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= A.n_chains) return;
  const uint32_t t = A.iter[c];
  const int np = A.np;
  const double* y = A.prop + (size_t)c * np;
  double py, lqd = 0.0;
  if (A.mode == MODE_MALA) {
    double* gy = A.gy + (size_t)c * np;
    if (D.prior_ready) {
      py = D.prior_y[c];
      for (int j = 0; j < np; ++j) gy[j] = D.gs[(size_t)c * np + j];
    } else {
      py = da_post_grad(A, D, c, y, D.gs + (size_t)c * np, gy);
    }
    const double* sd = A.sd + (size_t)c * np;
    const double* L = A.L ? A.L + (size_t)c * np * np : nullptr;
    double* my = A.my + (size_t)c * np;
    double* tmp = A.vbuf + (size_t)c * np;
    half_m_times(np, sd, L, gy, my, tmp);
    for (int j = 0; j < np; ++j) my[j] += y[j];
    lqd = log_q(np, sd, L, A.state + (size_t)c * np, my, tmp) -
          log_q(np, sd, L, y, A.mx + (size_t)c * np, tmp);
  } else {
    py = D.prior_ready ? D.prior_y[c] : InterpPrior::value(A, c, y);
  }
  D.prior_y[c] = py;
  Stream rs = make_stream(A, c);
  const double u = da_uniform(rs, t, 0xFFFF0001u);
  const double a1 = ((D.sll_y[c] + py) - (D.sll_x[c] + D.prior_x[c])) / A.temp[c] + lqd;
  const bool finite = A.mode != MODE_MALA || isfinite(D.sll_y[c] + py);
  D.flag[c] = (finite && log(u) < a1) ? 1u : 0u;
  A.ctr[c] = rs.ctr;
}

// Deterministic compaction: one block scans the flags in chain order.
static __global__ void da_compact_kernel(ChainArgs A, DaArgs D) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < A.n_chains; base += blockDim.x) {
    const int c = base + tid;
    const uint32_t f = c < A.n_chains ? D.flag[c] : 0u;
    uint32_t incl = f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int nw = blockDim.x >> 5;
      uint32_t ws = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, ws, off);
        if (lane >= off) ws += v;
      }
      if (lane < nw) warp_sums[lane] = ws;  // inclusive warp prefix
    }
    __syncthreads();
    const uint32_t before = carry + (warp > 0 ? warp_sums[warp - 1] : 0u) + incl - f;
    if (c < A.n_chains) D.slot[c] = before;
    __syncthreads();
    if (tid == blockDim.x - 1) carry += warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
  }
  if (tid == 0) D.active[0] = carry;
}

// Stage-1 survivors' proposals into the compacted f32 evaluation array.
static __global__ void da_pack_kernel(ChainArgs A, DaArgs D) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)A.n_chains * A.np) return;
  const int c = (int)(i / A.np), j = (int)(i % A.np);
  if (!D.flag[c]) return;
  D.params[(size_t)j * D.C_pad + D.slot[c]] = (float)A.prop[i];
}

// Stage 1, the compaction and the packing in one block, for a symmetric
// proposal whose priors are ready (prior_y): up to kScreenChains chains, two a
// thread.  Apart they were three launches of 3.7, 2.0 and 1.8 us and the gaps
// between them, each too short to fill the GPU.
constexpr int kScreenThreads = 1024, kScreenChains = 2 * kScreenThreads;
static __global__ void __launch_bounds__(kScreenThreads) da_screen_kernel(ChainArgs A, DaArgs D) {
  __shared__ uint32_t sums[2][32];
  __shared__ uint16_t who[kScreenChains];  // slot -> chain
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();
  uint32_t f[2], below[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = i * kScreenThreads + tid;
    f[i] = 0;
    if (c < A.n_chains) {
      Stream rs = make_stream(A, c);
      const double u = da_uniform(rs, A.iter[c], 0xFFFF0001u);
      const double a1 =
          ((D.sll_y[c] + D.prior_y[c]) - (D.sll_x[c] + D.prior_x[c])) / A.temp[c];
      f[i] = log(u) < a1 ? 1u : 0u;
      D.flag[c] = f[i];
      A.ctr[c] = rs.ctr;
    }
    const uint32_t b = __ballot_sync(0xffffffffu, f[i] != 0);
    below[i] = __popc(b & ((1u << lane) - 1u));
    if (lane == 0) sums[i][warp] = __popc(b);
  }
  __syncthreads();
  // survivors before each warp, in chain order
  if (warp < 2) {
    uint32_t v = sums[warp][lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += x;
    }
    sums[warp][lane] = v;  // inclusive
  }
  __syncthreads();
  const uint32_t first = sums[0][31], live = first + sums[1][31];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = i * kScreenThreads + tid;
    if (!f[i]) continue;
    const uint32_t k = (i ? first : 0u) + (warp > 0 ? sums[i][warp - 1] : 0u) + below[i];
    D.slot[c] = k;
    who[k] = (uint16_t)c;
  }
  if (tid == 0) D.active[0] = live;
  __syncthreads();
  for (uint32_t i = tid; i < live * (uint32_t)A.np; i += kScreenThreads) {
    const uint32_t k = i % live, j = i / live;
    D.params[(size_t)j * D.C_pad + k] = (float)A.prop[(size_t)who[k] * A.np + j];
  }
}

// Stage 2 for the survivors, the draw for every chain, the next proposal.
// One warp per chain: the lanes add the chain's observation-block partials in
// a fixed lane-strided order and a fixed shuffle tree (deterministic), lane 0
// takes the decision, and the lanes copy, record and propose in parallel.
static __global__ void da_finalize_kernel(ChainArgs A, DaArgs D,
                                          const double* __restrict__ partials,
                                          int CG, int total, int ntiles, int C_pad_eval) {
  const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  pdl_wait();
  pdl_trigger();
  if (c >= A.n_chains) return;
  const bool live = D.flag[c] != 0;
  double ll = 0.0;
  if (live) {
    int tpc = 0;
    const int nob = da_obs_blocks((int)D.active[0], CG, total, ntiles, &tpc);
    const uint32_t k = D.slot[c];
    for (int o = lane; o < nob; o += 32) ll += partials[(size_t)o * C_pad_eval + k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, off);
  }
  extern __shared__ double fin_sm[];  // [warps per block][2 np]
  const int np = A.np;
  const uint32_t t = A.iter[c];
  double* x = A.state + (size_t)c * np;
  const double* y = A.prop + (size_t)c * np;
  Stream rs = make_stream(A, c);
  int take = 0;
  if (live) {
    if (lane == 0) {
      const double plp = ll + D.prior_y[c];
      A.last_eval[c] = plp;
      const double u = da_uniform(rs, t, 0xFFFF0002u);
      const double llx = A.cur[c] - D.prior_x[c];
      const double a2 = ((ll - llx) - (D.sll_y[c] - D.sll_x[c])) / A.temp[c];
      take = log(u) < a2 ? 1 : 0;
      if (take) {
        A.cur[c] = plp;
        D.sll_x[c] = D.sll_y[c];
        D.prior_x[c] = D.prior_y[c];
        A.accepts[c] += 1;
      }
      D.stage1[c] += 1;
    } else if (rs.kind == RNG_TRIPLE32) {
      rs.ctr += 1;  // the stage-2 uniform lane 0 drew
    }
    take = __shfl_sync(0xffffffffu, take, 0);
    if (take) {
      for (int j = lane; j < np; j += 32) x[j] = y[j];
      if (A.mode == MODE_MALA) {  // the drift of the new state
        double* gx = A.gx + (size_t)c * np;
        const double* gy = A.gy + (size_t)c * np;
        for (int j = lane; j < np; j += 32) gx[j] = gy[j];
      }
    }
    __syncwarp();
  }
  if (t < A.n_iter)
    for (int j = lane; j < np; j += 32) A.draws[((size_t)t * np + j) * D.C_pad + c] = (float)x[j];
  __syncwarp();
  if (t + 1 < A.n_iter) {
    rs.it = t + 1;
    rs.k = 0;
    rs = propose_warp(A, c, rs, D.full, D.C_pad, lane, fin_sm + (size_t)(threadIdx.x >> 5) * 2 * np,
                      A.L ? A.L + (size_t)c * np * np : nullptr, np);
  }
  if (lane == 0) {
    A.ctr[c] = rs.ctr;
    A.iter[c] = t + 1;
  }
}

}  // namespace gpum
