// common.cuh -- the per-iteration kernel skeleton shared by the interpreter
// and the compiled (NVRTC) evaluation bodies, plus the accept/propose logic.
//
// One launch evaluates one Metropolis iteration's proposals of every chain (the
// reference runs a whole chain inside one CTA, src/rust/src/chain_kernel.rs
// :123-357; here the data sum of every chain is spread over the whole GPU):
//   grid.x = chain blocks of CG chains, grid.y = observation blocks;
//   each CTA streams its observation tiles through shared memory with TMA
//   (double-buffered, mbarrier completion, bounded waits) and evaluates its
//   CG chains on every observation, so one tile read serves CG chains;
//   per-thread compensated FP32 sums -> FP64 warp-shuffle tree -> FP64 sum
//   over warps in fixed order -> FP64 partial per (obs block, chain, value);
//   side rows of CTAs compute the chains' f64 priors and draws meanwhile; the
//   step kernel (kernels.cuh, step_kernel) then adds the partials up, makes the
//   tempered f64 accept decision, records the draw and draws the next proposal.
// Results are deterministic for a given launch geometry.
#pragma once
#include "device.cuh"

namespace gpum {

constexpr int kWarps = 8;  // warps per CTA
constexpr int kThreads = kWarps * 32;
// The tensor-core value kernel (gm_iter_value_tc): 128 chains per CTA (the
// MMA's M); its epilogue warps (a multiple of four, GenModel::tc_warps) and
// one control warp.
constexpr int kTcM = 128;
constexpr int kMaxStackF64 = 32;

enum Phase : int { PH_EVAL = 0, PH_INIT = 1, PH_STEP = 2, PH_POINTWISE = 3 };
enum RngKind : int { RNG_TRIPLE32 = 0, RNG_PHILOX = 1 };
enum ModeKind : int { MODE_RWM = 0, MODE_DE = 1, MODE_CHOL = 2, MODE_MALA = 3, MODE_DESYNC = 4 };

// What differs from one prepared run of a session to the next while its
// buffers and sizes stay: kept in device memory, so that the captured graph of
// the iterations serves every batch of an adaptive warmup (capturing,
// instantiating and destroying one took 0.4 ms per batch).
struct RunVars {
  uint32_t n_iter, seed;
  double gamma, de_noise;
  uint64_t rec_base;
  float* draws;
};

// Chain state of a run, all device pointers.
struct ChainArgs {
  int n_chains, np;
  double* state;        // [C][np]
  double* prop;         // [C][np]
  double* cur;          // [C]   current log posterior (untempered)
  double* last_eval;    // [C]   log posterior of the latest evaluated point
  uint32_t* ctr;        // [C]   triple32 counters
  uint32_t* accepts;    // [C]
  uint32_t* iter;       // [C]   iterations done
  const double* sd;     // [C][np]
  const double* temp;   // [C]
  const double* L;      // [C][np][np] row-major lower factors, or nullptr
  const double* snap;   // [C][np] DE pool snapshot (batch start states)
  float* draws;         // [n_iter][np][C_pad] internal layout
  uint32_t n_iter;
  uint32_t seed;
  int mode;             // ModeKind
  int rng;              // RngKind
  double gamma, de_noise;
  const uint32_t* prior_code;   // f64-interpreted prior (validated)
  const double* prior_consts;
  int n_prior;
  double* zbuf;         // [C][np] scratch: normals
  // MALA (mode 3)
  double* gx;           // [C][np] gradient of the log posterior at `state`
  double* gy;           // [C][np] gradient at `prop`
  double* mx;           // [C][np] proposal mean from `state`
  double* my;           // [C][np] proposal mean from `prop`
  double* vbuf;         // [C][np] scratch
  // Training pairs for the surrogate: every exactly evaluated proposal's
  // (theta, data-term log-likelihood), slot rec_base + t*C + c (< rec_cap).
  float* rec_theta;     // [rec_cap][np] or nullptr
  double* rec_ll;       // [rec_cap]
  uint64_t rec_base, rec_cap;
  // Power posteriors (thermodynamic integration): chain c targets
  // beta[c] * loglik + prior; nullptr means beta = 1.
  const double* beta;
  // The interpreted prior's gradient (MALA on the interpreter engine): per
  // chain a tape of n_prior values, adjoints and operand indices.
  double* ptape;        // [C][2][n_prior]
  uint32_t* ptape_i;    // [C][2][n_prior]
  const RunVars* vars;  // n_iter, seed, gamma, de_noise, rec_base and draws of the run
};

struct EvalArgs {
  int n_obs, ncols, T, ntiles, tiles_per_cta, CG, WC, C_pad, np;
  int U;                // tiles per stage (stage_tiles)
  int width;            // values per (chain, obs block): 1, or 1 + np with the gradient
  const float* params;  // [np][C_pad] evaluation points (f32)
  double* partials;     // [NOB][C_pad][width]
  float* pointwise;     // [C][n_obs] (PH_POINTWISE)
  int n_points;         // chains/points that are real (rest padding)
  uint32_t* err;        // device error word
  const uint32_t* active;  // if set: only the first *active points are live
  // A sampler step's side rows (side_block; 0: not a step): the points [C][np]
  // of the priors, or nullptr without a prior; the values [C] and, for MALA,
  // the gradients [C][np]; the logs of the acceptance uniforms [C], normals
  // [C][np], and L z or the DE differences [C][np], or nullptr (the step
  // kernel draws)
  int side_rows;
  const double* prior_pts;
  double* prior_out;
  double* prior_grad;
  double* side_lu;
  double* side_z;
  double* side_inc;
};

// Delayed acceptance evaluates the first `live` points of the compacted array
// with a fixed 1-D grid of `total` CTAs, whose split into chain blocks x
// observation blocks is decided on the device from `live`, so the GPU stays
// full whatever stage 1 accepted.  Returns the observation blocks used (0 if
// nothing is live) and the tiles per CTA.
__host__ __device__ inline int da_obs_blocks(int live, int CG, int total, int ntiles, int* tpc) {
  const int busy = (live + CG - 1) / CG;
  if (busy <= 0) {
    *tpc = 0;
    return 0;
  }
  if (ntiles <= 0) {
    *tpc = 0;
    return 1;
  }
  int nob = total / busy;
  nob = nob < 1 ? 1 : (nob > ntiles ? ntiles : nob);
  *tpc = (ntiles + nob - 1) / nob;
  return (ntiles + *tpc - 1) / *tpc;
}

// ------------------------------------------------------ f64 prior, interpreted
// The prior is a handful of ops once per chain per iteration; it is
// interpreted in f64 from the source bytecode (semantics of
// src/rust/src/cpu_native.rs:80-107) so the prior term carries no f32 error.
__device__ inline double prior_interp(const uint32_t* __restrict__ code, int n,
                                      const double* __restrict__ cst,
                                      const double* __restrict__ p) {
  if (n == 0) return 0.0;
  double st[kMaxStackF64];
  int sp = 0;
  for (int pc = 0; pc < n; ++pc) {
    const uint32_t op = code[2 * pc], a = code[2 * pc + 1];
    switch (op) {
      case 0: st[sp++] = cst[a]; break;
      case 1: st[sp++] = p[a]; break;
      case 2: st[sp++] = 0.0; break;  // rejected by validation
      case 3: st[sp - 2] += st[sp - 1]; --sp; break;
      case 4: st[sp - 2] -= st[sp - 1]; --sp; break;
      case 5: st[sp - 2] *= st[sp - 1]; --sp; break;
      case 6: st[sp - 2] /= st[sp - 1]; --sp; break;
      case 7: st[sp - 1] = -st[sp - 1]; break;
      case 8: st[sp - 1] = exp(st[sp - 1]); break;
      case 9: st[sp - 1] = log(st[sp - 1]); break;
      case 10: st[sp - 1] = sqrt(st[sp - 1]); break;
      case 12: st[sp - 1] = lgamma(st[sp - 1]); break;
      // x^2 squared exactly: the correctly rounded x*x, which is what the
      // host libm's pow returns for an exponent of 2
      default: {
        const double a = st[sp - 2], b = st[sp - 1];
        st[sp - 2] = b == 2.0 ? a * a : pow(a, b);
        --sp;
        break;
      }
    }
  }
  return st[0];
}

// Value and gradient of the f64 prior by a reverse-mode tape over its
// bytecode (the reference's tape AD, cpu_native.rs:148-279, for a program
// that reads no data): forward pass recording each instruction's value and
// operands, then adjoints in reverse order with the reference's local
// derivatives (POW's exponent term only where the base is positive; LGAMMA's
// derivative the digamma).  The gradient is added into g.  vals/adj/lhs/rhs
// are this chain's scratch of n entries each.  Used by delayed acceptance
// with the Langevin proposal, whose drift needs the prior's gradient in
// either evaluation engine.
__device__ inline double prior_value_grad_tape(const uint32_t* __restrict__ code, int n,
                                               const double* __restrict__ cst,
                                               const double* __restrict__ p, double* g,
                                               double* vals, double* adj, uint32_t* lhs,
                                               uint32_t* rhs) {
  if (n == 0) return 0.0;
  uint32_t ist[kMaxStackF64];
  int sp = 0;
  for (int pc = 0; pc < n; ++pc) {
    const uint32_t op = code[2 * pc], a = code[2 * pc + 1];
    if (op <= 2) {
      vals[pc] = op == 0 ? cst[a] : (op == 1 ? p[a] : 0.0);
      lhs[pc] = 0xFFFFFFFFu;
      ist[sp++] = (uint32_t)pc;
    } else if ((op >= 7 && op <= 10) || op == 12) {
      const uint32_t l = ist[sp - 1];
      const double x = vals[l];
      vals[pc] = op == 7 ? -x : op == 8 ? exp(x) : op == 9 ? log(x) : op == 10 ? sqrt(x)
                                                                                  : lgamma(x);
      lhs[pc] = l;
      rhs[pc] = 0xFFFFFFFFu;
      ist[sp - 1] = (uint32_t)pc;
    } else {
      const uint32_t r = ist[sp - 1], l = ist[sp - 2];
      const double a0 = vals[l], b0 = vals[r];
      vals[pc] = op == 3 ? a0 + b0 : op == 4 ? a0 - b0 : op == 5 ? a0 * b0 : op == 6 ? a0 / b0
                                                      : (b0 == 2.0 ? a0 * a0 : pow(a0, b0));
      lhs[pc] = l;
      rhs[pc] = r;
      ist[sp - 2] = (uint32_t)pc;
      --sp;
    }
  }
  const int root = n - 1;
  for (int i = 0; i < n; ++i) adj[i] = 0.0;
  adj[root] = 1.0;
  for (int k = n - 1; k >= 0; --k) {
    const double gk = adj[k];
    if (gk == 0.0) continue;
    const uint32_t op = code[2 * k], arg = code[2 * k + 1];
    const uint32_t l = lhs[k], r = rhs[k];
    switch (op) {
      case 0: case 2: break;
      case 1: g[arg] += gk; break;
      case 3: adj[l] += gk; adj[r] += gk; break;
      case 4: adj[l] += gk; adj[r] -= gk; break;
      case 5: adj[l] += gk * vals[r]; adj[r] += gk * vals[l]; break;
      case 6:
        adj[l] += gk / vals[r];
        adj[r] -= gk * vals[k] / vals[r];
        break;
      case 7: adj[l] -= gk; break;
      case 8: adj[l] += gk * vals[k]; break;
      case 9: adj[l] += gk / vals[l]; break;
      case 10: adj[l] += gk * 0.5 / vals[k]; break;
      case 12: adj[l] += gk * gm_digamma(vals[l]); break;
      default: {
        const double a0 = vals[l], b0 = vals[r];
        adj[l] += gk * b0 * pow(a0, b0 - 1.0);
        if (a0 > 0.0) adj[r] += gk * vals[k] * log(a0);
        break;
      }
    }
  }
  return vals[ist[0]];  // stack slot 0, as the value interpreter returns
}

// ------------------------------------------------------- uniform streams
struct Stream {
  int kind;
  uint32_t seedmix;             // triple32: hash(seed) + chain * 2654435761
  uint32_t ctr;                 // triple32 counter
  uint32_t seed, chain, it, k;  // philox counter fields
  __device__ __forceinline__ double next() {
    if (kind == RNG_TRIPLE32) {
      ctr += 1;
      return t32_uniform(seedmix, ctr);
    }
    const U4 r = philox4x32_10(U4{k++, it, chain, 0xB2000001u}, seed, 0x6A09E667u);
    return u53(r.x, r.y);
  }
  __device__ __forceinline__ double normal() {
    const double u1 = next();
    const double u2 = next();
    return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
  }
};

__device__ __forceinline__ Stream make_stream(const ChainArgs& A, int c) {
  Stream rs;
  rs.kind = A.rng;
  rs.seedmix = triple32(A.seed) + (uint32_t)c * 2654435761u;
  rs.ctr = A.ctr[c];
  rs.seed = A.seed;
  rs.chain = (uint32_t)c;
  rs.it = 0;
  rs.k = 0;
  return rs;
}

// The run's own values into a kernel's argument block.
__device__ __forceinline__ void load_vars(ChainArgs& A) {
  const RunVars v = *A.vars;
  A.n_iter = v.n_iter;
  A.seed = v.seed;
  A.gamma = v.gamma;
  A.de_noise = v.de_noise;
  A.rec_base = v.rec_base;
  A.draws = v.draws;
}

// The i-th uniform (i >= 1) a chain's stream `rs` would return from its
// current position, without advancing it: both streams are counter-based, so
// a chain's draws can be made by many threads.
__device__ __forceinline__ double stream_at(const Stream& rs, uint32_t i) {
  if (rs.kind == RNG_TRIPLE32) return t32_uniform(rs.seedmix, rs.ctr + i);
  const U4 r = philox4x32_10(U4{rs.k + i - 1u, rs.it, rs.chain, 0xB2000001u}, rs.seed,
                             0x6A09E667u);
  return u53(r.x, r.y);
}
__device__ __forceinline__ double stream_normal_at(const Stream& rs, uint32_t i0, int j) {
  const double u1 = stream_at(rs, i0 + 2u * (uint32_t)j + 1u);
  const double u2 = stream_at(rs, i0 + 2u * (uint32_t)j + 2u);
  return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
}
// The stream of chain c for this step's acceptance uniform, and, past it, for
// the next proposal's draws: three uniforms with DE (de_difference), then 2 np
// for the normals.  The step kernel's draws_used advances the triple32 counter by
// the same counts.
__device__ __forceinline__ Stream accept_stream(const ChainArgs& A, int c, uint32_t t) {
  Stream rs = make_stream(A, c);
  if (A.rng != RNG_TRIPLE32) {
    rs.it = t;
    rs.k = 0xFFFF0000u;
  }
  return rs;
}
__device__ __forceinline__ Stream propose_stream(const ChainArgs& A, int c, bool step,
                                                 uint32_t t) {
  Stream rs = make_stream(A, c);
  if (step) {
    if (A.rng == RNG_TRIPLE32) rs.ctr += 1u;  // the acceptance uniform
    rs.it = t + 1;
  }
  return rs;
}

// The DE difference of a chain's next proposal, coordinate j, from the pair of
// the snapshot that its stream draws first.
__device__ __forceinline__ double de_difference(const ChainArgs& A, const Stream& rs, int j) {
  const int n = A.n_chains, np = A.np;
  int a = (int)(stream_at(rs, 1) * (double)n);
  if (a >= n) a = n - 1;
  int b = (int)(stream_at(rs, 2) * (double)n);
  if (b >= n) b = n - 1;
  if (b == a) b = (b + 1) % n;
  const double g = stream_at(rs, 3) < 0.1 ? 1.0 : A.gamma;
  return g * (A.snap[(size_t)a * np + j] - A.snap[(size_t)b * np + j]);
}

// ------------------------------------------ the side of a step's evaluation
// What the end of a step needs besides the data sums depends on the points, the
// counters and the factors only, so extra rows of CTAs (blockIdx.y <
// E.side_rows) compute it beside the evaluation.  Row 0: the f64 priors
// (straight-line code, 65 divisions for the 65-parameter model), one thread
// per chain.  With E.side_z (few chains, where an iteration is a chain of
// latencies and SMs are free) also the logs of the acceptance uniforms, and
// the other rows, a share of the chain block's chains each, the next
// proposals' normals and L z or the DE differences: in the step kernel they
// were 2 of the 6.2 us of an iteration of 8 Gaussian chains.  Inlined: as a
// function of its own it returned wrong values in the tensor-core kernel, for a
// reason that reading and the compiler's statistics (96 registers, 480 bytes of
// stack) do not show.  test_gpu_tensor_cores.py compares that kernel's runs, side
// rows included, with the FP32 kernel's.
template <class Prior>
__device__ __forceinline__ void side_block(const EvalArgs& E, ChainArgs A, int cb, int CG,
                                           int phase, int nthreads) {
  load_vars(A);
  const int np = A.np;
  const bool step = phase == PH_STEP;
  if (blockIdx.y == 0) {
    for (int cl = threadIdx.x; cl < CG; cl += nthreads) {
      const int c = cb * CG + cl;
      if (c >= A.n_chains) continue;
      if (step && E.side_z) E.side_lu[c] = log(stream_at(accept_stream(A, c, A.iter[c]), 1u));
      if (!E.prior_pts) continue;
      const double* p = E.prior_pts + (size_t)c * np;
      if (E.prior_grad) {
        double* g = E.prior_grad + (size_t)c * np;
        for (int j = 0; j < np; ++j) g[j] = 0.0;
        E.prior_out[c] = Prior::value_grad(A, c, p, g);
      } else {
        E.prior_out[c] = Prior::value(A, c, p);
      }
    }
    return;
  }
  const int rows = E.side_rows - 1, row = (int)blockIdx.y - 1, per = (CG + rows - 1) / rows;
  const int c0 = cb * CG + row * per;
  const int n = min(min(per, CG - row * per), A.n_chains - c0);  // may be <= 0
  const bool de = A.mode == MODE_DE;
  for (int i = threadIdx.x; i < n * np; i += nthreads) {
    const int c = c0 + i / np, j = i % np;
    const uint32_t t = step ? A.iter[c] : 0u;
    if ((step ? t + 1 : 0u) >= A.n_iter) continue;  // no proposal follows
    const size_t o = (size_t)c * np + j;
    const Stream rs = propose_stream(A, c, step, t);
    E.side_z[o] = stream_normal_at(rs, de ? 3u : 0u, j);
    if (de) E.side_inc[o] = de_difference(A, rs, j);
  }
  if (!A.L) return;
  __syncthreads();  // uniform: the chains' normals are this block's own
  for (int i = threadIdx.x; i < n * np; i += nthreads) {
    const int c = c0 + i / np, k = i % np;
    const double* L = A.L + ((size_t)c * np + k) * np;
    const double* z = E.side_z + (size_t)c * np;
    double acc = 0.0;
#pragma unroll 8
    for (int j = 0; j <= k; ++j) acc += L[j] * z[j];
    E.side_inc[(size_t)c * np + k] = acc;
  }
}

// --------------------------------------------------------- kernel skeleton
// Tiles per stage: a narrow model's tile is a KB or two (a TMA box is at most
// 256 observations), so a stage holds as many as 16 KB do and the CTA's barrier
// and wait come once for all of them.  With the folds of the generated code
// (codegen.cpp) 40 steps of 2,048 chains x 2^18 observations of the one-column
// mixture went from 24.5 to 20.9 ms.
__host__ __device__ inline int stage_tiles(int T, int ncols) {
  const int bytes = T * ncols * 4;
  const int u = bytes > 0 ? (16 << 10) / bytes : 1;
  return u < 1 ? 1 : (u > 8 ? 8 : u);
}
// Shared-memory carve-up (the host's smem_bytes() must agree):
//   2 data stages [U][ncols][T] f32 | params [np][CG] f32 (rounded to 4; none
//   for chain-lane bodies, whose lanes read their parameters from global
//   memory) | reduction [kWarps][G][width] f64 | 2 mbarriers.
__host__ __device__ inline size_t skel_param_floats(int np, int CG, bool lanes) {
  return lanes ? 0 : (((size_t)np * CG + 3) & ~(size_t)3);
}
__host__ __device__ inline size_t skel_smem_bytes(int T, int ncols, int np, int CG, int G,
                                                  int width, bool lanes = false,
                                                  int warps = kWarps) {
  return 2 * (size_t)stage_tiles(T, ncols) * T * ncols * 4 + skel_param_floats(np, CG, lanes) * 4 +
         (size_t)warps * G * width * 8 + 2 * 8;
}

// Body contract (G chains per thread):
//   bool kChainLanes                       false: lanes are observations (below);
//                                          true: lanes are chains, G counts the
//                                          chains of a warp (32 kLaneChains: lane
//                                          l holds l, l + 32, ...), the body has
//                                          begin_lanes(pc, C_pad), eval4(xo, nv),
//                                          last4(k) instead of begin/eval/last
//   bool kLanesAcc (chain lanes)           true: the body accumulates values
//                                          1 .. W-1 in its own row of the
//                                          reduction buffer (begin_lanes_acc(pc,
//                                          C_pad, row), flush_tile() after each
//                                          tile); only value 0 is written here
//   void begin(const float* pc0, int CG)   pc0 = this thread's first chain in
//                                          the [np][CG] parameter tile
//   void eval(const float* xo, int T, bool valid)  one observation
//   kRounds == 2: eval_rounds(xo, xs, T, v0, v1) takes two, at xo and xo + xs
//   float last(int g)                      value of the last eval (pointwise)
//   void end()                             after the last observation
//   double total(int g, int w)             w = 0 value, 1.. gradient entries
//   W (compile time) = E.width values reduced per chain; NW warps per CTA
template <int G, int W, class Body, class Prior, int NW = kWarps>
__device__ __forceinline__ void run_iteration(const TmapDesc* tmap, const EvalArgs& E,
                                              const ChainArgs& A, int phase, Body& body) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int CG = E.CG, T = E.T, ncols = E.ncols, np = E.np;
  // Chain blocks vary fastest, so the CTAs that share an observation tile
  // run in the same wave and read it through L2 once.
  int cb = blockIdx.x, ob = blockIdx.y, tiles_per_cta = E.tiles_per_cta;
  if (E.side_rows) {
    if (ob < E.side_rows) {
      pdl_wait();
      pdl_trigger();
      side_block<Prior>(E, A, cb, CG, phase, 32 * NW);
      return;
    }
    ob -= E.side_rows;
  }
  if (E.active) {  // delayed acceptance: geometry from the live count
    pdl_wait();
    const int live = (int)*E.active;
    const int busy = (live + CG - 1) / CG;
    const int nob = da_obs_blocks(live, CG, (int)(gridDim.x * gridDim.y), E.ntiles,
                                  &tiles_per_cta);
    const int id = (int)(blockIdx.y * gridDim.x + blockIdx.x);
    if (busy == 0 || id >= busy * nob) return;
    cb = id % busy;
    ob = id / busy;
  }
  const int WO = NW / E.WC;
  const int wc = warp % E.WC, wo = warp / E.WC;

  const size_t tile_floats = (size_t)T * ncols, stage_floats = E.U * tile_floats;
  const int U = E.U;
  float* xs = reinterpret_cast<float*>(smem_raw);
  constexpr bool kLanes = Body::kChainLanes;
  float* psm = xs + 2 * stage_floats;
  double* red = reinterpret_cast<double*>(psm + skel_param_floats(np, CG, kLanes));
  uint64_t* bars = reinterpret_cast<uint64_t*>(red + (size_t)NW * G * W);

  const int t0 = ob * tiles_per_cta;
  const int t1 = min(t0 + tiles_per_cta, E.ntiles);
  const int nt = max(t1 - t0, 0);
  const int nst = (nt + U - 1) / U;  // stages
  // Stage s of this CTA: tiles t0 + s U .. into buffer s % 2.
  auto load_stage = [&](int s) {
    const int n = min(U, nt - s * U);
    float* dst = xs + (s & 1) * stage_floats;
    mbar_expect_tx(&bars[s & 1], (uint32_t)(n * tile_floats * sizeof(float)));
    for (int u = 0; u < n; ++u)
      tma_load_2d(dst + u * tile_floats, tmap, &bars[s & 1], (t0 + s * U + u) * T, 0);
  };
  // No tiles (or no data columns): the tensor map is never touched.
  const bool staged = ncols > 0 && nt > 0;
  if (tid == 0 && staged) {
    tma_prefetch_desc(tmap);
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_fence_init();
    // The data does not change during a run: the first tiles are on their way
    // before the previous step's proposals are waited for.
    for (int s = 0; s < 2 && s < nst; ++s) load_stage(s);
  }
  pdl_wait();
  pdl_trigger();
  if constexpr (!kLanes) {
    for (int i = tid; i < np * CG; i += 32 * NW) {
      const int p = i / CG, cl = i % CG;
      psm[i] = E.params[(size_t)p * E.C_pad + (size_t)cb * CG + cl];
    }
  }
  __syncthreads();
  if constexpr (kLanes) {
    const float* pc = E.params + (size_t)cb * CG + (size_t)wc * G + lane;
    if constexpr (Body::kLanesAcc)
      body.begin_lanes_acc(pc, E.C_pad, red + ((size_t)warp * G + lane) * W);
    else
      body.begin_lanes(pc, E.C_pad);
  } else {
    body.begin(psm + wc * G, CG);
  }

  for (int k = 0; k < nst; ++k) {
    const int st = k & 1;
    int gave_up = 0;
    if (staged && !mbar_wait_bounded(&bars[st], (uint32_t)((k >> 1) & 1))) {
      gave_up = 1;
      if (lane == 0) atomicOr(E.err, DEV_ERR_TMA_TIMEOUT);
    }
    const int nu = min(U, nt - k * U);
    for (int u = 0; u < nu; ++u) {
      const float* tile = xs + st * stage_floats + u * tile_floats;
      const int obs0 = (t0 + k * U + u) * T;
      if constexpr (kLanes) {
        // quads of observations (o .. o + 3), the WO warps of a chain group
        // taking every WO-th quad; all lanes read the same addresses
        for (int o = 4 * wo; o < T; o += 4 * WO) {
          const long long left = (long long)E.n_obs - (obs0 + o);
          if (left <= 0) break;
          const int nv = left >= 4 ? 4 : (int)left;
          body.eval4(tile + o, nv);
          if (phase == PH_POINTWISE) {
            const int c = cb * CG + wc * 32 + lane;
            if (c < E.n_points) {
  #pragma unroll
              for (int q = 0; q < 4; ++q)  // constant indices keep the values in registers
                if (q < nv) E.pointwise[(size_t)c * E.n_obs + obs0 + o + q] = body.last4(q);
            }
          }
        }
        if constexpr (Body::kLanesAcc) body.flush_tile();
      } else if constexpr (Body::kObsPerEval == 2) {
        // observation pairs (2 pi, 2 pi + 1); T is even, so each pair is
        // 8-byte aligned in every column of the tile
        auto pair = [&](int pi) {
          const int obs = obs0 + 2 * pi;
          const bool v0 = obs < E.n_obs, v1 = obs + 1 < E.n_obs;
          body.eval2(tile + 2 * pi, T, v0, v1);
          if (phase == PH_POINTWISE && v0) {
  #pragma unroll
            for (int g = 0; g < G; ++g) {
              const int c = cb * CG + wc * G + g;
              if (c < E.n_points) {
                const float2 lv = body.last2(g);
                E.pointwise[(size_t)c * E.n_obs + obs] = lv.x;
                if (v1) E.pointwise[(size_t)c * E.n_obs + obs + 1] = lv.y;
              }
            }
          }
        };
        constexpr int kT = Body::kTileObs;  // compile-time tile height, or 0
        if (kT > 0 && kT % 64 == 0 && WO == 1) {
          // every warp covers the tile: a fixed trip count, unrolled so the
          // compiler can overlap one pair's loads with another's arithmetic
          bool done = false;
          if constexpr (kT > 0) {
            if (phase != PH_POINTWISE && obs0 + kT <= E.n_obs) {  // a full tile
  #pragma unroll
              for (int it = 0; it < kT / 64; ++it) body.eval2_full(tile + 2 * (lane + 32 * it));
              body.flush();
              done = true;
            }
          }
          if (!done) {
  #pragma unroll
            for (int it = 0; it < (kT > 0 ? kT : 64) / 64; ++it) pair(lane + 32 * it);
          }
        } else {
          for (int pi = lane + 32 * wo; 2 * pi < T; pi += 32 * WO) pair(pi);
        }
      } else if constexpr (Body::kRounds == 2) {
        // two of a lane's observations per call (the host chooses this body
        // where 64 WO divides T)
        for (int ol = lane + 32 * wo; ol < T; ol += 64 * WO) {
          const int obs = obs0 + ol, xs = 32 * WO;
          const bool v0 = obs < E.n_obs, v1 = obs + xs < E.n_obs;
          body.eval_rounds(tile + ol, xs, T, v0, v1);
          if (phase == PH_POINTWISE) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
              const int c = cb * CG + wc * G + g;
              if (c >= E.n_points) continue;
              float* out = E.pointwise + (size_t)c * E.n_obs + obs;
              if (v0) out[0] = body.last(g, 0);
              if (v1) out[xs] = body.last(g, 1);
            }
          }
        }
      } else {
        for (int ol = lane + 32 * wo; ol < T; ol += 32 * WO) {
          const int obs = obs0 + ol;
          const bool valid = obs < E.n_obs;
          body.eval(tile + ol, T, valid);
          if (phase == PH_POINTWISE && valid) {
  #pragma unroll
            for (int g = 0; g < G; ++g) {
              const int c = cb * CG + wc * G + g;
              if (c < E.n_points) E.pointwise[(size_t)c * E.n_obs + obs] = body.last(g);
            }
          }
        }
      }
    }
    // Every warp is done with this stage.  A wait that gave up anywhere in
    // the CTA (the error bit is set) stops the tile loop for the whole CTA:
    // no more loads are issued, thread 0 waits (bounded) for the loads still
    // in flight into this CTA's stages, and the CTA goes on to the reduction
    // (its partial is written whatever happened).
    if (__syncthreads_or(gave_up)) {
      if (tid == 0 && staged) {
        mbar_wait_bounded(&bars[st], (uint32_t)((k >> 1) & 1));
        if (k + 1 < nst) mbar_wait_bounded(&bars[st ^ 1], (uint32_t)(((k + 1) >> 1) & 1));
      }
      __syncthreads();
      break;
    }
    if (tid == 0 && staged && k + 2 < nst) load_stage(k + 2);
  }
  if (phase == PH_POINTWISE) return;
  body.end();

  // FP64 fixed-order reduction of each of the W values: lanes (shuffle
  // tree), then the WO warps that share a chain group, in warp order.
#pragma unroll
  for (int w = 0; w < W; ++w) {
    if constexpr (kLanes) {  // each lane holds its own chains' sums
      if (!Body::kLanesAcc || w == 0) {
#pragma unroll
        for (int c = 0; c < Body::kLaneChains; ++c)
          red[((size_t)warp * G + 32 * c + lane) * W + w] = body.total(c, w);
      }
    } else {
      double tot[G];
#pragma unroll
      for (int g = 0; g < G; ++g) tot[g] = body.total(g, w);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int g = 0; g < G; ++g) tot[g] += __shfl_down_sync(0xffffffffu, tot[g], off);
      }
      if (lane == 0) {
#pragma unroll
        for (int g = 0; g < G; ++g) red[((size_t)warp * G + g) * W + w] = tot[g];
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < CG * W; i += 32 * NW) {
    const int cl = i / W, w = i % W;
    const int wcc = cl / G, g = cl % G;
    double v = 0.0;
    for (int o = 0; o < WO; ++o) v += red[((size_t)(o * E.WC + wcc) * G + g) * W + w];
    E.partials[((size_t)ob * E.C_pad + (size_t)cb * CG + cl) * W + w] = v;
  }
}

}  // namespace gpum
