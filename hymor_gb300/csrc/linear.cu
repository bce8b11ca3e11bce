// Linearised residual on the device: coloured finite-difference Jacobian assembly
// into stencil blocks, the block-stencil matvec (and its transpose) and the
// Taylor propagator exp(A dt)^n used by the exponential-transform eigen solvers.
//
// Device layout of the Jacobian: 144 planes of N doubles (plane (q*4 + vout)*4 + vin,
// q = neighbour slot), so that consecutive threads (cells) read consecutive
// addresses. hymor_jacobian_get/set convert to the per-cell block layout of
// include/hymor.h.
#include <cmath>
#include <cstdio>
#include <vector>

#include <cooperative_groups.h>

#include <algorithm>

#include "ff.cuh"
#include "fx.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace hymor {
DevCtx& ctx_dev(hymor_ctx* c);
cudaStream_t ctx_stream(hymor_ctx* c);
int ctx_fail(hymor_ctx* c, int code, const char* msg);
int ctx_check_waits(hymor_ctx* c);  // reports (once) a resident propagation that gave up
int ctx_select_device(hymor_ctx* c);
bool linear_spare_release(hymor_ctx* ctx);
cudaError_t ctx_malloc(hymor_ctx* ctx, void** p, size_t bytes);
cudaError_t ctx_malloc_async(hymor_ctx* ctx, void** p, size_t bytes);
std::vector<void*>& ctx_allocs(hymor_ctx* c);
void*& ctx_linear_state(hymor_ctx* c);
void launch_shock_bc_flags(const DevCtx& d, bool on_S, bool copy_pts, bool do_shock, bool do_bc, int a_mode,
                           cudaStream_t st);

namespace {

constexpr int kMvThreads = 256;

// Threads per block of a matvec over `items` work items: 256, or fewer when that would
// leave SMs idle. One vector on a 100 x 80 grid is 8000 items: in 256-thread blocks they
// sit on 32 SMs, whose FP64 pipes then bound the matvec; in 64-thread blocks they spread
// over 125.
int mv_threads(long items, int sms) {
  if (items >= (long)sms * kMvThreads) return kMvThreads;
  const long per_sm = (items + sms - 1) / sms;
  const long t = ((per_sm + 31) / 32) * 32;
  return (int)(t < 32 ? 32 : t);
}
constexpr int kVecChunk = 4;

struct Wrap {
  int nchi, neta, per_chi, per_eta;
  // input cell of output (i, j) at offset (a, b); -1 if the reference assembles no entry
  __device__ __forceinline__ long nbr(int i, int j, int a, int b) const {
    int ii = i + a, jj = j + b;
    const bool wi = ii < 0 || ii >= nchi, wj = jj < 0 || jj >= neta;
    if ((wi && !per_chi) || (wj && !per_eta) || (wi && wj)) return -1;
    if (wi) ii = ii < 0 ? ii + nchi : ii - nchi;
    if (wj) jj = jj < 0 ? jj + neta : jj - neta;
    return (long)ii + (long)jj * nchi;
  }
};

Wrap make_wrap(const hymor_config& c) {
  return Wrap{c.nchi, c.neta, c.bc_chi0 == HYMOR_BC_PERIODIC && c.bc_chi1 == HYMOR_BC_PERIODIC,
              c.bc_eta0 == HYMOR_BC_PERIODIC && c.bc_eta1 == HYMOR_BC_PERIODIC};
}

// Y = S with variable `var` of every interior cell of colour `colour` (1..9, the
// pattern of GET_PERTURBATION_MATRIX, LINEARIZE_EQUATIONS_NO_DISCONTINUITY.jl:959-983)
// raised by flow_cells * eps; then p, T of Y. shock_row = j > 0 raises instead the
// cell (i, sc_i - j) of every column by eps (the flow-to-shock-speed perturbations,
// :140-258).
// Lane z of a batched launch (DevCtx::lane_stride) evaluates the perturbation `first + z`:
// colour and variable of the A11 colours (var * 9 + colour - 1, when `colours`), else the
// members as they are.
struct PertArgs {
  Cons S, Y;
  double *p, *T;
  double* aY;
  int nrcbc;
  const int* cell_idx;
  double eps, gm1;
  int nchi, neta, var, colour, shock, shock_row;
  int j0, j1;        // rows written, j0 <= j < j1 (ghosted)
  long lane;
  int first, batch;  // batch: 0 one perturbation; 1 the A11 colours; 2 the A21 rows (j, var)
};

__global__ void k_perturb_thermo(PertArgs a) {
  const long off = blockIdx.z * a.lane;
  a.Y.rho += off; a.Y.ru += off; a.Y.rv += off; a.Y.rE += off;
  a.p += off; a.T += off; a.aY += off;
  const int id = a.first + blockIdx.z;
  if (a.batch == 1) {
    a.var = id / 9;
    a.colour = id % 9 + 1;
  } else if (a.batch == 2) {
    a.shock_row = id / 4 + 1;
    a.var = id % 4;
  }
  const int NI = a.nchi + 2;
  const long G = (long)NI * a.j1;
  const int si = (a.colour % 3 == 0) ? 3 : a.colour % 3;  // 1-based start in chi
  const int sj = (a.colour + 2) / 3;                       // 1-based start in eta
  for (long k = (long)NI * a.j0 + blockIdx.x * (long)blockDim.x + threadIdx.x; k < G; k += (long)gridDim.x * blockDim.x) {
    const int j = (int)((unsigned)k / (unsigned)NI), i = (int)((unsigned)k - (unsigned)j * (unsigned)NI);
    double v[4] = {a.S.rho[k], a.S.ru[k], a.S.rv[k], a.S.rE[k]};
    if (a.var >= 0 && i >= 1 && i <= a.nchi && j >= 1 && j <= a.neta) {
      if (a.shock_row) {
        if (j == a.cell_idx[i - 1] - a.shock_row) v[a.var] += a.eps;
      } else {
        const bool hit = (i >= si) && ((i - si) % 3 == 0) && (j >= sj) && ((j - sj) % 3 == 0);
        const double flow = (!a.shock || j < a.cell_idx[i - 1]) ? 1.0 : 0.0;
        v[a.var] = v[a.var] + flow * (hit ? 1.0 : 0.0) * a.eps;
      }
    }
    a.Y.rho[k] = v[0]; a.Y.ru[k] = v[1]; a.Y.rv[k] = v[2]; a.Y.rE[k] = v[3];
    const double ir = 1.0 / v[0];
    const double ke = fma(v[1], v[1], v[2] * v[2]) * ir;
    const double eint = fma(-0.5, ke, v[3]);
    a.p[k] = eint * a.gm1;
    a.T[k] = eint * ir;
    if (a.nrcbc) {
      const int NJ = a.neta + 2;
      const bool nb = ((a.nrcbc & 1) && i == 1) || ((a.nrcbc & 2) && i == NI - 2) ||
                      ((a.nrcbc & 4) && j == 1) || ((a.nrcbc & 8) && j == NJ - 2);
      if (nb) a.aY[k] = sqrt((a.gm1 + 1) * (eint * a.gm1) / v[0]);
    }
  }
}

// coef[plane(q, vo, var)][m] = (Fp[vo][m] - Fb[vo][m]) / eps with Fp the residual of the colour
// of slot q's input cell m + offset(q) (GET_OUTPUT_INDEXING_A11,
// LINEARIZE_EQUATIONS_NO_DISCONTINUITY.jl:306-788; REMOVE_BASE_OUTPUT :935-946), for one
// variable (grid z: first_var + z) whose nine colours are nine consecutive lanes. A thread
// takes a cell and loops over its slots, so that a warp writes whole rows of a plane and its
// reads of the three colours of a row of slots share their lines in L1; one colour at a time
// every warp wrote a third of the sectors of three planes. Linearisation at 600 x 300: 3.29 ms
// with a pass per colour, 2.70 ms so. PART: the lanes are some of a variable's colours (a device
// without the memory for nine), one group after another on one stream.
struct ScatArgs {
  const double* Fp[4];
  const double* Fb[4];
  double* coef;
  unsigned char* nz;    // 4 x N, byte var N + m: cell m has a non-zero entry of that variable
  Wrap w;
  double eps, inv_eps;  // inv_eps: the rounded reciprocal of eps, 0 to divide
  long N;
  long lane;
  int first_var;
  int colour0, colours;  // PART: the lanes' colours
};

// d / eps, correctly rounded. The FP64 division of the compiler takes ~25 FP64 instructions
// and this GPU issues one per ~70 cycles, so that the four quotients of a cell bounded the
// scatter. With y = RN(1 / eps): q0 = d y is within two ulps; one residual correction
// (r = d - eps q0 exact by FMA) makes it faithful, and by Markstein's theorem (IBM J. Res.
// Dev. 34 (1990) 111-119) the second gives the rounded quotient: five instructions. Outside
// the exponents where every step is exact (d below 2^-500, infinite or NaN) it divides; the
// host gives inv_eps = 0 for an eps whose reciprocal the theorem leaves out (significand of
// all ones) or whose exponent is extreme. 600 x 300, one colour's scatter: 35.7 -> 25.4 us.
__device__ __forceinline__ double div_eps(double d, double eps, double y) {
  const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
  if (y != 0.0) {
    if ((__double_as_longlong(d) << 1) == 0) return d;  // +-0 / eps, eps > 0
    if (e - 523u < 1000u) {
      double q = d * y;
      q = fma(fma(-eps, q, d), y, q);
      return fma(fma(-eps, q, d), y, q);
    }
  }
  return d / eps;
}
// the rounded reciprocal of eps for div_eps, or 0
double div_eps_reciprocal(double eps) {
  int ex = 0;
  const double m = std::frexp(std::fabs(eps), &ex);
  if (!(eps > 0) || !(m < 1) || ex < -200 || ex > 200 || m == 1.0 - 0x1p-53) return 0.0;
  return 1.0 / eps;
}

template <bool PART>
__global__ void __launch_bounds__(256) k_scatter(ScatArgs a) {
  const long N = a.N, off = 9L * blockIdx.z * a.lane;
  const int var = a.first_var + blockIdx.z;
  const unsigned nchi_u = (unsigned)a.w.nchi;
  for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < N; m += (long)gridDim.x * blockDim.x) {
    const int j = (int)((unsigned)m / nchi_u), i = (int)((unsigned)m - (unsigned)j * nchi_u);
    double fb[4];
    unsigned long long any = 0;
#pragma unroll
    for (int vo = 0; vo < 4; ++vo) fb[vo] = a.Fb[vo][m];
#pragma unroll
    for (int b = -1; b <= 1; ++b)
#pragma unroll
      for (int aa = -1; aa <= 1; ++aa) {
        const long n = a.w.nbr(i, j, aa, b);
        if (n < 0) continue;
        const unsigned nj = (unsigned)n / nchi_u, ni = (unsigned)n - nj * nchi_u;
        const int colour = (int)(3 * (nj % 3u) + ni % 3u) - (PART ? a.colour0 : 0);  // of the input cell
        if (PART && (colour < 0 || colour >= a.colours)) continue;
        const long o = off + (long)colour * a.lane + m;
        const int q = (b + 1) * 3 + (aa + 1);
#pragma unroll
        for (int vo = 0; vo < 4; ++vo) {
          const double d = div_eps(a.Fp[vo][o] - fb[vo], a.eps, a.inv_eps);
          any |= (unsigned long long)__double_as_longlong(d) << 1;
          a.coef[((long)(q * 4 + vo) * 4 + var) * N + m] = d;
        }
      }
    a.nz[var * N + m] = any != 0 || (PART && a.colour0 && a.nz[var * N + m]);
  }
}

// y_j = scale * (L x_j) (transpose 0) or scale * (Lᵀ x_j) (transpose 1); optionally
// acc_j += c_acc * y_j. Vectors: 4N each, column-major batch.
struct MvArgs {
  const double* coef;
  const unsigned char* nz;
  const double* X;
  double* Y;
  double* acc;
  double scale, c_acc;
  // a term of the previous matvec to add into acc first (acc += c_prev acc_prev), or null:
  // the propagator accumulates each Taylor term one matvec late, so that the first matvec
  // of a step can read acc as its input without a copy
  const double* acc_prev;
  double c_prev;
  // per-vector scale (k entries) replacing `scale`, or null: a batch of propagations with
  // different time steps (transient-growth horizons)
  const double* vscale;
  Wrap w;
  long N;
  long ld;  // vector stride (4N, or 4N + Nchi with the shock unknowns)
  int k, transpose;
};

// Cells without entries: at and above the shocked rows the residual is masked, so a quarter to
// four fifths of the cells of a shock-fitted flow have all-zero blocks, which need not be read
// nor multiplied. nz[m] (written with the blocks): kMaskRow when cell m's own blocks have a
// non-zero entry (its outputs), kMaskCol when a block that takes cell m as its input does (the
// transpose's outputs). A skipped output is zero, except that a zero times an infinity or NaN
// is NaN: it takes a NaN where an input of its neighbours is not finite. Only the matvecs whose
// time is the blocks' read or their FP64 products test the mask, with a quarter of the cells
// empty: the FP64 batch (800 x 400, 64 vectors: 4.88 -> 3.64 ms; one vector 82.9 -> 66.2 us),
// and one float-float vector on a large grid (1200 x 400, 200 matvecs: 19.6 -> 16.5 ms). The
// thread-per-output ones and the float-float batches wait for the latency of their loads, which
// the test lengthens (100 x 80: one vector 840 -> 927 us, 64 vectors 7.6 -> 9.1 ms).
constexpr unsigned kMaskRow = 1, kMaskCol = 2;
__device__ __forceinline__ unsigned poison(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) == 0x7ff00000u;
}
__device__ __forceinline__ double poisoned(double y, unsigned bad) {
  return bad ? __longlong_as_double(0x7ff8000000000000LL) : y;
}

// ST: the blocks exceed L2 and are read with streaming (evict-first) loads, which keep the
// vectors that every neighbour re-reads in L2; blocks that fit stay cached from one matvec
// of a propagation to the next (a compile-time choice: a branch per load slowed the loads)
template <bool ST>
__device__ __forceinline__ double ld_coef(const double* p) {
  return ST ? __ldcs(p) : *p;
}

// y = scale * A x (or A^T x), acc += c_acc y. The work items are (cell, chunk of
// kVecChunk vectors) pairs, cell fastest, over a grid-stride loop: a batch of vectors on
// a small grid still spreads over every SM (a 100 x 80 grid is 8000 cells, 64 vectors are
// 16 chunks of it), and neighbouring threads read neighbouring cells.
// Few cells x vectors (a small grid, one or a few vectors): one thread per (cell, output
// component, vector), the same FMA chain per output as matvec_multi (bit-identical). On
// GB300 one warp issues one FP64 instruction per ~76 cycles of its SM sub-partition, so a
// warp per 32 cells (148 FP64 instructions each, per vector) would bound a small grid's
// matvec by its own issue rate; a thread per output spreads the work over four times the
// warps per vector. The next neighbour block's coefficients and inputs are loaded while
// the current block's FMAs run.
template <bool ST>
__device__ __forceinline__ void matvec_one(const MvArgs& a) {
  const long N = a.N;
  const long outs = 4 * N;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < outs * a.k; t += (long)gridDim.x * blockDim.x) {
    const long vec = t / outs;
    const long w = t - vec * outs;
    const long m = w % N;
    const int comp = (int)(w / N);  // output component (v_out, or v_in of the transpose)
    const int i = (int)(m % a.w.nchi), j = (int)(m / a.w.nchi);
    const double* xv = a.X + vec * a.ld;
    double y = 0;
    double B[2][4], X[2][4];
    bool ok[2];
    auto load = [&](int q, int slot) {
      const int b = q / 3 - 1, aa = q % 3 - 1;
      long n, cell;  // input cell, and the cell that owns the block
      if (!a.transpose) {
        n = a.w.nbr(i, j, aa, b);
        cell = m;
      } else {
        // m is the input cell of output cell n = m - (aa, b); block slot of (aa, b)
        n = a.w.nbr(i, j, -aa, -b);
        cell = n;
      }
      ok[slot] = n >= 0;
      if (n >= 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // row comp of the block (columns e), or column comp of it for the transpose
          const int plane = a.transpose ? q * 16 + e * 4 + comp : q * 16 + comp * 4 + e;
          B[slot][e] = ld_coef<ST>(a.coef + (long)plane * N + cell);
          X[slot][e] = xv[e * N + n];
        }
      }
    };
    load(0, 0);
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int c = q & 1;
      if (q + 1 < 9) load(q + 1, c ^ 1);
      if (!ok[c]) continue;
      y = fma(B[c][0], X[c][0], fma(B[c][1], X[c][1], fma(B[c][2], X[c][2], fma(B[c][3], X[c][3], y))));
    }
    const double val = (a.vscale ? a.vscale[vec] : a.scale) * y;
    const long o = vec * a.ld + comp * N + m;
    a.Y[o] = val;
    if (a.acc) {
      double r = a.acc[o];
      if (a.acc_prev) r = fma(a.acc_prev[o], a.c_prev, r);
      a.acc[o] = fma(val, a.c_acc, r);
    }
  }
}

// The thread-per-output path (matvec_one) when the cells x vectors are fewer than 32 per
// warp slot of 8 warps on every SM sub-partition; more of them already fill those slots
// with one thread per (cell, chunk of vectors) (matvec_multi, whose single pass over the
// 144 coefficients for a chunk of vectors is then cheaper).
__host__ __device__ inline long mv_one_limit(int sms) { return 8L * 32 * 4 * sms; }
// the Jacobian's blocks (144 per cell, 8 bytes each) larger than this many bytes take
// streaming loads in the matvecs (about a third of the L2, leaving the rest to the
// vectors); smaller blocks stay cached from one matvec of a propagation to the next
constexpr long kCoefStreamBytes = 48L << 20;
bool mv_one(long N, int k, int sms) { return N * k < mv_one_limit(sms); }

// Work items of a matvec over k vectors: (cell, output component, vector) on the
// thread-per-output path, (cell, chunk of kVecChunk vectors) otherwise.
long mv_items(long N, int k, int sms) {
  return mv_one(N, k, sms) ? 4 * N * k : N * ((k + kVecChunk - 1) / kVecChunk);
}

template <bool ST>
__device__ __forceinline__ void matvec_multi(const MvArgs& a) {
  const long N = a.N;
  const long n4 = a.ld;
  const int chunks = (a.k + kVecChunk - 1) / kVecChunk;
  const long items = N * chunks;
  for (long w = blockIdx.x * (long)blockDim.x + threadIdx.x; w < items; w += (long)gridDim.x * blockDim.x) {
    const long m = w % N;
    const int i = (int)(m % a.w.nchi), j = (int)(m / a.w.nchi);
    {
      const int v0 = (int)(w / N) * kVecChunk;
      const int nv = min(kVecChunk, a.k - v0);
      double y[kVecChunk][4];
#pragma unroll
      for (int v = 0; v < kVecChunk; ++v)
#pragma unroll
        for (int c = 0; c < 4; ++c) y[v][c] = 0;
      unsigned bad = 0;  // bit v: a non-finite input of vector v met a zero block
      if (!(a.nz[m] & (a.transpose ? kMaskCol : kMaskRow))) {
        for (int b = -1; b <= 1; ++b)
          for (int aa = -1; aa <= 1; ++aa) {
            const long n = a.transpose ? a.w.nbr(i, j, -aa, -b) : a.w.nbr(i, j, aa, b);
            if (n < 0) continue;
            for (int v = 0; v < nv; ++v) {
              const double* x = a.X + (long)(v0 + v) * n4 + n;
              bad |= (poison(x[0]) | poison(x[N]) | poison(x[2 * N]) | poison(x[3 * N])) << v;
            }
          }
      } else
#pragma unroll
      for (int b = -1; b <= 1; ++b)
#pragma unroll
        for (int aa = -1; aa <= 1; ++aa) {
          long n;
          long cell;  // cell that owns the block
          int q;
          if (!a.transpose) {
            n = a.w.nbr(i, j, aa, b);
            cell = m;
            q = (b + 1) * 3 + (aa + 1);
          } else {
            // m is the input cell of output cell n = m - (aa, b); block slot of (aa, b)
            n = a.w.nbr(i, j, -aa, -b);
            cell = n;
            q = (b + 1) * 3 + (aa + 1);
          }
          if (n < 0) continue;
          double B[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) B[e] = ld_coef<ST>(a.coef + (long)(q * 16 + e) * N + cell);
          for (int v = 0; v < nv; ++v) {
            const double* x = a.X + (long)(v0 + v) * n4;
            const double x0 = x[n], x1 = x[N + n], x2 = x[2 * N + n], x3 = x[3 * N + n];
            if (!a.transpose) {
#pragma unroll
              for (int vo = 0; vo < 4; ++vo)
                y[v][vo] = fma(B[vo * 4 + 0], x0, fma(B[vo * 4 + 1], x1, fma(B[vo * 4 + 2], x2, fma(B[vo * 4 + 3], x3, y[v][vo]))));
            } else {
#pragma unroll
              for (int vi = 0; vi < 4; ++vi)
                y[v][vi] = fma(B[0 * 4 + vi], x0, fma(B[1 * 4 + vi], x1, fma(B[2 * 4 + vi], x2, fma(B[3 * 4 + vi], x3, y[v][vi]))));
            }
          }
        }
      for (int v = 0; v < nv; ++v) {
        double* yo = a.Y + (long)(v0 + v) * n4;
        const double sc = a.vscale ? a.vscale[v0 + v] : a.scale;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const double val = sc * poisoned(y[v][c], bad & (1u << v));
          yo[c * N + m] = val;
          if (a.acc) {
            double* ac = a.acc + (long)(v0 + v) * n4;
            double r = ac[c * N + m];
            if (a.acc_prev) r = fma(a.acc_prev[(long)(v0 + v) * n4 + c * N + m], a.c_prev, r);
            ac[c * N + m] = fma(val, a.c_acc, r);
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The batched FP64 matvec in fixed point (fx.cuh). A is kept as integer parts for the direction
// applied, made once per write of the blocks: entry (input component e, slot q, output row r) of
// output cell m at plane ((e 9 + q) 4 + r), against the power of two shared by the nine slots of
// (r, e), whose exponents are 16 planes of 16 bits. A block of 256 threads stages a tile of 32 x
// 4 cells of up to kFxVecs vectors, each component against the largest exponent of its tile and
// halo, and a thread forms two rows of its cell: per component the nine slots' products exactly
// in 64-bit integers, then the four components' sums aligned to the largest and added.
//
// Accuracy: the parts and the dropped low product leave ~2^-57 of (largest |a| of a row's nine
// slots) x (largest |x| of the tile), against 2^-52 to 2^-51 of the sum of |a x| of the FP64
// chain. Where that sum (formed beside it from 12 leading bits of the factors, a lower bound) is
// below 2^-5 of that product, the row is formed in FP64 instead: so it is for single small
// entries (L e_i stays exact: an entry above the line has all its 53 bits within the 58), for
// tiles with an infinity or a NaN, and for exponents beyond +-900 (subnormal factors among them).
//
// What bounds it: waiting, with four warps per sub-partition (124 registers a thread): 48 % of the
// issue slots are used, and the stalls are the multiplies' fixed latency (2.3 cycles an issue) and
// the loads of the blocks' parts (1.7). No pipe is full: the integer multiplies, 432 wide
// multiply-adds per cell and vector (FP64: 144 multiply-adds at a fifteenth of that rate, 0.98 of
// the pipe), keep the heavy half of the FMA pipe 52 % busy, the shifts of the alignment and the
// parts the ALU 44 %, the FP64 rows that pipe 11 %. 800 x 400, 64 vectors: 3.64 -> 2.29 ms. Error against sums in 113 bits, relative in the 2-norm, random rows of
// magnitudes 1e-4 .. 2 and component scales 1e-2 .. 1e2: 5.3e-17 (the FP64 chain: 2.1e-16).
constexpr int kFxVecs = 4, kFxRows = 4;
constexpr int kFxHx = 34, kFxHalo = kFxHx * (kFxRows + 2);
constexpr unsigned kFxLeast = 1u << 19;  // 2^-5 of a full-scale product of the 12-bit leads

struct FxArgs {
  const int2* part;
  const short* ex;  // 16 x N, plane r 4 + e
  MvArgs mv;        // the FP64 blocks, vectors and sizes
};

template <bool T>
__global__ void __launch_bounds__(256) k_fx_build(const double* coef, int2* part, short* ex, Wrap w, long N) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < 16 * N; t += (long)gridDim.x * blockDim.x) {
    const long m = t % N;
    const int re = (int)(t / N), r = re >> 2, e = re & 3;
    const int j = (int)((unsigned)m / (unsigned)w.nchi), i = (int)((unsigned)m - (unsigned)j * (unsigned)w.nchi);
    double a[9];
    int f = 0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int da = q % 3 - 1, db = q / 3 - 1;
      const long n = T ? w.nbr(i, j, -da, -db) : w.nbr(i, j, da, db);
      a[q] = n < 0 ? 0.0 : (T ? coef[(long)(q * 16 + e * 4 + r) * N + n] : coef[(long)(q * 16 + re) * N + m]);
      f = max(f, fx_field(a[q]));
    }
    const int E = fx_exponent(f);
    ex[t] = (short)E;
#pragma unroll
    for (int q = 0; q < 9; ++q)
      part[(long)((e * 9 + q) * 4 + r) * N + m] = E == kFxZero || E == kFxBad ? make_int2(0, 0) : fx_split(a[q], E);
  }
}

// row r of cell m on the vector x, in FP64 (matvec_multi's chain)
__device__ __noinline__ double fx_row_f64(const MvArgs& a, const double* x, long m, int i, int j, int r) {
  const long N = a.N;
  double y = 0;
#pragma unroll 3
  for (int q = 0; q < 9; ++q) {
    const int da = q % 3 - 1, db = q / 3 - 1;
    const long n = a.transpose ? a.w.nbr(i, j, -da, -db) : a.w.nbr(i, j, da, db);
    if (n < 0) continue;
    const double* c = a.transpose ? a.coef + (long)(q * 16 + r) * N + n : a.coef + (long)(q * 16 + r * 4) * N + m;
    const long ce = a.transpose ? 4 * N : N;
    y = fma(c[0], x[n], fma(c[ce], x[N + n], fma(c[2 * ce], x[2 * N + n], fma(c[3 * ce], x[3 * N + n], y))));
  }
  return y;
}

__global__ void __launch_bounds__(256, 2) k_matvec_fx(FxArgs A) {
  __shared__ int2 xs[kFxVecs * 4 * kFxHalo];
  __shared__ int smax[kFxVecs * 4];
  const MvArgs& a = A.mv;
  const long N = a.N;
  const int nchi = a.w.nchi, neta = a.w.neta, tx = (nchi + 31) / 32, chunks = (a.k + kFxVecs - 1) / kFxVecs;
  const int lane = threadIdx.x & 31, row = (threadIdx.x >> 5) % kFxRows, r0 = (threadIdx.x >> 7) * 2;
  // the chunk runs fastest: the blocks of a tile's chunks read its parts at about the same time
  const int tile = blockIdx.x / chunks, v0 = (blockIdx.x - tile * chunks) * kFxVecs, nv = min(kFxVecs, a.k - v0);
  const int i0 = (tile % tx) * 32, j0 = (tile / tx) * kFxRows;
  const int i = i0 + lane, j = j0 + row;
  const long m = i + (long)j * nchi;
  const bool in = i < nchi && j < neta;
  if (threadIdx.x < kFxVecs * 4) smax[threadIdx.x] = 0;
  __syncthreads();
  // a halo cell per thread: its values, the tile's largest exponent of each, then the parts
  // (cells past the grid's edge wrap where it is periodic; the others' parts meet zero entries)
  double xv[kFxVecs * 4];
  const int h = threadIdx.x;
  if (h < (kFxHalo + 31) / 32 * 32) {
    int ii = i0 - 1 + h % kFxHx, jj = j0 - 1 + h / kFxHx;
    if (a.w.per_chi) ii = ii < 0 ? ii + nchi : (ii >= nchi ? ii - nchi : ii);
    if (a.w.per_eta) jj = jj < 0 ? jj + neta : (jj >= neta ? jj - neta : jj);
    const bool ok = h < kFxHalo && ii >= 0 && ii < nchi && jj >= 0 && jj < neta;
    const double* x = a.X + (long)v0 * a.ld + (ok ? ii + (long)jj * nchi : 0);
    int mine = 0;
#pragma unroll
    for (int c = 0; c < kFxVecs * 4; ++c) {
      xv[c] = ok && (c >> 2) < nv ? x[(c >> 2) * a.ld + (c & 3) * N] : 0.0;
      const int f = __reduce_max_sync(0xffffffffu, fx_field(xv[c]));
      if (lane == c) mine = f;
    }
    if (lane < kFxVecs * 4) atomicMax(&smax[lane], mine);
  }
  __syncthreads();
  if (h < kFxHalo) {
#pragma unroll
    for (int c = 0; c < kFxVecs * 4; ++c) {
      const int E = fx_exponent(smax[c]);
      xs[c * kFxHalo + h] = E == kFxZero || E == kFxBad ? make_int2(0, 0) : fx_split(xv[c], E);
    }
  }
  __syncthreads();
  if (!in) return;
  const int sg = a.transpose ? -1 : 1;
  const int2* x0 = xs + (lane + 1) + (row + 1) * kFxHx;
  long long T[2][kFxVecs];
  unsigned S[2][kFxVecs];
  int top[2][kFxVecs];  // the largest exponent of the four components' products
  bool f64[2] = {false, false};
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int v = 0; v < kFxVecs; ++v) {
      T[r][v] = 0;
      S[r][v] = 0;
      top[r][v] = -0x7fffffff;
    }
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int ea = A.ex[((r0 + r) * 4 + e) * N + m];
      if (ea == kFxBad) f64[r] = true;
      if (ea == kFxZero) continue;
#pragma unroll
      for (int v = 0; v < kFxVecs; ++v) {
        const int ev = fx_exponent(smax[v * 4 + e]);
        if (ev != kFxZero) top[r][v] = max(top[r][v], ea + ev);
      }
    }
  // (a cell without entries has nothing to sum: its outputs are zero, or FP64's NaN)
  const int ne = a.nz[m] & (a.transpose ? kMaskCol : kMaskRow) ? 4 : 0;
#pragma unroll 1
  for (int e = 0; e < ne; ++e) {
    long long hh[2][kFxVecs], cr[2][kFxVecs];
    unsigned se[2][kFxVecs];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int v = 0; v < kFxVecs; ++v) {
        hh[r][v] = cr[r][v] = 0;
        se[r][v] = 0;
      }
#pragma unroll 1
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int2* p = A.part + (long)((e * 9 + b * 3 + c) * 4 + r0) * N + m;
        const int2 p0 = p[0], p1 = p[N];
        // the leads' sum over the cell and its four face neighbours: a lower bound
        const bool face = c == 1 || b == 1;
        const unsigned l0 = (unsigned)abs(p0.x) >> 17, l1 = (unsigned)abs(p1.x) >> 17;
        const int2* xq = x0 + e * kFxHalo + sg * (c - 1) + sg * (b - 1) * kFxHx;
#pragma unroll
        for (int v = 0; v < kFxVecs; ++v) {
          const int2 x = xq[v * 4 * kFxHalo];
          hh[0][v] += (long long)p0.x * x.x;
          hh[1][v] += (long long)p1.x * x.x;
          cr[0][v] += (long long)p0.x * x.y;
          cr[1][v] += (long long)p1.x * x.y;
          cr[0][v] += (long long)p0.y * x.x;
          cr[1][v] += (long long)p1.y * x.x;
          if (face) {
            const unsigned lx = (unsigned)abs(x.x) >> 17;
            se[0][v] += l0 * lx;
            se[1][v] += l1 * lx;
          }
        }
      }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int ea = A.ex[((r0 + r) * 4 + e) * N + m];
#pragma unroll
      for (int v = 0; v < kFxVecs; ++v) {
        const long long W = hh[r][v] + ((cr[r][v] + (1ll << (kFxLow - 1))) >> kFxLow);
        const int sh = top[r][v] - ea - fx_exponent(smax[v * 4 + e]) + 1;  // >= 1 where W != 0
        if (W != 0 && sh < 63) T[r][v] += (W + (1ll << (sh - 1))) >> sh;
        if (se[r][v] && sh <= 32) S[r][v] += se[r][v] >> (sh - 1);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < kFxVecs; ++v) {
    if (v >= nv) continue;
    bool bad = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) bad |= fx_exponent(smax[v * 4 + e]) == kFxBad;
    const double sc = a.vscale ? a.vscale[v0 + v] : a.scale;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      double y = 0.0;
      bool ok = !bad && !f64[r];
      if (ok && top[r][v] != -0x7fffffff) {
        y = fx_to_double(T[r][v], top[r][v] - kFxBits + 1, ok);
        ok = ok && S[r][v] >= kFxLeast;
      }
      if (!ok) y = fx_row_f64(a, a.X + (long)(v0 + v) * a.ld, m, i, j, r0 + r);
      a.Y[(long)(v0 + v) * a.ld + (r0 + r) * N + m] = sc == 1.0 ? y : sc * y;
    }
  }
}

// ONE: the one-vector path (its own kernel, so that its registers do not lower the
// occupancy of the batched path)
template <bool ONE, bool ST>
__device__ __forceinline__ void matvec_cells(const MvArgs& a) {
  if (ONE) matvec_one<ST>(a);
  else matvec_multi<ST>(a);
}

template <bool ONE, bool ST>
__global__ void __launch_bounds__(kMvThreads) k_matvec(MvArgs a) { matvec_cells<ONE, ST>(a); }

// The Taylor coefficients 1 / j! of a propagation, formed on the host: a warp's
// FP64 division takes the sub-partition's FP64 pipe for ~800 cycles, and in every warp once per
// matvec it cost a small grid's matvec ~0.3 us (100 x 80, one vector: 523 -> 487 us for 250).
constexpr int kMaxOrder = 20;
struct Taylor {
  double c[kMaxOrder + 1];
};
Taylor taylor_coefficients(int order) {
  Taylor t{};
  long fact = 1;
  for (int j = 1; j <= order && j <= kMaxOrder; ++j) {
    fact *= j;
    t.c[j] = 1.0 / (double)fact;
  }
  return t;
}

// The whole Taylor propagation in one cooperative launch: the blocks are co-resident
// (cudaLaunchCooperativeKernel) and meet at a grid barrier after every matvec, instead of
// one kernel per matvec. Same per-cell arithmetic, in the same order, as launch_expm.
// vsteps (k entries, non-increasing, or null): vector c takes vsteps[c] steps, so that at
// step s only the first #{c : vsteps[c] > s} vectors advance (a contiguous prefix).
template <bool ONE, bool ST>
__global__ void __launch_bounds__(kMvThreads, 2) k_expm_coop(MvArgs base, Taylor tc, int nsteps, int order, double* v,
                                                             double* t1, double* t2, double* vout,
                                                             const int* vsteps) {
  cg::grid_group grid = cg::this_grid();
  for (int s = 0; s < nsteps; ++s) {
    if (vsteps) {
      int ka = 0;
      while (ka < base.k && vsteps[ka] > s) ++ka;
      base.k = ka;
    }
    const long n = 4 * base.N * (long)base.k;
    // order >= 2: the first matvec reads vout itself and adds nothing to it, the second
    // adds the first term before its own (the same additions in the same order as adding
    // each term in its own matvec), so no copy vout -> v closes the step
    const bool late = order >= 2;
    const double* src = late ? vout : v;
    const double* prev = nullptr;
    double c_prev = 0;
    for (int j = 1; j <= order; ++j) {
      MvArgs a = base;
      a.X = src;
      a.Y = (j % 2) ? t1 : t2;
      a.acc = (late && j == 1) ? nullptr : vout;
      a.acc_prev = prev;
      a.c_prev = c_prev;
      a.c_acc = tc.c[j];
      matvec_cells<ONE, ST>(a);
      grid.sync();
      src = a.Y;
      prev = (late && j == 1) ? a.Y : nullptr;
      c_prev = a.c_acc;
    }
    if (!late) {
      for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        v[q] = vout[q];
      grid.sync();
    }
  }
}

// ---------------------------------------------------------------------------
// Float-float Taylor propagation (the cooperative propagator's default arithmetic). The
// Taylor terms and their running sum are float-float pairs (ff.cuh) and the blocks a
// float-float copy of the Jacobian (coef_ff, split once per linearisation), so that the
// 144 multiply-adds per cell and vector run on the FP32 pipe, which this GPU issues ~70x
// faster than FP64; only the input and output vectors are FP64. Each neighbour block adds
// its four products with ff_dot4 (the products' high parts exact by FMA, the sums by
// TwoSum, one renormalisation per block), in the order of the FP64 chains (input component
// 3 down to 0), so that the one-vector and the batched paths give the same pairs. A Taylor step of degree 4-5 at the CFL time step truncates at a far larger
// relative level than this rounding; the Jacobian is a finite-difference one (~1e-8).
struct MvFf {
  const float2* coef;
  const unsigned char* nz;
  const float2* X;
  float2* Y;
  float2* acc;             // the running sum, or null
  const float2* acc_prev;  // the previous term, added into acc first (acc += c_prev acc_prev)
  double scale;            // the time step (split on the device, as the per-vector ones)
  ff c_acc, c_prev;
  const double* vscale;    // per-vector time steps, or null
  Wrap w;
  long N, ld;
  int k, transpose;
  int chunk;  // vectors per item of matvec_tile_ff
};

__device__ __forceinline__ ff ldff(const float2* p, long i) {
  const float2 v = p[i];
  return ff{v.x, v.y};
}
__device__ __forceinline__ void stff(float2* p, long i, ff v) { p[i] = make_float2(v.h, v.l); }
// the block entries, read once per cell and chunk of vectors: when they exceed L2, streaming
// loads (evict-first), so that they do not push the vectors, which every neighbour re-reads,
// out of L2; when they fit, ordinary loads, which keep them cached across the matvecs
template <bool ST>
__device__ __forceinline__ ff ldff_coef(const float2* p, long i) {
  const float2 v = ST ? __ldcs(p + i) : p[i];
  return ff{v.x, v.y};
}

// the sum of the inputs of cell (i, j)'s neighbours times zero: 0, or NaN where one is not
// finite (a cell without entries)
__device__ __forceinline__ float ff_poison_window(const MvFf& a, const float2* x, int i, int j) {
  float s = 0.0f;
  for (int q = 0; q < 9; ++q) {
    const long n = a.transpose ? a.w.nbr(i, j, 1 - q % 3, 1 - q / 3) : a.w.nbr(i, j, q % 3 - 1, q / 3 - 1);
    if (n < 0) continue;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = x[e * a.N + n];
      s = __fmaf_rn(v.x, 0.0f, __fmaf_rn(v.y, 0.0f, s));
    }
  }
  return s;
}

// one output of a term: val = scale y into Y, and the running sum
__device__ __forceinline__ void mvff_out(const MvFf& a, int vec, long o, ff y) {
  const ff sc = ff_from_double(a.vscale ? a.vscale[vec] : a.scale);
  const ff val = ff_mul(sc, y);
  stff(a.Y, o, val);
  if (a.acc) {
    ff r = ldff(a.acc, o);
    if (a.acc_prev) r = ff_add(r, ff_mul(ldff(a.acc_prev, o), a.c_prev));
    stff(a.acc, o, ff_add(r, ff_mul(val, a.c_acc)));
  }
}

// thread per (cell, output component, vector), as matvec_one
template <bool ST>
__device__ __forceinline__ void matvec_one_ff(const MvFf& a) {
  const long N = a.N;
  const long outs = 4 * N;
  // 32-bit decomposition of the work item (the host keeps the items below 2^31)
  const unsigned outs_u = (unsigned)outs, N_u = (unsigned)N, nchi_u = (unsigned)a.w.nchi;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < outs * a.k; t += (long)gridDim.x * blockDim.x) {
    const unsigned tu = (unsigned)t;
    const unsigned vec = tu / outs_u;
    const unsigned w = tu - vec * outs_u;
    const unsigned comp_u = w / N_u;
    const unsigned m = w - comp_u * N_u;
    const int comp = (int)comp_u;
    const unsigned j_u = m / nchi_u;
    const int i = (int)(m - j_u * nchi_u), j = (int)j_u;
    const float2* xv = a.X + (long)vec * a.ld;
    ff y{0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int b = q / 3 - 1, aa = q % 3 - 1;
      const long n = a.transpose ? a.w.nbr(i, j, -aa, -b) : a.w.nbr(i, j, aa, b);
      if (n < 0) continue;
      const long cell = a.transpose ? n : m;
      ff B[4], X[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int plane = a.transpose ? q * 16 + e * 4 + comp : q * 16 + comp * 4 + e;
        B[e] = ldff_coef<ST>(a.coef, (long)plane * N + cell);
        X[e] = ldff(xv, e * N + n);
      }
      y = ff_dot4(B, X, y);
    }
    mvff_out(a, (int)vec, (long)vec * a.ld + comp * N + m, y);
  }
}

// One vector on a large grid: a cell per thread and vector, one neighbour block at a time (its
// 16 pairs in registers). The 144 block entries are read once per cell and vector, so this case
// is bound by HBM, and the small register set raises the occupancy that keeps its loads in
// flight.
template <bool ST>
__device__ __forceinline__ void matvec_cell_ff(const MvFf& a) {
  const long N = a.N;
  const unsigned N_u = (unsigned)N, nchi_u = (unsigned)a.w.nchi;
  for (long w = blockIdx.x * (long)blockDim.x + threadIdx.x; w < N * a.k; w += (long)gridDim.x * blockDim.x) {
    const unsigned wu = (unsigned)w, vec = wu / N_u, m = wu - vec * N_u;
    const unsigned j_u = m / nchi_u;
    const int i = (int)(m - j_u * nchi_u), j = (int)j_u;
    const float2* x = a.X + (long)vec * a.ld;
    const long o = (long)vec * a.ld + m;
    if (!(a.nz[m] & (a.transpose ? kMaskCol : kMaskRow))) {
      const float z = ff_poison_window(a, x, i, j);
#pragma unroll
      for (int c = 0; c < 4; ++c) mvff_out(a, (int)vec, o + c * N, ff{z, 0.0f});
      continue;
    }
    ff y[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = ff{0.0f, 0.0f};
#pragma unroll 1
    for (int b = -1; b <= 1; ++b)
#pragma unroll 1
      for (int aa = -1; aa <= 1; ++aa) {
        const long n = a.transpose ? a.w.nbr(i, j, -aa, -b) : a.w.nbr(i, j, aa, b);
        if (n < 0) continue;
        const long cell = a.transpose ? n : m;
        const int q = (b + 1) * 3 + (aa + 1);
        ff B[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) B[e] = ldff_coef<ST>(a.coef, (long)(q * 16 + e) * N + cell);
        const ff xs[4] = {ldff(x, n), ldff(x, N + n), ldff(x, 2 * N + n), ldff(x, 3 * N + n)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // row c of the block, or column c for the transpose
          const ff bs[4] = {B[a.transpose ? c : c * 4], B[a.transpose ? 4 + c : c * 4 + 1],
                            B[a.transpose ? 8 + c : c * 4 + 2], B[a.transpose ? 12 + c : c * 4 + 3]};
          y[c] = ff_dot4(bs, xs, y[c]);
        }
      }
#pragma unroll
    for (int c = 0; c < 4; ++c) mvff_out(a, (int)vec, o + c * N, y[c]);
  }
}

// A batch of vectors: a block takes a tile of 32 x kFfRows cells and a chunk of up to kVecChunk
// vectors, stages the vectors' tile and halo in shared memory, and a thread forms the outputs of
// its cell for the chunk (four components each). What bounds it is the latency of the 16 pairs of a
// neighbour block (4.0 of 8.7 cycles an issue wait for loads), which four blocks of four warps on
// an SM, each at its own place, hide in part: the ~1950 FP32 instructions per cell and vector, 16
// independent chains per thread, keep that pipe 36 % and the issue slots 46 % busy. Before, a thread per component
// read the inputs from global memory for every neighbour: 38 x 4 loads of L2 per cell and vector.
// 600 x 300, 8 vectors, adjoint, us per matvec of the batch: 279 before; 178 in tiles of 32 x 8
// cells; 159 in tiles of 32 x 4 with the cells without entries left out (187 with the pairs by
// cp.async through a double buffer, 181 with an L2 prefetch of them, 174 with two components of
// eight vectors per thread and the next pairs in registers). The chunk index runs fastest, so
// that the blocks of a tile's chunks read its pairs at about the same time.
constexpr int kFfRows = 4;
constexpr int kFfHx = 34, kFfHalo = kFfHx * (kFfRows + 2), kFfThreads = 32 * kFfRows;
template <int KV>
constexpr int ff_tile_smem() { return KV * 4 * kFfHalo * (int)sizeof(float2); }
long ff_tiles(const Wrap& w) { return (long)((w.nchi + 31) / 32) * ((w.neta + kFfRows - 1) / kFfRows); }

template <int KV, bool ST>
__device__ __forceinline__ void matvec_tile_ff(const MvFf& a, float2* xs) {
  const long N = a.N;
  const int nchi = a.w.nchi, neta = a.w.neta;
  const int kv = a.chunk, chunks = (a.k + kv - 1) / kv, tx = (nchi + 31) / 32;
  const int items = tx * ((neta + kFfRows - 1) / kFfRows) * chunks;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  // block slot q of (aa, b): input cell (i + aa, j + b), or of the transpose the output cell
  // (i - aa, j - b), which owns the block
  const int sg = a.transpose ? -1 : 1;
  const long sc = a.transpose ? N : 4 * N, se = a.transpose ? 4 * N : N;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int tile = it / chunks, v0 = (it - tile * chunks) * kv, nv = min(kv, a.k - v0);
    const int i0 = (tile % tx) * 32, j0 = (tile / tx) * kFfRows;
    const int i = i0 + lane, j = j0 + row;
    const long m = i + (long)j * nchi;
    const bool in = i < nchi && j < neta;
    const bool act = in && (a.nz[m] & (a.transpose ? kMaskCol : kMaskRow));
    // cells past the grid's edge wrap where it is periodic; the others are never used
    for (int h = threadIdx.x; h < kFfHalo; h += kFfThreads) {
      int ii = i0 - 1 + h % kFfHx, jj = j0 - 1 + h / kFfHx;
      if (a.w.per_chi) ii = ii < 0 ? ii + nchi : (ii >= nchi ? ii - nchi : ii);
      if (a.w.per_eta) jj = jj < 0 ? jj + neta : (jj >= neta ? jj - neta : jj);
      if (ii < 0 || ii >= nchi || jj < 0 || jj >= neta) continue;
      const float2* x = a.X + (long)v0 * a.ld + ii + (long)jj * nchi;
#pragma unroll
      for (int v = 0; v < KV; ++v)
        if (v < nv)
#pragma unroll
          for (int e = 0; e < 4; ++e) xs[(v * 4 + e) * kFfHalo + h] = x[v * a.ld + e * N];
    }
    __syncthreads();
    if (in) {
      ff y[KV][4];
#pragma unroll
      for (int v = 0; v < KV; ++v)
#pragma unroll
        for (int c = 0; c < 4; ++c) y[v][c] = ff{0.0f, 0.0f};
#pragma unroll 1
      for (int q = 0; q < 9; ++q) {
        const int da = sg * (q % 3 - 1), db = sg * (q / 3 - 1);
        const float2* xq = xs + (lane + 1 + da) + (row + 1 + db) * kFfHx;
        const long n = a.w.nbr(i, j, da, db);
        if (n < 0) continue;
        if (act) {
          const float2* p = a.coef + (long)(q * 16) * N + (a.transpose ? n : m);
          ff B[16];
#pragma unroll
          for (int c = 0; c < 4; ++c)  // row c of the block, or column c for the transpose
#pragma unroll
            for (int e = 0; e < 4; ++e) B[c * 4 + e] = ldff_coef<ST>(p, c * sc + e * se);
#pragma unroll
          for (int v = 0; v < KV; ++v) {
            if (v >= nv) continue;
            const ff xv[4] = {ldff(xq, (v * 4) * kFfHalo), ldff(xq, (v * 4 + 1) * kFfHalo),
                              ldff(xq, (v * 4 + 2) * kFfHalo), ldff(xq, (v * 4 + 3) * kFfHalo)};
#pragma unroll
            for (int c = 0; c < 4; ++c) y[v][c] = ff_dot4(B + c * 4, xv, y[v][c]);
          }
        } else {  // a cell without entries: zero, or NaN where an input is not finite
#pragma unroll
          for (int v = 0; v < KV; ++v)
            if (v < nv)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 t = xq[(v * 4 + e) * kFfHalo];
                y[v][0].h = __fmaf_rn(t.x, 0.0f, __fmaf_rn(t.y, 0.0f, y[v][0].h));
              }
        }
      }
#pragma unroll
      for (int v = 0; v < KV; ++v)
        if (v < nv)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            mvff_out(a, v0 + v, (long)(v0 + v) * a.ld + c * N + m, act ? y[v][c] : y[v][0]);
    }
    __syncthreads();  // the next item's inputs take the shared memory
  }
}

// The cooperative propagation in float-float (degree >= 2, the late-sum order of
// k_expm_coop): the input vectors are split into the running sum, and the sum is joined
// into the FP64 output after the last step. MODE 0: matvec_tile_ff (a batch), 1: matvec_one_ff
// (few cells x vectors: ff_one), 2: matvec_cell_ff (one vector).
template <int MODE, bool ST>
__global__ void __launch_bounds__(MODE == 0 ? kFfThreads : kMvThreads, MODE == 0 ? 4 : (MODE == 2 ? 3 : 2)) k_expm_coop_ff(MvFf base, Taylor tc, int nsteps, int order, const double* xin,
                                                                double* yout, float2* t1, float2* t2, float2* vout,
                                                                const int* vsteps) {
  extern __shared__ float2 ff_tile[];
  cg::grid_group grid = cg::this_grid();
  const long nall = base.ld * (long)base.k;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < nall; q += (long)gridDim.x * blockDim.x)
    stff(vout, q, ff_from_double_checked(xin[q]));
  grid.sync();
  const int kall = base.k;
  for (int s = 0; s < nsteps; ++s) {
    if (vsteps) {
      int ka = 0;
      while (ka < kall && vsteps[ka] > s) ++ka;
      base.k = ka;
    }
    const float2* src = vout;
    const float2* prev = nullptr;
    ff c_prev{0.0f, 0.0f};
    for (int j = 1; j <= order; ++j) {
      MvFf a = base;
      a.X = src;
      a.Y = (j % 2) ? t1 : t2;
      a.acc = j == 1 ? nullptr : vout;
      a.acc_prev = prev;
      a.c_prev = c_prev;
      a.c_acc = ff_from_double(tc.c[j]);
      if (MODE == 1) matvec_one_ff<ST>(a);
      else if (MODE == 2) matvec_cell_ff<ST>(a);
      else matvec_tile_ff<kVecChunk, ST>(a, ff_tile);
      grid.sync();
      src = a.Y;
      prev = j == 1 ? a.Y : nullptr;
      c_prev = a.c_acc;
    }
  }
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < nall; q += (long)gridDim.x * blockDim.x)
    yout[q] = ff_to_double(ldff(vout, q));
}

// ---------------------------------------------------------------------------
// The float-float propagation of a small grid, resident on chip: a block owns a tile of cells for
// the whole propagation, with the tile's blocks, the terms and the running sums in shared memory
// (one thread per cell and component); from one matvec to the next only the ring of halo values
// goes through global memory, and a block waits for its neighbours' terms only, not for the
// grid. The same pairs as k_expm_coop_ff.
//
// The values of a tile's edge are published with their term's number beside each half, two 64-bit
// words {h, s} and {l, s}, and a reader of the ring polls the value itself until both words carry
// its term's number: no flag, no fence, and one block barrier per matvec. A half and its number
// are one 64-bit element of the access (.v2.b64), because the memory model orders the elements of
// a vector access in no way and keeps only each of them whole; so a number seen means its half
// seen, and the two words need no order between them. Two buffers take the terms
// in turn: a block writes term s + 2 over term s only after it has read term s + 1 of all its
// neighbours, which they form after they have read term s. The waits are bounded (kResPolls): a
// block that gives up sets the context's word in host memory (ctx_check_waits), leaves NaN and
// stops, and so do its neighbours in turn; the blocks are co-resident (a cooperative launch).
//
// What bounds it: the latency of a term, i.e. 36 float-float products in a chain of nine blocks
// (~3 instructions in four cycles with two warps per sub-partition), the write of a value and its
// neighbours' read. 100 x 80, one vector, us per matvec alone and with three contexts at once: a
// thread per output with the blocks from L2 and a grid barrier (1.15 us by itself) 5.6 and 3.4;
// resident with a flag per tile behind a fence 4.9 and 2.0; so 3.8 and 1.5. Several vectors are
// shared by groups of threads, so that neither their chains nor their polls follow one another in
// one thread: 60 x 40, twelve vectors, us for the propagation 1660 with the blocks from L2, 1500
// in one group, 762 so.
constexpr int kResThreads = 512;  // of a block with several groups: two blocks' registers per SM

struct ResTile {
  int tw, th, tx, ty;  // tile size in cells, tiles
  int groups;          // of threads, a thread per cell and component each, that share the vectors
  int polls;           // of a value, after which its reader gives up (0: at the first wait)
  unsigned* gave_up;   // set by a block that gave up (host memory)
};

long res_smem(const ResTile& t, int k) {
  const long items = 4L * t.tw * t.th, halo = (long)(t.tw + 2) * (t.th + 2);
  return (long)sizeof(float2) * (36 * items + 8L * k * halo + 2L * k * items);
}
// the tiling of at most `blocks` tiles with the fewest cells per tile (then the smallest halo)
ResTile res_tiling(const Wrap& w, int blocks, int k) {
  ResTile best{0, 0, 0, 0, 1, 0, nullptr};
  for (int tw = 4; tw <= 64; ++tw) {
    const int tx = (w.nchi + tw - 1) / tw;
    if (tx > blocks) continue;
    const int rows = blocks / tx, th = std::max(2, (w.neta + rows - 1) / rows), ty = (w.neta + th - 1) / th;
    const long c = (long)tw * th, b = (long)best.tw * best.th;
    if (!best.tw || c < b || (c == b && tw + th < best.tw + best.th)) best = ResTile{tw, th, tx, ty, 1, 0, nullptr};
  }
  best.groups = std::max(1, std::min(k, kResThreads / (4 * best.tw * best.th)));
  return best;
}

// a half of a published value with its term's number
__device__ __forceinline__ unsigned long long res_word(float x, unsigned s) {
  return (unsigned long long)s << 32 | __float_as_uint(x);
}
__device__ __forceinline__ float res_half(unsigned long long w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ unsigned res_term(unsigned long long w) { return (unsigned)(w >> 32); }

__global__ void __launch_bounds__(1024) k_expm_res_ff(MvFf a, ResTile rt, Taylor tc, int nsteps, int order, const double* xin,
                                                      double* yout, ulonglong2* g0, ulonglong2* g1, const int* vsteps) {
  extern __shared__ float2 ff_tile[];
  const long N = a.N;
  const int nchi = a.w.nchi, neta = a.w.neta;
  const int cells = rt.tw * rt.th, items = 4 * cells, hw = rt.tw + 2, halo = hw * (rt.th + 2);
  const int kall = a.k;
  float2* const cA = ff_tile;                                   // (36, items)
  float2* const xs = cA + 36 * items;                           // (2, k, 4, halo)
  float2* const sum = xs + (long)8 * kall * halo;               // (k, items)
  float2* const old = sum + (long)kall * items;                 // (k, items): the first term, added late
  const int tile = blockIdx.x, tX = tile % rt.tx, tY = tile / rt.tx;
  const int i0 = tX * rt.tw, j0 = tY * rt.th, w = min(rt.tw, nchi - i0), hgt = min(rt.th, neta - j0);
  const int tid = threadIdx.x, nt = blockDim.x, vg = tid / items, t = tid - vg * items;  // vectors vg, vg + groups, ...
  const int comp = t / cells, cell = t - comp * cells, ly = cell / rt.tw, lx = cell - ly * rt.tw;
  const int i = i0 + lx, j = j0 + ly;
  const long m = i + (long)j * nchi;
  const bool in = vg < rt.groups && lx < w && ly < hgt;
  const bool edge = in && (lx == 0 || ly == 0 || lx == w - 1 || ly == hgt - 1);
  const int sg = a.transpose ? -1 : 1;
  unsigned ok = 0;  // bit q: the neighbour exists
  if (in) {
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const long n = a.w.nbr(i, j, sg * (q % 3 - 1), sg * (q / 3 - 1));
      if (n < 0) continue;
      ok |= 1u << q;
      if (vg > 0) continue;  // the first group brings the blocks for all
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // row comp of the block (columns e), or column comp of it for the transpose
        const int plane = a.transpose ? q * 16 + e * 4 + comp : q * 16 + comp * 4 + e;
        cA[(q * 4 + e) * items + t] = a.coef[(long)plane * N + (a.transpose ? n : m)];
      }
    }
  }
  const int own = comp * halo + (lx + 1) + (ly + 1) * hw;
  unsigned seq = 1;  // the number of the term being formed; its buffer is seq & 1
  // the ring of the term just published; false when a wait gave up
  const int ring = 2 * (w + 2) + 2 * hgt;
  auto exchange = [&](int ka) -> bool {
    const ulonglong2* g = seq & 1 ? g1 : g0;
    float2* x = xs + (long)(seq & 1) * kall * 4 * halo;
    bool good = rt.polls > 0;
    for (int r = tid; r < ring * 4 * ka; r += nt) {  // the vectors spread over the threads too: a poll is a wait
      const int ve = r / ring, v = ve >> 2, e = ve & 3, c = r - ve * ring;
      int hx, hy;
      if (c < 2 * (w + 2)) {
        hy = c < w + 2 ? 0 : hgt + 1;
        hx = c < w + 2 ? c : c - (w + 2);
      } else {
        const int c2 = c - 2 * (w + 2);
        hy = 1 + (c2 >> 1);
        hx = c2 & 1 ? w + 1 : 0;
      }
      int ii = i0 - 1 + hx, jj = j0 - 1 + hy;
      const bool wi = ii < 0 || ii >= nchi, wj = jj < 0 || jj >= neta;
      if ((wi && !a.w.per_chi) || (wj && !a.w.per_eta) || (wi && wj)) continue;  // no such input (Wrap::nbr)
      if (wi) ii = ii < 0 ? ii + nchi : ii - nchi;
      if (wj) jj = jj < 0 ? jj + neta : jj - neta;
      const ulonglong2* p = g + v * a.ld + e * N + ii + (long)jj * nchi;
      unsigned long long uh, ul;
      int polls = 0;
      do {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(uh), "=l"(ul) : "l"(p) : "memory");
      } while ((res_term(uh) != seq || res_term(ul) != seq) && ++polls < rt.polls && good);
      good = good && res_term(uh) == seq && res_term(ul) == seq;
      x[((long)v * 4 + e) * halo + hx + hy * hw] = make_float2(res_half(uh), res_half(ul));
    }
    if (!__syncthreads_and(good)) {
      if (tid == 0) *reinterpret_cast<volatile unsigned*>(rt.gave_up) = 1u;
      return false;
    }
    ++seq;
    return true;
  };
  // a value of the term: into the tile's shared copy and, on the tile's edge, published
  auto put = [&](int v, ff val) {
    xs[((long)(seq & 1) * kall + v) * 4 * halo + own] = make_float2(val.h, val.l);
    if (edge)
      asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"((seq & 1 ? g1 : g0) + v * a.ld + comp * N + m),
                   "l"(res_word(val.h, seq)), "l"(res_word(val.l, seq))
                   : "memory");
  };
  if (in)
    for (int v = vg; v < kall; v += rt.groups) {
      const ff x = ff_from_double_checked(xin[v * a.ld + comp * N + m]);
      stff(sum, v * items + t, x);
      put(v, x);
    }
  // (a propagation that gave up leaves NaN)
  auto fail = [&]() {
    if (in)
      for (int v = vg; v < kall; v += rt.groups) yout[v * a.ld + comp * N + m] = __longlong_as_double(0x7ff8000000000000LL);
  };
  if (!exchange(kall)) return fail();
  int ka = kall;
  for (int s = 0; s < nsteps; ++s) {
    if (vsteps) {
      ka = 0;
      while (ka < kall && vsteps[ka] > s) ++ka;
    }
    ff c1{0.0f, 0.0f};
    for (int jt = 1; jt <= order; ++jt) {
      const ff c = ff_from_double(tc.c[jt]);
      const bool last = jt == order;
      if (in)
        for (int v = vg; v < ka; v += rt.groups) {
          const float2* x = xs + ((long)((seq - 1) & 1) * kall + v) * 4 * halo + (lx + 1) + (ly + 1) * hw;
          ff y{0.0f, 0.0f};
#pragma unroll
          for (int q = 0; q < 9; ++q) {
            if (!(ok >> q & 1)) continue;
            const float2* xq = x + sg * (q % 3 - 1) + sg * (q / 3 - 1) * hw;
            ff B[4], X[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              B[e] = ldff(cA, (q * 4 + e) * items + t);
              X[e] = ldff(xq, e * halo);
            }
            y = ff_dot4(B, X, y);
          }
          // mvff_out's term and running sum
          const ff val = ff_mul(ff_from_double(a.vscale ? a.vscale[v] : a.scale), y);
          if (jt == 1) {
            stff(old, v * items + t, val);
          } else {
            ff r = ldff(sum, v * items + t);
            if (jt == 2) r = ff_add(r, ff_mul(ldff(old, v * items + t), c1));
            r = ff_add(r, ff_mul(val, c));
            stff(sum, v * items + t, r);
            if (last) put(v, r);
          }
          if (!last) put(v, val);
        }
      c1 = c;
      if (last && s + 1 == nsteps) break;
      if (!exchange(ka)) return fail();
    }
  }
  if (in)
    for (int v = vg; v < kall; v += rt.groups) yout[v * a.ld + comp * N + m] = ff_to_double(ldff(sum, v * items + t));
}

__global__ void k_coef_to_ff(const double* __restrict__ c, float2* __restrict__ f, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
    stff(f, q, ff_from_double_checked(c[q]));
}

__global__ void k_copy(const double* __restrict__ s, double* __restrict__ d, long n) {
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) d[k] = s[k];
}

// per-cell block layout <-> plane layout
// (nz, zeroed: byte (input variable) N + m set where cell m has a non-zero entry of it)
__global__ void k_blocks_to_planes(const double* blk, double* pl, unsigned char* nz, long N) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < N * 144; t += (long)gridDim.x * blockDim.x) {
    const long m = t / 144;
    const int e = (int)(t % 144);
    const double c = blk[t];
    pl[(long)e * N + m] = c;
    if (((unsigned long long)__double_as_longlong(c) << 1) != 0) nz[(e & 3) * N + m] = 1;
  }
}
// the masks of the matvecs (kMaskRow, kMaskCol) from the 4 x N bytes of the input variables
__global__ void k_masks(unsigned char* mask, const unsigned char* nz, Wrap w, long N) {
  for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < N; m += (long)gridDim.x * blockDim.x) {
    const int j = (int)((unsigned)m / (unsigned)w.nchi), i = (int)((unsigned)m - (unsigned)j * (unsigned)w.nchi);
    auto any = [&](long c) { return nz[c] | nz[N + c] | nz[2 * N + c] | nz[3 * N + c]; };
    unsigned r = any(m) ? kMaskRow : 0;
    for (int q = 0; q < 9; ++q) {
      const long n = w.nbr(i, j, 1 - q % 3, 1 - q / 3);
      if (n >= 0 && any(n)) r |= kMaskCol;
    }
    mask[m] = (unsigned char)r;
  }
}
__global__ void k_planes_to_blocks(const double* pl, double* blk, long N) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < N * 144; t += (long)gridDim.x * blockDim.x) {
    const long m = t / 144;
    const int e = (int)(t % 144);
    blk[t] = pl[(long)e * N + m];
  }
}


// ---------------------------------------------------------------------------
// Krylov helpers on device-resident bases. Reductions are deterministic: stage 1
// gives each (block, column) a fixed slice of rows and a fixed warp-shuffle tree,
// stage 2 sums the block partials of a column in a fixed order.
constexpr int kDotBlocks = 296;  // 2 x 148-152 SMs
constexpr int kDotThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// partial[j * kDotBlocks + b] = Σ_{rows of block b} A[i + j lda] * w[i]
__global__ void __launch_bounds__(kDotThreads) k_dot_stage1(const double* A, long lda, const double* w, long n,
                                                            double* partial) {
  const int j = blockIdx.y;
  const double* a = A + (long)j * lda;
  double acc = 0;
  for (long i = blockIdx.x * (long)kDotThreads + threadIdx.x; i < n; i += (long)kDotBlocks * kDotThreads)
    acc = fma(a[i], w[i], acc);
  acc = warp_sum(acc);
  __shared__ double red[kDotThreads / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < kDotThreads / 32 ? red[threadIdx.x] : 0.0;
    v = warp_sum(v);
    if (threadIdx.x == 0) partial[(long)j * kDotBlocks + blockIdx.x] = v;
  }
}

// out[j] (+)= Σ_b partial[j * kDotBlocks + b]; mode 0 store, 1 add
__global__ void k_dot_stage2(const double* partial, double* out, int mode) {
  const int j = blockIdx.x;
  double acc = 0;
  for (int b = threadIdx.x; b < kDotBlocks; b += 32) acc += partial[(long)j * kDotBlocks + b];
  acc = warp_sum(acc);
  if (threadIdx.x == 0) out[j] = mode ? out[j] + acc : acc;
}

// w -= A[:, 0:m] h
__global__ void __launch_bounds__(256) k_gemv_sub(const double* A, long lda, long n, int m, const double* h, double* w) {
  extern __shared__ double sh[];
  for (int j = threadIdx.x; j < m; j += blockDim.x) sh[j] = h[j];
  __syncthreads();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int j = 0; j < m; ++j) acc = fma(A[i + (long)j * lda], sh[j], acc);
    w[i] -= acc;
  }
}

// dst = src / sqrt(nrm2[0])
__global__ void k_normalize(const double* src, double* dst, long n, const double* nrm2) {
  const double s = 1.0 / sqrt(nrm2[0]);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) dst[i] = src[i] * s;
}

// out[:, c] = A[:, 0:m] Q[:, c] for c < k (Q column-major m x k, in global memory)
__global__ void __launch_bounds__(128) k_rotate(const double* A, long lda, long n, int m, int k, const double* Q,
                                                double* out, long ldo) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    for (int c0 = 0; c0 < k; c0 += 8) {
      double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      const int nc = min(8, k - c0);
      for (int j = 0; j < m; ++j) {
        const double a = A[i + (long)j * lda];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < nc) acc[c] = fma(a, Q[j + (long)(c0 + c) * m], acc[c]);
      }
      for (int c = 0; c < nc; ++c) out[i + (long)(c0 + c) * ldo] = acc[c];
    }
  }
}

// y = blockdiag(B) x with B row-major 4x4 per cell (N x 16), vectors [v0; v1; v2; v3] x N, k columns
__global__ void k_block4(const double* B, const double* x, double* y, long N, int k) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < N * k; t += (long)gridDim.x * blockDim.x) {
    const long m = t % N;
    const long col = t / N;
    const double* xc = x + col * 4 * N;
    double* yc = y + col * 4 * N;
    const double x0 = xc[m], x1 = xc[N + m], x2 = xc[2 * N + m], x3 = xc[3 * N + m];
    const double* b = B + m * 16;
#pragma unroll
    for (int r = 0; r < 4; ++r) yc[r * N + m] = fma(b[4 * r], x0, fma(b[4 * r + 1], x1, fma(b[4 * r + 2], x2, b[4 * r + 3] * x3)));
  }
}

// Tail of vectors of 4N + nt entries: y = B x on the cells (k_block4), y = t x on the tail.
__global__ void k_block4_tail(const double* B, const double* tail, const double* x, double* y, long N, long nt,
                              int k) {
  const long ld = 4 * N + nt;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < N * k; t += (long)gridDim.x * blockDim.x) {
    const long m = t % N;
    const long col = t / N;
    const double* xc = x + col * ld;
    double* yc = y + col * ld;
    const double x0 = xc[m], x1 = xc[N + m], x2 = xc[2 * N + m], x3 = xc[3 * N + m];
    const double* b = B + m * 16;
#pragma unroll
    for (int r = 0; r < 4; ++r) yc[r * N + m] = fma(b[4 * r], x0, fma(b[4 * r + 1], x1, fma(b[4 * r + 2], x2, b[4 * r + 3] * x3)));
  }
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < nt * k; t += (long)gridDim.x * blockDim.x) {
    const long m = t % nt, col = t / nt;
    y[col * ld + 4 * N + m] = tail[m] * x[col * ld + 4 * N + m];
  }
}

// ---------------------------------------------------------------------------
// Shock-position blocks (perturb_shock, LINEARIZE_EQUATIONS_NO_DISCONTINUITY.jl:140-274).

// PERTURB_SHOCK (:906-913) direction of every point: ang = beta - pi/2 - phi with
// phi = atan(rho_v_0, rho_u_0), so (cos ang, sin ang) = (sin(beta - phi), -cos(beta - phi)),
// from the sine and cosine of beta that the last shock update of S stored.
__global__ void k_shock_dir(const double* beta, double* dir, int nchi, double cph, double sph) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchi) return;
  const double sb = beta[i], cb = beta[nchi + i];
  dir[i] = sb * cph - cb * sph;
  dir[nchi + i] = -(cb * cph + sb * sph);
}

// Y's shock points = S's, point p displaced by eps along its PERTURB_SHOCK direction.
// Lane z of a batched launch displaces point first + z.
__global__ void k_perturb_point(ShockPts S, ShockPts Y, const double* dir, int nchi, int first, double eps,
                                long lane) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchi) return;
  const long off = blockIdx.z * lane;
  Y = ShockPts{Y.x + off, Y.y + off, Y.chi + off, Y.eta + off};
  double x = S.x[i], y = S.y[i];
  if (i == first + (int)blockIdx.z) {
    x = x + eps * dir[i];
    y = y + eps * dir[nchi + i];
  }
  Y.x[i] = x;
  Y.y[i] = y;
  Y.chi[i] = S.chi[i];
  Y.eta[i] = S.eta[i];
}

// A21 column (j, var) of every point: (speed_i(x + eps e) - speed_i(x)) / eps
// (GET_OUTPUT_INDEXING_A21, :800-820; REMOVE_BASE_OUTPUT, :935-946)
__global__ void k_gather_a21(const double* rel, const double* rel_b, double* a21, int nchi, int first, double eps,
                             long lane) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchi) return;
  a21[i * 8 + first + blockIdx.z] = (rel[blockIdx.z * lane + i] - rel_b[i]) / eps;
}

// A12 and A22 columns of point p (GET_OUTPUT_INDEXING_A12_A22, :854-903): the flux of the
// cells (i, sc_i - 1) and the shock speeds of every column.
struct Flux4 {
  const double* v[4];
};
__global__ void k_gather_a12(Flux4 Fp, Flux4 Fb, const double* rel, const double* rel_b, const int* rows,
                             double* a12, double* a22, int nchi, int first, double eps, long lane) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchi) return;
  const long off = blockIdx.z * lane;
  const int p = first + blockIdx.z;
  const long m = i + (long)(rows[i] - 2) * nchi;
#pragma unroll
  for (int v = 0; v < 4; ++v) a12[((long)v * nchi + i) * nchi + p] = (Fp.v[v][off + m] - Fb.v[v][m]) / eps;
  a22[(long)i * nchi + p] = (rel[off + i] - rel_b[i]) / eps;
}

// out (cols x rows) = in (rows x cols) transposed, both row-major
__global__ void k_transpose(const double* in, double* out, long rows, long cols) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < rows * cols; t += (long)gridDim.x * blockDim.x) {
    const long r = t / cols, c = t % cols;
    out[c * rows + r] = in[t];
  }
}

struct ShockMvArgs {
  ShockJac sj;
  const double* X;
  double* Y;
  long N, ld;
  double scale;
  int nchi, k, transpose;
};

// The shock-block part of y = scale A x (after the stencil matvec has written y's cell
// rows). Block (bx, col) stages what every row of vector col reads — r, and for the
// transpose the cells (i, sc_i - 1) of q — in shared memory, then gives each of its warps
// whole output rows: lanes over the row's entries (coalesced), a fixed shuffle tree.
//   forward:   rows (v, i) of A12 add scale (A12 r) into the flux rows (i, sc_i - 1);
//              speed rows i set y_r = scale (A21 q + A22 r).
//   transpose: speed rows p set y_r = scale (A12ᵀ q + A22ᵀ r); lanes 0-7 of the same warp
//              add scale A21ᵀ r into the cells (p, sc_p - j).
constexpr int kShockThreads = 128;
__host__ __device__ inline long shock_mv_smem(int nchi, int transpose) {
  return (long)(transpose ? 5 : 1) * nchi * (long)sizeof(double);
}

// Σ_p a[p] b[p] over the lane's entries p = lane, lane + 32, ... (one FMA chain: the FP64
// pipe, not the loads, bounds these rows; partial sums would add FP64 instructions)
__device__ __forceinline__ double lane_dot(const double* __restrict__ a, const double* b, int n, int lane) {
  double t = 0;
#pragma unroll 8
  for (int p = lane; p < n; p += 32) t = fma(a[p], b[p], t);
  return t;
}

__global__ void __launch_bounds__(kShockThreads) k_shock_mv(ShockMvArgs a) {
  extern __shared__ double sh[];
  const int lane = threadIdx.x & 31;
  const int nchi = a.nchi;
  const long N = a.N;
  const int* rows = a.sj.rows;
  const long col = blockIdx.y;
  const double* x = a.X + col * a.ld;
  double* y = a.Y + col * a.ld;
  const double* xr = x + 4 * N;
  double* sr = sh;  // r
  if (a.transpose) {
    sr = sh + 4 * nchi;
    for (int t = threadIdx.x; t < 4 * nchi; t += blockDim.x) {
      const int v = t / nchi, i = t % nchi;
      sh[t] = x[v * N + i + (long)(rows[i] - 2) * nchi];
    }
  }
  for (int t = threadIdx.x; t < nchi; t += blockDim.x) sr[t] = xr[t];
  __syncthreads();
  const int per = a.transpose ? nchi : 5 * nchi;
  const int wpb = blockDim.x / 32;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < per; r += gridDim.x * wpb) {
    double s = 0;
    if (!a.transpose) {
      if (r < 4 * nchi) {
        s = warp_sum(lane_dot(a.sj.a12 + (long)r * nchi, sr, nchi, lane));
        if (lane == 0) {
          const int v = r / nchi, i = r % nchi;
          y[v * N + i + (long)(rows[i] - 2) * nchi] += a.scale * s;
        }
      } else {
        const int i = r - 4 * nchi;
        s = lane_dot(a.sj.a22 + (long)i * nchi, sr, nchi, lane);
        if (lane < 8) {
          const int j = lane / 4 + 1, v = lane % 4;
          s = fma(a.sj.a21[i * 8 + lane], x[v * N + i + (long)(rows[i] - 1 - j) * nchi], s);
        }
        s = warp_sum(s);
        if (lane == 0) y[4 * N + i] = a.scale * s;
      }
    } else {
      const int p = r;
      s = lane_dot(a.sj.a12t + (long)p * 4 * nchi, sh, 4 * nchi, lane);
      s += lane_dot(a.sj.a22t + (long)p * nchi, sr, nchi, lane);
      s = warp_sum(s);
      if (lane == 0) y[4 * N + p] = a.scale * s;
      if (lane < 8) {
        const int j = lane / 4 + 1, v = lane % 4;
        y[v * N + p + (long)(rows[p] - 1 - j) * nchi] += a.scale * (a.sj.a21[p * 8 + lane] * sr[p]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Upstream-boundary operator B (freestream receptivity, Freestream_receptivity/LINEARIZE_B.jl).

// Per-column upstream state: the freestream, with variable `var` of the columns i = colour
// (mod 3) raised by eps (LINEARIZE_B.jl:49-70; var < 0: the unperturbed state).
// Lane z of a batched launch (lane > 0) raises variable (first + z) / 3 of colour (first + z) % 3.
__global__ void k_up_cols(double* cols, int nchi, double r0, double ru0, double rv0, double rE0, int var,
                          int colour, double eps, int first = 0, long lane = 0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchi) return;
  cols += blockIdx.z * lane;
  if (lane) {
    var = (first + (int)blockIdx.z) / 3;
    colour = (first + (int)blockIdx.z) % 3;
  }
  const double f[4] = {r0, ru0, rv0, rE0};
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const double hit = (v == var && i % 3 == colour) ? 1.0 : 0.0;
    cols[v * nchi + i] = f[v] + eps * hit;
  }
}

// GET_BLOCK (LINEARIZE_B.jl:186-253): the raised column n = m + d (d in -1, 0, 1) of output
// column m is the one of this colour; its entries are the flux change of the cell
// (m, sc_m - 1) and the change of speed m over eps.
__global__ void k_gather_b(Flux4 Fp, Flux4 Fb, const double* rel, const double* rel_b, const int* rows, double* bq,
                           double* bs, int nchi, int first, double eps, long lane) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= nchi) return;
  const long off = blockIdx.z * lane;
  const int var = (first + (int)blockIdx.z) / 3, colour = (first + (int)blockIdx.z) % 3;
  int d = 2;  // the offset in -1..1 whose column has this colour
  for (int dd = -1; dd <= 1; ++dd)
    if (((m + dd) % 3 + 3) % 3 == colour) d = dd;
  const int n = m + d;
  if (d == 2 || n < 0 || n >= nchi) return;
  const long cell = m + (long)(rows[m] - 2) * nchi;
#pragma unroll
  for (int vo = 0; vo < 4; ++vo)
    bq[((m * 3 + d + 1) * 4 + vo) * 4 + var] = (Fp.v[vo][off + cell] - Fb.v[vo][cell]) / eps;
  if (bs) bs[(m * 3 + d + 1) * 4 + var] = (rel[off + m] - rel_b[m]) / eps;
}

struct RecArgs {
  const double* X;
  double* Y;
  const double *bq, *bs, *w;
  const int* rows;
  long N, ld, nop;  // vector stride; nop = start of the freestream blocks
  double scale;
  int nchi, nw, k, adjoint, shock;
};

// The freestream part of the receptivity operator L_ = [L, B ... B; 0, diag(-i w_k I)]
// (LINEARIZE_L_.jl:60-68) on k complex vectors, each stored as its real and imaginary
// parts (real vectors 2c and 2c + 1 of stride ld), after the matvec with L has written the
// downstream rows. Forward: the flux rows (m, sc_m - 1) (and speed rows) add B (sum_k u_k);
// the freestream rows are -i w_k u_k. Adjoint (the conjugate transpose): every freestream
// block gets B^T q + i w_k u_k.
__global__ void __launch_bounds__(256) k_recept_mv(RecArgs a) {
  const int nchi = a.nchi;
  const long p4 = 4L * nchi;
  const long nre = 2L * a.k;
  const long items = a.adjoint ? nre * p4 : nre * nchi + nre * a.nw * p4;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < items; t += (long)gridDim.x * blockDim.x) {
    if (a.adjoint) {
      const long r = t / p4;
      const int e = (int)(t % p4), vin = e / nchi, n = e % nchi;
      const double* x = a.X + r * a.ld;
      const double* xo = a.X + (r ^ 1) * a.ld;
      double* y = a.Y + r * a.ld;
      double bt = 0;
      for (int m = max(n - 1, 0); m <= min(n + 1, nchi - 1); ++m) {
        const int slot = (m * 3 + (n - m) + 1) * 4;
        const long cell = m + (long)(a.rows[m] - 2) * nchi;
#pragma unroll
        for (int vo = 0; vo < 4; ++vo) bt = fma(a.bq[(slot + vo) * 4 + vin], x[vo * a.N + cell], bt);
        if (a.shock) bt = fma(a.bs[slot + vin], x[4 * a.N + m], bt);
      }
      const double sg = (r & 1) ? 1.0 : -1.0;  // i w u: real part -w u_im, imaginary part +w u_re
      for (int kk = 0; kk < a.nw; ++kk) {
        const long idx = a.nop + kk * p4 + e;
        y[idx] = a.scale * fma(sg * a.w[kk], xo[idx], bt);
      }
    } else if (t < nre * nchi) {
      const long r = t / nchi;
      const int m = (int)(t % nchi);
      const double* x = a.X + r * a.ld;
      double* y = a.Y + r * a.ld;
      double acc[4] = {0, 0, 0, 0}, accs = 0;
      for (int dd = -1; dd <= 1; ++dd) {
        const int n = m + dd;
        if (n < 0 || n >= nchi) continue;
        const int slot = (m * 3 + dd + 1) * 4;
#pragma unroll
        for (int vin = 0; vin < 4; ++vin) {
          double u = 0;
          for (int kk = 0; kk < a.nw; ++kk) u += x[a.nop + kk * p4 + vin * nchi + n];
#pragma unroll
          for (int vo = 0; vo < 4; ++vo) acc[vo] = fma(a.bq[(slot + vo) * 4 + vin], u, acc[vo]);
          accs = fma(a.bs[slot + vin], u, accs);
        }
      }
      const long cell = m + (long)(a.rows[m] - 2) * nchi;
#pragma unroll
      for (int vo = 0; vo < 4; ++vo) y[vo * a.N + cell] += a.scale * acc[vo];
      if (a.shock) y[4 * a.N + m] += a.scale * accs;
    } else {
      const long u = t - nre * nchi;
      const long r = u / (a.nw * p4);
      const long f = u % (a.nw * p4);
      const int kk = (int)(f / p4);
      const long idx = a.nop + f;
      const double sg = (r & 1) ? -1.0 : 1.0;  // -i w u: real part +w u_im, imaginary part -w u_re
      a.Y[r * a.ld + idx] = a.scale * (sg * a.w[kk] * a.X[(r ^ 1) * a.ld + idx]);
    }
  }
}

// t *= c, acc += t (n entries): one term of EXPONENTIAL!'s recurrence (CONSTRUCT_C.jl:78-111)
__global__ void k_scale_acc(double* t, double* acc, double c, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
    const double v = t[q] * c;
    t[q] = v;
    acc[q] += v;
  }
}

// acc += c t (n entries)
__global__ void k_axpy(double* acc, const double* t, double c, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
    acc[q] = fma(t[q], c, acc[q]);
}

int grid_for(long n, int threads) {
  long b = (n + threads - 1) / threads;
  const long cap = 152L * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

// ---------------------------------------------------------------------------
// The Taylor propagation of the extended operators (the shock-position unknowns, the
// receptivity operator, or both) in one cooperative launch, FP64: per term one pass over all
// outputs and one grid barrier, instead of three or four launches (stencil, shock rows,
// receptivity rows, accumulation) that each wait for the last.
//
// So that a term needs a single pass, every output is formed whole by one owner: a thread per
// (cell, component, vector) for the stencil outputs, as matvec_one, and a warp for the outputs
// with long rows, their stencil products and the rows' products shared over the lanes: a
// column's cell (i, sc_i - 1) that A12 writes with its shock speed, each component of that cell
// where B writes it, and the adjoint's tails. The
// warps take the long rows first. What bounds it: the FP64 pipe (144 FMA per cell and vector,
// 4.6 us at 160 x 97) and the latency of one pass and a barrier per term; 8 warps per SM keep
// that pipe busy (a dependent FP64 instruction waits about as long as one issues) and leave
// room for the propagations of other contexts (two blocks per SM: a single context's term 20 %
// faster, three contexts' 1.8 times slower). A term of one context alone, and of three at once
// per context: adjoint with the shock unknowns, 160 x 97, 17.0 -> 11.7 us and 10.8 -> 6.3;
// receptivity 98 x 73 with 24 frequencies 38.6 -> 17.6 and 22.1 -> 8.0.
struct ExtArgs {
  const double* coef;
  ShockJac sj;
  const double *bq, *bs, *w;  // receptivity: B and the frequencies (w null: no receptivity)
  const int* brows;
  Wrap wr;
  long N, ld, nop;  // ld: vector stride; nop: start of the freestream blocks
  double dt;
  int nchi, k, nw, shock, divide;  // k real vectors; divide: EXPONENTIAL!'s term / j recurrence
};

struct ExtTerm {
  const double* X;
  double* Y;
  double* acc;         // the running sum, or null (the first term is added one term late)
  const double* prev;  // the previous term, added first, or null
  double c, c_prev;
};

__device__ __forceinline__ void ext_out(const ExtArgs& a, const ExtTerm& t, long o, double y) {
  double val = a.dt * y;
  if (a.divide) val *= t.c;
  t.Y[o] = val;
  if (!t.acc) return;
  double r = t.acc[o];
  if (a.divide) {
    if (t.prev) r += t.prev[o];
    t.acc[o] = r + val;
  } else {
    if (t.prev) r = fma(t.prev[o], t.c_prev, r);
    t.acc[o] = fma(val, t.c, r);
  }
}

// The warp's sums of four values: lanes 0, 8, 16, 24 end with those of s[0], s[1], s[2], s[3]
// (two values folded per lane and step while there are several: 6 additions for the four, FP64
// ones, instead of 20).
__device__ __forceinline__ double warp_sum4(const double (&s)[4], int lane) {
  const bool hi = lane & 16, hi2 = lane & 8;
  const double a = (hi ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[2], 16);
  const double b = (hi ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, hi ? s[1] : s[3], 16);
  double r = (hi2 ? b : a) + __shfl_xor_sync(0xffffffffu, hi2 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// the lane's share of the four stencil rows of cell m = (i, j)
__device__ __forceinline__ void ext_stencil_lane4(const ExtArgs& a, const double* x, long m, int i, int j, int lane,
                                                  double (&s)[4]) {
#pragma unroll 1
  for (int e = lane; e < 36; e += 32) {
    const int q = e >> 2, v = e & 3;
    const long n = a.wr.nbr(i, j, q % 3 - 1, q / 3 - 1);
    if (n < 0) continue;
    const double xv = x[v * a.N + n];
#pragma unroll
    for (int c = 0; c < 4; ++c) s[c] = fma(a.coef[(long)(q * 16 + c * 4 + v) * a.N + m], xv, s[c]);
  }
}
// the lane's share of the stencil row of component c
__device__ __forceinline__ double ext_stencil_lane(const ExtArgs& a, const double* x, int c, long m, int i, int j,
                                                   int lane, double s) {
  for (int e = lane; e < 36; e += 32) {
    const int q = e >> 2, v = e & 3;
    const long n = a.wr.nbr(i, j, q % 3 - 1, q / 3 - 1);
    if (n >= 0) s = fma(a.coef[(long)(q * 16 + c * 4 + v) * a.N + m], x[v * a.N + n], s);
  }
  return s;
}

// the lane's share of Σ_d Σ_vin b[d * db + vin] Σ_k u_k,vin(m + d - 1): a row of B (b: its first
// entry) on the freestream blocks u of x
__device__ __forceinline__ double ext_upstream_lane(const ExtArgs& a, const double* x, const double* b, int db, int m,
                                                    int lane, double s) {
  const int p4 = 4 * a.nchi;
#pragma unroll 4
  for (int e = lane; e < 12 * a.nw; e += 32) {
    const int kk = e / 12, r = e - 12 * kk, d = r >> 2, vin = r & 3, n = m + d - 1;
    if (n >= 0 && n < a.nchi) s = fma(b[d * db + vin], x[a.nop + (long)kk * p4 + vin * a.nchi + n], s);
  }
  return s;
}

template <bool T>
__device__ __forceinline__ void ext_pass(const ExtArgs& a, const ExtTerm& t) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int nchi = a.nchi, p4 = 4 * nchi;
  const long N = a.N;
  const unsigned N_u = (unsigned)N, nchi_u = (unsigned)nchi;
  const bool rec = a.w != nullptr;
  // the warps' items: columns of the shock unknowns (the speeds, forward without B also the
  // cells (i, sc_i - 1); the adjoint's tail rows), with B the rows of those cells (A12's, then
  // B's: a row each, because B's 12 products per frequency make them the longest items),
  // freestream entries (by 32; the adjoint: a warp per entry of a block, lanes over the
  // frequencies), stencil outputs (by 32)
  const int r_sh = a.shock ? a.k * nchi : 0;
  const int r_a12 = !T && rec && a.shock ? a.k * p4 : 0;
  const int r_b = !T && rec ? a.k * p4 : 0;
  const int per_free = T ? p4 : (a.nw * p4 + 31) / 32;
  const int r_free = rec ? a.k * per_free : 0;
  const int b0 = r_sh, b1 = b0 + r_a12, b2 = b1 + r_b, b3 = b2 + r_free;
  const unsigned outs = 4u * N_u;
  const int items = b3 + (int)((outs * (unsigned)a.k + 31) / 32);
  for (int it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += warps) {
    if (it >= b3) {
      const unsigned g = (unsigned)(it - b3) * 32 + lane;
      if (g >= outs * (unsigned)a.k) continue;
      const unsigned vec = g / outs, w = g - vec * outs, comp = w / N_u, m = w - comp * N_u;
      const int j = (int)(m / nchi_u), i = (int)(m - (unsigned)j * nchi_u);
      if (!T && ((a.shock && j == a.sj.rows[i] - 2) || (rec && j == a.brows[i] - 2))) continue;
      const double* x = t.X + vec * a.ld;
      double y = 0, B[2][4], V[2][4];
      bool ok[2];
      auto load = [&](int q, int slot) {
        const int b = q / 3 - 1, aa = q % 3 - 1;
        const long n = T ? a.wr.nbr(i, j, -aa, -b) : a.wr.nbr(i, j, aa, b);
        const long cell = T ? n : (long)m;
        ok[slot] = n >= 0;
        if (n >= 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const long plane = T ? q * 16 + e * 4 + (int)comp : q * 16 + (int)comp * 4 + e;
            B[slot][e] = a.coef[plane * N + cell];
            V[slot][e] = x[e * N + n];
          }
        }
      };
      load(0, 0);
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const int c = q & 1;
        if (q + 1 < 9) load(q + 1, c ^ 1);
        if (!ok[c]) continue;
        y = fma(B[c][0], V[c][0], fma(B[c][1], V[c][1], fma(B[c][2], V[c][2], fma(B[c][3], V[c][3], y))));
      }
      if (T && a.shock) {  // A21^T r into the two cells below the shocked cell
        const int d = a.sj.rows[i] - 2 - j;
        if (d == 0 || d == 1) y = fma(a.sj.a21[i * 8 + d * 4 + comp], x[4 * N + i], y);
      }
      ext_out(a, t, vec * a.ld + w, y);
    } else if (T && it < b0) {  // A12^T q + A22^T r
      const int vec = it / nchi, i = it - vec * nchi;
      const double* x = t.X + vec * a.ld;
      double s = lane_dot(a.sj.a22t + (long)i * nchi, x + 4 * N, nchi, lane);
      const double* row = a.sj.a12t + (long)i * p4;
#pragma unroll 2
      for (int p = lane; p < nchi; p += 32) {
        const double* xp = x + p + (long)(a.sj.rows[p] - 2) * nchi;
#pragma unroll
        for (int v = 0; v < 4; ++v) s = fma(row[v * nchi + p], xp[v * N], s);
      }
      s = warp_sum(s);
      if (lane == 0) ext_out(a, t, vec * a.ld + 4 * N + i, s);
    } else if (it < b0) {
      // column i: the speed A21 q + A22 r (+ B's), and without B the cell (i, sc_i - 1), whose
      // stencil rows A12 r joins
      const int vec = it / nchi, i = it - vec * nchi, j = a.sj.rows[i] - 2;
      const long m = i + (long)j * nchi;
      const double* x = t.X + vec * a.ld;
      const double* xr = x + 4 * N;
      double spd = 0;
      if (lane < 8) spd = a.sj.a21[i * 8 + lane] * x[(lane & 3) * N + m - (long)(lane >> 2) * nchi];
      if (rec) {
        spd += lane_dot(a.sj.a22 + (long)i * nchi, xr, nchi, lane);
        spd = ext_upstream_lane(a, x, a.bs + i * 12, 4, i, lane, spd);
      } else {
        double s[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int p = lane; p < nchi; p += 32) {
          const double rp = xr[p];
          spd = fma(a.sj.a22[(long)i * nchi + p], rp, spd);
#pragma unroll
          for (int v = 0; v < 4; ++v) s[v] = fma(a.sj.a12[((long)v * nchi + i) * nchi + p], rp, s[v]);
        }
        ext_stencil_lane4(a, x, m, i, j, lane, s);
        const double y = warp_sum4(s, lane);
        if ((lane & 7) == 0) ext_out(a, t, vec * a.ld + (lane >> 3) * N + m, y);
      }
      spd = warp_sum(spd);
      if (lane == 0) ext_out(a, t, vec * a.ld + 4 * N + i, spd);
    } else if (it < b2) {
      // a row of A12 (with B's when both write the cell), or of B alone
      const bool sh = it < b1;
      const int r = it - (sh ? b0 : b1), vec = r / p4, e = r - vec * p4, v = e / nchi, i = e - v * nchi;
      const bool both = a.shock && a.sj.rows[i] == a.brows[i];
      if (!sh && both) continue;
      const int j = (sh ? a.sj.rows[i] : a.brows[i]) - 2;
      const long m = i + (long)j * nchi;
      const double* x = t.X + vec * a.ld;
      double s = sh ? lane_dot(a.sj.a12 + (long)e * nchi, x + 4 * N, nchi, lane) : 0.0;
      if (!sh || both) s = ext_upstream_lane(a, x, a.bq + (i * 12 + v) * 4, 16, i, lane, s);
      s = warp_sum(ext_stencil_lane(a, x, v, m, i, j, lane, s));
      if (lane == 0) ext_out(a, t, vec * a.ld + v * N + m, s);
    } else if (!T) {  // freestream rows -i w u of real vectors (re, im)
      const int r = it - b2, vec = r / per_free, f = (r - vec * per_free) * 32 + lane;
      if (f >= a.nw * p4) continue;
      const long idx = a.nop + f;
      const double sg = (vec & 1) ? -1.0 : 1.0;
      ext_out(a, t, vec * a.ld + idx, sg * a.w[f / p4] * t.X[(vec ^ 1) * a.ld + idx]);
    } else {  // every freestream block gets B^T q + i w u
      const int r = it - b2, vec = r / p4, e = r - vec * p4, vin = e / nchi, n = e - vin * nchi;
      const double* x = t.X + vec * a.ld;
      const double* xo = t.X + (vec ^ 1) * a.ld;
      // lanes 0 .. 14: the products of three columns and their speeds, then summed
      double bt = 0;
      const int d = lane / 5, vo = lane - 5 * d, m = n + d - 1;
      if (lane < 15 && m >= 0 && m < nchi) {
        const int slot = (m * 3 + (n - m) + 1) * 4;
        if (vo < 4) bt = a.bq[(slot + vo) * 4 + vin] * x[vo * N + m + (long)(a.brows[m] - 2) * nchi];
        else if (a.shock) bt = a.bs[slot + vin] * x[4 * N + m];
      }
      bt = warp_sum(bt);
      const double sg = (vec & 1) ? 1.0 : -1.0;
      for (int kk = lane; kk < a.nw; kk += 32) {
        const long idx = a.nop + (long)kk * p4 + e;
        ext_out(a, t, vec * a.ld + idx, fma(sg * a.w[kk], xo[idx], bt));
      }
    }
  }
}

// k_expm_coop's schedule (the first term added one term late, degree 1 with a pass of its own)
// over ext_pass; sum holds the input when the steps begin.
template <bool T>
__global__ void __launch_bounds__(kMvThreads, 3) k_expm_ext(ExtArgs a, int nsteps, int order, const double* xin,
                                                            double* sum, double* t1, double* t2) {
  cg::grid_group grid = cg::this_grid();
  const long n = a.ld * (long)a.k;
  if (xin != sum) {
    for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) sum[q] = xin[q];
    grid.sync();
  }
  for (int s = 0; s < nsteps; ++s) {
    ExtTerm t{sum, nullptr, nullptr, nullptr, 0, 0};
    long fact = 1;
    for (int j = 1; j <= order; ++j) {
      fact *= j;
      t.Y = (j % 2) ? t1 : t2;
      t.acc = j == 1 ? nullptr : sum;
      t.c = 1.0 / (double)(a.divide ? j : fact);
      ext_pass<T>(a, t);
      grid.sync();
      t.X = t.Y;
      t.prev = j == 1 ? t.Y : nullptr;
      t.c_prev = t.c;
    }
    if (order == 1) {
      for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        sum[q] = sum[q] + t1[q];
      grid.sync();
    }
  }
}

}  // namespace

void launch_shock_mv(const DevCtx& d, int k, const double* X, double* Y, int transpose, double scale,
                     cudaStream_t st, long ld) {
  ShockMvArgs a;
  a.sj = d.sj;
  a.X = X;
  a.Y = Y;
  a.N = d.N;
  a.ld = ld;
  a.scale = scale;
  a.nchi = d.nchi;
  a.k = k;
  a.transpose = transpose;
  // enough blocks per vector to spread the rows over the SMs, few enough that staging
  // the vector into each block stays small next to the blocks' reads of A12 and A22
  const long per = (transpose ? 1L : 5L) * d.nchi;
  const long wpb = kShockThreads / 32;
  const long cap = std::max(1L, 8L * d.sms / k);
  const int bx = (int)std::max(1L, std::min((per + wpb - 1) / wpb, cap));
  k_shock_mv<<<dim3(bx, k), kShockThreads, shock_mv_smem(d.nchi, transpose), st>>>(a);
}

// y = scale A x over k vectors of op_size(d) entries (stride ld, 0: op_size(d)): the stencil
// blocks, then the shock-position blocks when the operator has them.
int coef_stream(const DevCtx& d) { return 144L * d.N * 8 > kCoefStreamBytes ? 1 : 0; }

void launch_k_matvec(const DevCtx& d, int k, const MvArgs& a, int grid, int th, cudaStream_t st) {
  const bool one = mv_one(d.N, k, d.sms), stream = coef_stream(d);
  if (one && stream) k_matvec<true, true><<<grid, th, 0, st>>>(a);
  else if (one) k_matvec<true, false><<<grid, th, 0, st>>>(a);
  else if (stream) k_matvec<false, true><<<grid, th, 0, st>>>(a);
  else k_matvec<false, false><<<grid, th, 0, st>>>(a);
}

// Batches that take the fixed-point matvec: those where even the first one after a write of the
// blocks, which makes their parts (~0.35 ns a cell and their storage, against ~66 ps saved per
// cell and vector), is no slower than in FP64. Repeated, smaller ones would gain too (300 x 200,
// 16 vectors: 173 -> 125 us), but their first took 75 us longer. hymor_set_expm_arith(0) keeps FP64.
static bool fx_takes(const DevCtx& d, int k) {
  return d.expm_ff && k >= 8 && (long)(k - 6) * d.N >= 1000000 && !mv_one(d.N, k, d.sms);
}

// the integer parts of the blocks for one direction, made again after each write of the blocks
static void launch_fx_build(DevCtx& d, int transpose, cudaStream_t st) {
  if (d.fx_version[transpose] == d.coef_version) return;
  (transpose ? k_fx_build<true> : k_fx_build<false>)<<<grid_for(16 * d.N, 256), 256, 0, st>>>(
      d.coef, d.fx_part[transpose], d.fx_ex[transpose], make_wrap(d.cfg), d.N);
  d.fx_version[transpose] = d.coef_version;
}

// fx: the fixed-point parts are current for this direction (the entry points that may allocate
// make them: fx_ready)
void launch_matvec(const DevCtx& d, int k, const double* X, double* Y, int transpose, double scale,
                   cudaStream_t st, long ld, bool fx) {
  if (ld <= 0) ld = op_size(d);
  MvArgs a;
  a.acc_prev = nullptr;
  a.c_prev = 0;
  a.vscale = nullptr;
  a.coef = d.coef;
  a.nz = d.coef_nz;
  a.X = X;
  a.Y = Y;
  a.acc = nullptr;
  a.scale = scale;
  a.c_acc = 0;
  a.w = make_wrap(d.cfg);
  a.N = d.N;
  a.ld = ld;
  a.k = k;
  a.transpose = transpose;
  const long items = mv_items(d.N, k, d.sms);
  const int th = mv_threads(items, d.sms);
  if (fx && fx_takes(d, k)) {
    FxArgs f{d.fx_part[transpose != 0], d.fx_ex[transpose != 0], a};
    const long tiles = (long)((d.nchi + 31) / 32) * ((d.neta + kFxRows - 1) / kFxRows);
    k_matvec_fx<<<(unsigned)(tiles * ((k + kFxVecs - 1) / kFxVecs)), 256, 0, st>>>(f);
  } else {
    launch_k_matvec(d, k, a, grid_for(items, th), th, st);
  }
  if (d.sj.on) launch_shock_mv(d, k, X, Y, transpose, scale, st, ld);
}

long recept_size(const DevCtx& d, int nw) { return op_size(d) + (long)nw * 4 * d.nchi; }

// y = scale L_ x (or scale L_^H x) for k complex vectors ([re; im] of recept_size each)
void launch_recept_apply(const DevCtx& d, int k, int nw, const double* dw, const double* X, double* Y, int adjoint,
                         double scale, cudaStream_t st) {
  const long ld = recept_size(d, nw);
  launch_matvec(d, 2 * k, X, Y, adjoint, scale, st, ld);
  RecArgs a;
  a.X = X;
  a.Y = Y;
  a.bq = d.bq;
  a.bs = d.bs;
  a.w = dw;
  a.rows = d.brows;
  a.N = d.N;
  a.ld = ld;
  a.nop = op_size(d);
  a.scale = scale;
  a.nchi = d.nchi;
  a.nw = nw;
  a.k = k;
  a.adjoint = adjoint;
  a.shock = d.sj.on;
  const long items = adjoint ? 8L * k * d.nchi : 2L * k * d.nchi + 8L * k * nw * d.nchi;
  k_recept_mv<<<grid_for(items, 256), 256, 0, st>>>(a);
}

// Runs `step` (the launches of one Taylor step, the same every step) nsteps times: captured
// once into a CUDA graph and replayed, so that the dozen small launches of a step cost one
// graph launch; launched directly when the stream is already being captured by the caller
// or the capture fails.
// graph_ok false: always launch directly (the allocation-free propagator builds no graph).
template <class Step>
static void repeat_steps(int nsteps, cudaStream_t st, Step step, bool graph_ok = true) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  if (graph_ok && nsteps > 1 && cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone &&
      cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    step();
    if (cudaStreamEndCapture(st, &g) == cudaSuccess && g && cudaGraphInstantiate(&ge, g, 0) == cudaSuccess) {
      for (int s = 0; s < nsteps; ++s) cudaGraphLaunch(ge, st);
      cudaGraphExecDestroy(ge);
      cudaGraphDestroy(g);
      return;
    }
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();  // a failed capture leaves nothing launched: run the steps directly
  }
  for (int s = 0; s < nsteps; ++s) step();
}

// EXPONENTIAL! (Transient_growth_downstream/CONSTRUCT_C.jl:78-111) with L_: per step term =
// vout, then term = (L_ dt) term / j and vout += term for j = 1..order. work: 2 x 2k x ld.
void launch_recept_expm(const DevCtx& d, int k, int nw, const double* dw, double dt, int nsteps, int order,
                        const double* X, double* Y, int adjoint, double* work, cudaStream_t st) {
  const long n = 2L * k * recept_size(d, nw);
  double* term = work;
  double* t2 = work + n;
  k_copy<<<grid_for(n, 256), 256, 0, st>>>(X, Y, n);
  repeat_steps(nsteps, st, [&]() {
    k_copy<<<grid_for(n, 256), 256, 0, st>>>(Y, term, n);
    double* src = term;
    double* dst = t2;
    for (int j = 1; j <= order; ++j) {
      launch_recept_apply(d, k, nw, dw, src, dst, adjoint, dt, st);
      k_scale_acc<<<grid_for(n, 256), 256, 0, st>>>(dst, Y, 1.0 / (double)j, n);
      std::swap(src, dst);
    }
  });
}

// POWER_METHOD! (Eigenvalues/ARNOLDI_POWER_GPU.jl:64-82): per step vout = v,
// term_j = (A dt) term_{j-1}, vout += term_j / j!, v = vout. The body assumes v and vout
// already hold the input.
static void launch_expm_body(const DevCtx& d, int k, double dt, int nsteps, int order, double* v, double* t1,
                             double* t2, double* vout, int transpose, cudaStream_t st, bool graph_ok) {
  const long n = op_size(d) * (long)k;
  if (d.sj.on) {
    // with the shock blocks every term is a full operator application, then vout += term / j!
    repeat_steps(nsteps, st, [&]() {
      const double* src = v;
      long fact = 1;
      for (int j = 1; j <= order; ++j) {
        fact *= j;
        double* dst = (j % 2) ? t1 : t2;
        launch_matvec(d, k, src, dst, transpose, dt, st);
        k_axpy<<<grid_for(n, 256), 256, 0, st>>>(vout, dst, 1.0 / (double)fact, n);
        src = dst;
      }
      k_copy<<<grid_for(n, 256), 256, 0, st>>>(vout, v, n);
    }, graph_ok);
    return;
  }
  const long items = mv_items(d.N, k, d.sms);
  const int th = mv_threads(items, d.sms);
  MvArgs a;
  a.acc_prev = nullptr;
  a.c_prev = 0;
  a.vscale = nullptr;
  a.coef = d.coef;
  a.nz = d.coef_nz;
  a.w = make_wrap(d.cfg);
  a.N = d.N;
  a.ld = n / k;
  a.k = k;
  a.transpose = transpose;
  a.scale = dt;
  const bool late = order >= 2;  // as k_expm_coop: the first term is added one matvec late
  for (int s = 0; s < nsteps; ++s) {
    const double* src = late ? vout : v;
    const double* prev = nullptr;
    double c_prev = 0;
    long fact = 1;
    for (int j = 1; j <= order; ++j) {
      fact *= j;
      double* dst = (j % 2) ? t1 : t2;
      a.X = src;
      a.Y = dst;
      a.acc = (late && j == 1) ? nullptr : vout;
      a.acc_prev = prev;
      a.c_prev = c_prev;
      a.c_acc = 1.0 / (double)fact;
      launch_k_matvec(d, k, a, grid_for(items, th), th, st);
      src = dst;
      prev = (late && j == 1) ? dst : nullptr;
      c_prev = a.c_acc;
    }
    if (!late) k_copy<<<grid_for(n, 256), 256, 0, st>>>(vout, v, n);
  }
}


// The extended operators' propagation in one cooperative launch (k_expm_ext): from as many
// launches as the stencil operator's, up to `most` cells x vectors: its 8 warps per SM have fewer
// loads on their way than the launches' full SMs, so that a term of many cells takes longer alone
// (with three contexts at once it is the faster one to ~75 000). One propagation of 60 steps of
// degree 5 alone, ms, in launches and in one: shock-position unknowns 160 x 97 4.3 and 3.0,
// 180 x 100 4.45 and 4.37, 210 x 105 5.2 and 5.7, 300 x 150 7.8 and 8.9, 500 x 250 17.7 and 33.9;
// one adjoint vector 243 x 111 6.5 and 6.1, 390 x 190 12.9 and 17.8; the receptivity operator
// (three launches a term more) 200 x 160, 64 000 in real vectors, 9.6 and 9.3.
constexpr int kExpmCoopMinLaunches = 16;
constexpr long kExtShock = 20000, kExtShockAdj = 30000, kExtRecept = 64000;
static bool expm_ext_fits(const DevCtx& d, int k, int nsteps, int order, long most) {
  return (long)nsteps * (order + 1) >= kExpmCoopMinLaunches && mv_one(d.N, k, d.sms) && d.N * k <= most;
}
static ExtArgs ext_args(const DevCtx& d, int k, double dt) {
  ExtArgs a;
  a.coef = d.coef;
  a.sj = d.sj;
  a.bq = a.bs = a.w = nullptr;
  a.brows = nullptr;
  a.wr = make_wrap(d.cfg);
  a.N = d.N;
  a.ld = a.nop = op_size(d);
  a.dt = dt;
  a.nchi = d.nchi;
  a.k = k;
  a.nw = 0;
  a.shock = d.sj.on;
  a.divide = 0;
  return a;
}
// work: 2 x k x ld doubles
static cudaError_t launch_expm_ext(const DevCtx& d, const ExtArgs& a, int transpose, int nsteps, int order,
                                   const double* dX, double* dY, double* work, cudaStream_t st) {
  double *t1 = work, *t2 = work + a.ld * (long)a.k;
  const int grid = (int)std::min<long>((4 * d.N * a.k / 32 + a.k * d.nchi + 7) / 8, d.sms);
  void* args[] = {(void*)&a, &nsteps, &order, (void*)&dX, &dY, &t1, &t2};
  return cudaLaunchCooperativeKernel(transpose ? (const void*)k_expm_ext<true> : (const void*)k_expm_ext<false>,
                                     std::max(grid, 1), kMvThreads, args, 0, st);
}

void launch_expm(const DevCtx& d, int k, double dt, int nsteps, int order, const double* X, double* Yout,
                 int transpose, double* work, cudaStream_t st, bool graph_ok) {
  if (d.sj.on && expm_ext_fits(d, k, nsteps, order, transpose && k == 1 ? kExtShockAdj : kExtShock)) {
    launch_expm_ext(d, ext_args(d, k, dt), transpose, nsteps, order, X, Yout, work, st);
    return;
  }
  const long n = op_size(d) * (long)k;
  double* v = work;
  double* t1 = work + n;
  double* t2 = work + 2 * n;
  k_copy<<<grid_for(n, 256), 256, 0, st>>>(X, v, n);
  k_copy<<<grid_for(n, 256), 256, 0, st>>>(X, Yout, n);
  launch_expm_body(d, k, dt, nsteps, order, v, t1, t2, Yout, transpose, st, graph_ok);
}

// Workspaces of the perturbed residuals of a linearisation (the A11 colours, the shock-point
// residuals, LINEARIZE_B's columns): each lane has its own stage array, p, T, edge sound
// speed, shock points, spline workspace, shock speeds, prescribed upstream columns and flux.
// The lanes form two groups with a stream each; a group evaluates one perturbation per lane,
// every kernel launched once for all its lanes (grid z), and the other group's launches run
// beside it. The base state, the mesh, the base flux and the assembled blocks are shared:
// read-only, or written at entries no other perturbation writes, with the same arithmetic as
// one after another, so the result does not depend on the lanes. Where the memory for the lanes is
// missing, fewer serve (ensure_lanes), down to one group of three.
// One launch per kernel and group instead of one per residual, because the ~9 launches of a
// residual cost the host ~2 us each: the assembly with the shock unknowns at 200 x 100 (245
// residuals) took 4.2 ms, bound by them, and takes 1.06 ms so (with its point residuals on the
// shock band's tiles only). Lanes per group: enough cells to fill the GPU (1.2 M), at least 9
// and at most 32; the 36 colours take 9 or 18 at a time (one or two variables).
constexpr int kLaneGroups = 2;
constexpr int kMaxGroupLanes = 32;
static PertArgs pert_args(const DevCtx& d);
struct JacLane {
  Cons Y;
  double *p, *T, *aY, *spl, *speed_x, *speed_y, *rel, *cols;
  ShockPts Yp;
  double* F[4];
};
struct JacLanes {
  JacLane first[kLaneGroups];  // the first lane of each group; the next is `stride` doubles on
  cudaStream_t st[kLaneGroups] = {};
  cudaEvent_t done[kLaneGroups] = {};
  cudaEvent_t fork = nullptr;
  double* mem = nullptr;
  long stride = 0;
  int groups = 0, per_group = 0;
};
int lanes_per_group(long N) {
  const long want = (1200000 + N - 1) / N;
  for (int g : {9, 18})
    if (want <= g) return g;
  return kMaxGroupLanes;
}

// The group's view of the context: its lanes' buffers in place of the shared ones, `count` of
// them. TMA descriptors name the context's own stage array, so a lane loads its halo thread by
// thread (the same values, the same arithmetic). own_fit: each lane fits its own shock points
// (else they are S's, and all read the fit that the base residual left in the context's
// workspace).
DevCtx lane_ctx(const DevCtx& d, const JacLanes& L, int group, int count, bool own_fit = false) {
  DevCtx ld = d;
  const JacLane& l = L.first[group];
  ld.Y = l.Y;
  ld.p = l.p;
  ld.T = l.T;
  ld.aY = l.aY;
  if (own_fit) ld.spl = l.spl;
  ld.spl_shared = !own_fit;
  ld.speed_x = l.speed_x;
  ld.speed_y = l.speed_y;
  ld.rel = l.rel;
  ld.Yp = l.Yp;
  ld.tma = 0;
  if (d.up_cols) ld.up_cols = l.cols;
  ld.lanes = count;
  ld.lane_stride = L.stride;
  return ld;
}

// every group waits for the work enqueued on st so far
void lanes_fork(JacLanes& L, cudaStream_t st) {
  cudaEventRecord(L.fork, st);
  for (cudaStream_t s : L.st) cudaStreamWaitEvent(s, L.fork, 0);
}
// st waits for every group
void lanes_join(JacLanes& L, cudaStream_t st) {
  for (int g = 0; g < kLaneGroups; ++g) {
    cudaEventRecord(L.done[g], L.st[g]);
    cudaStreamWaitEvent(st, L.done[g], 0);
  }
}
// run(first perturbation, group, lanes) over n perturbations, at most `most` at a time
template <class Run>
static void for_groups(const JacLanes& L, int n, int most, Run run) {
  const int g = std::min(most, L.per_group);
  int group = 0;
  for (int q = 0; q < n; q += g, group = (group + 1) % L.groups) run(q, group, std::min(g, n - q));
}

// The shock-position blocks (perturb_shock), after the A11 assembly has left the base
// flux in Fb and the base shock speeds in sj.rel_b, on the shocked rows d.cell_idx:
//   A21 (LINEARIZE_EQUATIONS_NO_DISCONTINUITY.jl:140-258): the shock speed of column i
//     reads only the cells (i, sc_i - 1) and (i, sc_i - 2) of its own column
//     (UPDATE_SHOCK_JUMP_PROPERTIES.jl:354-405), so raising the cell (i, sc_i - j) of every
//     column at once gives each column's speed the same inputs, and the same result, as the
//     reference's one perturbed cell per residual; the reference's other entries of such
//     a column are exact zeros. 8 residuals (j = 1, 2; 4 variables), no flux needed.
//   A12, A22 (:262-274): one residual per shock point, the point moved by eps along the
//     PERTURB_SHOCK direction (the smoothing spline couples every point to every other).
//     Only the flux of the cells (i, sc_i - 1) and the speeds are read: the residuals cover the
//     tiles that hold those cells (launch_band_tiles; the same per-cell arithmetic as the whole
//     grid) and copy only the rows those tiles read; what the boundary kernels make of the
//     other rows is not used. hrows: the shocked rows on the host.
void launch_shock_assemble(DevCtx& d, const double* const Fb[4], JacLanes& L, const int* hrows, cudaStream_t st) {
  const hymor_config& c = d.cfg;
  const int nchi = d.nchi;
  const int cb = (nchi + 127) / 128;
  const double eps = c.perturbation_magnitude;
  const double h = std::hypot(c.rho_u_0, c.rho_v_0);
  k_shock_dir<<<cb, 128, 0, st>>>(d.beta, d.sj.dir, nchi, c.rho_u_0 / h, c.rho_v_0 / h);
  cudaMemcpyAsync(d.sj.rows, d.cell_idx, sizeof(int) * nchi, cudaMemcpyDeviceToDevice, st);
  int jlo = 0, jhi = 0;
  launch_band_tiles(d, hrows, jlo, jhi, st);
  lanes_fork(L, st);
  for_groups(L, 8, 4, [&](int q, int group, int n) {
    const DevCtx ld = lane_ctx(d, L, group, n);
    cudaStream_t ls = L.st[group];
    PertArgs pl = pert_args(ld);
    pl.first = q;
    pl.batch = 2;
    pl.j0 = jlo;
    pl.j1 = jhi;
    k_perturb_thermo<<<dim3(grid_for((long)d.NI * (jhi - jlo), 256), 1, n), 256, 0, ls>>>(pl);
    launch_columns_bc(ld, false, false, 0, 0, 0, true, false, ls);
    k_gather_a21<<<dim3(cb, 1, n), 128, 0, ls>>>(ld.rel, d.sj.rel_b, d.sj.a21, nchi, q, eps, L.stride);
  });
  Flux4 fb;
  for (int v = 0; v < 4; ++v) fb.v[v] = Fb[v];
  for_groups(L, nchi, kMaxGroupLanes, [&](int q, int group, int n) {
    const DevCtx ld = lane_ctx(d, L, group, n, true);
    cudaStream_t ls = L.st[group];
    const JacLane& l = L.first[group];
    Flux4 fp;
    for (int v = 0; v < 4; ++v) fp.v[v] = l.F[v];
    double* const Fp[4] = {l.F[0], l.F[1], l.F[2], l.F[3]};
    PertArgs pl = pert_args(ld);
    pl.j0 = jlo;
    pl.j1 = jhi;
    k_perturb_thermo<<<dim3(grid_for((long)d.NI * (jhi - jlo), 256), 1, n), 256, 0, ls>>>(pl);
    k_perturb_point<<<dim3(cb, 1, n), 128, 0, ls>>>(d.Sp, ld.Yp, d.sj.dir, nchi, q, eps, L.stride);
    launch_shock_bc_flags(ld, false, false, true, true, 0, ls);
    launch_flux_class(ld, false, Fp, 1, ls);
    k_gather_a12<<<dim3(cb, 1, n), 128, 0, ls>>>(fp, fb, ld.rel, d.sj.rel_b, d.sj.rows, d.sj.a12, d.sj.a22, nchi, q,
                                                 eps, L.stride);
  });
  lanes_join(L, st);
  k_transpose<<<grid_for(4L * nchi * nchi, 256), 256, 0, st>>>(d.sj.a12, d.sj.a12t, 4L * nchi, nchi);
  k_transpose<<<grid_for((long)nchi * nchi, 256), 256, 0, st>>>(d.sj.a22, d.sj.a22t, nchi, nchi);
}

static PertArgs pert_args(const DevCtx& d) {
  const hymor_config& c = d.cfg;
  PertArgs pa;
  pa.S = d.S;
  pa.Y = d.Y;
  pa.p = d.p;
  pa.T = d.T;
  pa.cell_idx = d.cell_idx;
  pa.eps = c.perturbation_magnitude;
  pa.gm1 = c.gamma - 1;
  pa.nchi = d.nchi;
  pa.neta = d.neta;
  pa.shock = c.shock_enabled;
  pa.shock_row = 0;
  pa.aY = d.aY;
  pa.nrcbc = (c.bc_chi0 == HYMOR_BC_OUTFLOW_NRCBC) | ((c.bc_chi1 == HYMOR_BC_OUTFLOW_NRCBC) << 1) |
             ((c.bc_eta0 == HYMOR_BC_OUTFLOW_NRCBC) << 2) | ((c.bc_eta1 == HYMOR_BC_OUTFLOW_NRCBC) << 3);
  pa.var = -1;
  pa.colour = 1;
  pa.j0 = 0;
  pa.j1 = d.NJ;
  pa.lane = d.lane_stride;
  pa.first = 0;
  pa.batch = 0;
  return pa;
}

void launch_jacobian_assemble(DevCtx& d, cudaStream_t st, JacLanes& L, const int* hrows) {
  ++d.coef_version;
  const hymor_config& c = d.cfg;
  const long N = d.N;
  double* Fb[4];
  for (int v = 0; v < 4; ++v) Fb[v] = d.jwork + v * N;
  const bool shock_blocks = c.shock_enabled && c.perturb_shock;
  PertArgs pa = pert_args(d);
  // base output: NON_LINEAR_DYNAMICS(deepcopy(s))
  k_perturb_thermo<<<grid_for(d.G, 256), 256, 0, st>>>(pa);
  launch_shock_bc_flags(d, false, true, c.shock_enabled, true, 0, st);
  launch_flux(d, false, Fb, st);
  if (shock_blocks)
    cudaMemcpyAsync(d.sj.rel_b, d.rel, sizeof(double) * d.nchi, cudaMemcpyDeviceToDevice, st);
  cudaMemsetAsync(d.coef, 0, sizeof(double) * 144 * N, st);
  ScatArgs sa;
  for (int v = 0; v < 4; ++v) sa.Fb[v] = Fb[v];
  sa.coef = d.coef;
  sa.nz = d.coef_nz + N;
  sa.w = make_wrap(c);
  sa.eps = c.perturbation_magnitude;
  sa.inv_eps = div_eps_reciprocal(sa.eps);
  sa.N = N;
  sa.lane = L.stride;
  // the 36 colour x variable residuals over the lanes; the shock points of all are S's, so
  // the smoothing-spline fit of the base residual serves them
  lanes_fork(L, st);
  const int most = L.per_group >= 18 ? 18 : (L.per_group >= 9 ? 9 : 3);
  for_groups(L, 36, most, [&](int q, int group, int n) {
    const DevCtx ld = lane_ctx(d, L, group, n);
    cudaStream_t ls = L.st[group];
    const JacLane& l = L.first[group];
    PertArgs pl = pert_args(ld);
    pl.first = q;
    pl.batch = 1;
    double* const Fp[4] = {l.F[0], l.F[1], l.F[2], l.F[3]};
    k_perturb_thermo<<<dim3(grid_for(d.G, 256), 1, n), 256, 0, ls>>>(pl);
    launch_columns_bc(ld, false, false, 0, 0, 0, c.shock_enabled, true, ls);
    launch_flux(ld, false, Fp, ls);
    ScatArgs sl = sa;
    for (int v = 0; v < 4; ++v) sl.Fp[v] = l.F[v];
    sl.first_var = q / 9;
    sl.colour0 = q % 9;
    sl.colours = n;
    if (most < 9) k_scatter<true><<<grid_for(N, 256), 256, 0, ls>>>(sl);
    else k_scatter<false><<<dim3(grid_for(N, 256), 1, n / 9), 256, 0, ls>>>(sl);
  });
  lanes_join(L, st);
  k_masks<<<grid_for(N, 256), 256, 0, st>>>(d.coef_nz, d.coef_nz + N, make_wrap(c), N);
  if (shock_blocks) launch_shock_assemble(d, Fb, L, hrows, st);
}

// LINEARIZE_B (Freestream_receptivity/LINEARIZE_B.jl:40-170): the residual with a prescribed
// per-column upstream state (rho_0_upstream_p), once unperturbed and once per variable and
// colour of columns (i = colour mod 3 raised by eps): 13 residuals. Each output column m has
// exactly one raised column among m - 1, m, m + 1 per colour.
void launch_b_assemble(DevCtx& d, cudaStream_t st, JacLanes& L) {
  const hymor_config& c = d.cfg;
  const long N = d.N;
  const int nchi = d.nchi, cb = (nchi + 127) / 128;
  const double eps = c.perturbation_magnitude;
  double* Fb[4];
  Flux4 fb;
  for (int v = 0; v < 4; ++v) {
    Fb[v] = d.jwork + v * N;
    fb.v[v] = Fb[v];
  }
  double* cols = d.bwork;
  double* rel_b = d.bwork + 4 * nchi;
  cudaMemcpyAsync(d.brows, d.cell_idx, sizeof(int) * nchi, cudaMemcpyDeviceToDevice, st);
  cudaMemsetAsync(d.bq, 0, sizeof(double) * 48 * nchi, st);
  cudaMemsetAsync(d.bs, 0, sizeof(double) * 12 * nchi, st);
  d.up_cols = cols;
  // base: the uniform upstream state
  k_up_cols<<<cb, 128, 0, st>>>(cols, nchi, c.rho_0, c.rho_u_0, c.rho_v_0, c.rho_E_0, -1, 0, eps);
  k_perturb_thermo<<<grid_for(d.G, 256), 256, 0, st>>>(pert_args(d));
  launch_shock_bc_flags(d, false, true, true, true, 0, st);
  launch_flux(d, false, Fb, st);
  cudaMemcpyAsync(rel_b, d.rel, sizeof(double) * nchi, cudaMemcpyDeviceToDevice, st);
  // one residual per variable and colour of columns, over the lanes (each with its own upstream
  // columns; the shock points are S's, so the base residual's fit serves them all)
  lanes_fork(L, st);
  for_groups(L, 12, 6, [&](int q, int group, int n) {
    const DevCtx ld = lane_ctx(d, L, group, n);
    cudaStream_t ls = L.st[group];
    const JacLane& l = L.first[group];
    Flux4 fp;
    for (int v = 0; v < 4; ++v) fp.v[v] = l.F[v];
    double* const Fp[4] = {l.F[0], l.F[1], l.F[2], l.F[3]};
    k_up_cols<<<dim3(cb, 1, n), 128, 0, ls>>>(l.cols, nchi, c.rho_0, c.rho_u_0, c.rho_v_0, c.rho_E_0, 0, 0, eps, q,
                                              L.stride);
    k_perturb_thermo<<<dim3(grid_for(d.G, 256), 1, n), 256, 0, ls>>>(pert_args(ld));
    launch_columns_bc(ld, false, false, 0, 0, 0, true, true, ls);
    launch_flux(ld, false, Fp, ls);
    k_gather_b<<<dim3(cb, 1, n), 128, 0, ls>>>(fp, fb, ld.rel, rel_b, d.brows, d.bq, d.bs, nchi, q, eps, L.stride);
  });
  lanes_join(L, st);
  d.up_cols = nullptr;
}

}  // namespace hymor

using namespace hymor;

namespace {
// Device memory that the context's linear entry points keep: counted against
// hymor_set_workspace_limit, and for the context's life unless lin_free gives it back. What is
// not to be had at first is tried again without the fixed-point parts (spare: it is they).
cudaError_t lin_malloc(hymor_ctx* ctx, void** p, size_t bytes, bool spare = false);
void lin_free(hymor_ctx* ctx, void* p, size_t bytes);

// Storage of the shock-position blocks and their rows.
int ensure_shock(hymor_ctx* ctx) {
  DevCtx& d = ctx_dev(ctx);
  if (d.sj.a12) return 0;
  const long n = d.nchi;
  // the transposed shock matvec stages 5 Nchi doubles per block
  const long smem = shock_mv_smem(d.nchi, 1);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(k_shock_mv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return ctx_fail(ctx, HYMOR_ERR_INVALID, "perturb_shock: Nchi too large for the shock matvec's shared memory");
  const long doubles = 11 * n + 10 * n * n;
  void* p = nullptr;
  if (lin_malloc(ctx, &p, sizeof(double) * doubles + sizeof(int) * n) != cudaSuccess)
    return ctx_fail(ctx, HYMOR_ERR_CUDA, "shock-block allocation failed");
  ctx_allocs(ctx).push_back(p);
  double* b = static_cast<double*>(p);
  ShockJac& j = d.sj;
  j.a21 = b;
  j.a12 = j.a21 + 8 * n;
  j.a22 = j.a12 + 4 * n * n;
  j.a12t = j.a22 + n * n;
  j.a22t = j.a12t + 4 * n * n;
  j.rel_b = j.a22t + n * n;
  j.dir = j.rel_b + n;
  j.rows = reinterpret_cast<int*>(b + doubles);
  return 0;
}

// The A21 block reads the cells (i, sc_i - 2): a shocked row below 3 has no such cell (the
// reference's column index i + (sc_i - 3) Nchi would be out of range).
int check_shock_rows_for_blocks(hymor_ctx* ctx, const int* rows, int nchi, int neta) {
  for (int i = 0; i < nchi; ++i)
    if (rows[i] < 3 || rows[i] > neta - 1) {
      char msg[200];
      snprintf(msg, sizeof msg, "perturb_shock: shocked row %d of column %d outside 3..%d", rows[i], i + 1, neta - 1);
      return ctx_fail(ctx, HYMOR_ERR_SHOCK_RANGE, msg);
    }
  return 0;
}

// Storage of the upstream-boundary operator B.
int ensure_b(hymor_ctx* ctx) {
  DevCtx& d = ctx_dev(ctx);
  if (d.bq) return 0;
  void* p = nullptr;
  if (lin_malloc(ctx, &p, (sizeof(double) * 65 + sizeof(int)) * (long)d.nchi) != cudaSuccess)
    return ctx_fail(ctx, HYMOR_ERR_CUDA, "upstream-boundary operator allocation failed");
  ctx_allocs(ctx).push_back(p);
  d.bq = static_cast<double*>(p);
  d.bs = d.bq + 48 * d.nchi;
  d.bwork = d.bs + 12 * d.nchi;
  d.brows = reinterpret_cast<int*>(d.bq + 65 * (long)d.nchi);
  return 0;
}

// B's flux rows are the cells (m, sc_m - 1): sc_m must leave one flow cell below it.
int check_b_rows(hymor_ctx* ctx, const int* rows, int nchi, int neta) {
  for (int i = 0; i < nchi; ++i)
    if (rows[i] < 2 || rows[i] > neta - 1) {
      char msg[200];
      snprintf(msg, sizeof msg, "upstream-boundary operator: shocked row %d of column %d outside 2..%d", rows[i], i + 1,
               neta - 1);
      return ctx_fail(ctx, HYMOR_ERR_SHOCK_RANGE, msg);
    }
  return 0;
}

int ensure_linear(hymor_ctx* ctx) {
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) {
    void *coef = nullptr, *nz = nullptr, *work = nullptr;
    const size_t bc = sizeof(double) * 144 * d.N, bn = 5 * d.N, bw = sizeof(double) * 8 * d.N;
    if (lin_malloc(ctx, &coef, bc) != cudaSuccess || lin_malloc(ctx, &nz, bn) != cudaSuccess ||
        lin_malloc(ctx, &work, bw) != cudaSuccess) {
      lin_free(ctx, coef, bc);
      lin_free(ctx, nz, bn);
      return ctx_fail(ctx, HYMOR_ERR_CUDA, "Jacobian allocation failed");
    }
    for (void* p : {coef, nz, work}) ctx_allocs(ctx).push_back(p);
    d.coef_nz = static_cast<unsigned char*>(nz);
    d.jwork = static_cast<double*>(work);
    d.coef = static_cast<double*>(coef);
  }
  return 0;
}

int cuda_check(hymor_ctx* ctx, cudaError_t e) {
  if (e != cudaSuccess) return ctx_fail(ctx, HYMOR_ERR_CUDA, cudaGetErrorString(e));
  return 0;
}

// Propagations of more than a few launches run as one cooperative kernel (k_expm_coop)
// over four context buffers (v, two Taylor terms, vout): a call copies its input into v
// and vout, launches once and copies vout out. This removes the per-launch overhead that
// dominates small grids (a 200 x 100 stencil matvec is ~5 us of FP64 work).
struct ExpmCache {
  double* buf = nullptr;
  long cap = 0;  // doubles
};
struct KrylovScratch {
  double* partial = nullptr;
  int cols = 0;
  double* h = nullptr;  // device coefficients (2 x cols + 2)
  double* tmp = nullptr;
  long tmp_n = 0;
};
// Per-context state of the linear entry points, owned by the context (created on first
// use, released by hymor_ctx_destroy).
struct LinearState {
  size_t used = 0, limit = 0;  // bytes of lin_malloc, and their limit (0: none)
  void* fx_mem[2] = {};        // the fixed-point parts of each direction and their size
  size_t fx_bytes = 0;
  int fx_refused[2] = {-1, -1};  // the write of the blocks whose parts did not fit
  ExpmCache expm;
  KrylovScratch kry;
  bool res_ready = false;  // k_expm_res_ff's shared memory is set
  int coop_blocks[10] = {};  // co-resident blocks per SM of k_expm_coop<false>, <true>,
                             // k_expm_coop_ff<0>, <1>, <2>, each with ordinary and
                             // streaming block loads
  JacLanes lanes;               // workspaces of the linearisations' perturbed residuals
};
LinearState& linear_state(hymor_ctx* ctx) {
  void*& slot = ctx_linear_state(ctx);
  if (!slot) slot = new LinearState();
  return *static_cast<LinearState*>(slot);
}
ExpmCache& expm_cache(hymor_ctx* ctx) { return linear_state(ctx).expm; }

// whether the context's stream is being captured (or in error)
bool stream_captured(hymor_ctx* ctx) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(ctx_stream(ctx), &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
}
// an error reported here, and not again by a later check of the launches
cudaError_t settled(cudaError_t e) {
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}
// an allocation, and if there is no room for it another try without the fixed-point parts, which
// then stay away until the next write of the blocks
template <class Take>
cudaError_t with_spare(hymor_ctx* ctx, Take take) {
  const cudaError_t e = settled(take());
  if (e != cudaErrorMemoryAllocation || !linear_spare_release(ctx)) return e;
  for (int& v : linear_state(ctx).fx_refused) v = ctx_dev(ctx).coef_version;
  return settled(take());
}
cudaError_t lin_malloc(hymor_ctx* ctx, void** p, size_t bytes, bool spare) {
  LinearState& s = linear_state(ctx);
  auto take = [&]() { return s.limit && s.used + bytes > s.limit ? cudaErrorMemoryAllocation : cudaMalloc(p, bytes); };
  const cudaError_t e = spare ? settled(take()) : with_spare(ctx, take);
  if (e == cudaSuccess) s.used += bytes;
  return e;
}
void lin_free(hymor_ctx* ctx, void* p, size_t bytes) {
  if (!p) return;
  cudaFree(p);
  linear_state(ctx).used -= bytes;
}

// The linearisation lanes, made on first use: two groups of 9 to 32 lanes of ~88 bytes a cell
// (800 x 400: 18 lanes, 507 MB), or, where the memory is missing, the first of two groups of 9,
// one of 9 and one of 3 that fits.
int ensure_lanes(hymor_ctx* ctx, JacLanes** out) {
  JacLanes& L = linear_state(ctx).lanes;
  *out = &L;
  if (L.mem) return 0;
  const DevCtx& d = ctx_dev(ctx);
  const size_t G = d.G, N = d.N, n = d.nchi;
  auto pad = [](size_t k) { return (k + 31) & ~size_t(31); };  // 256-byte aligned parts
  const size_t total = 7 * pad(G) + 4 * pad(N) + 4 * pad(n) + pad(17 * n + 16) + 3 * pad(n) + pad(4 * n);
  if (!L.fork && cudaEventCreateWithFlags(&L.fork, cudaEventDisableTiming) != cudaSuccess)
    return ctx_fail(ctx, HYMOR_ERR_CUDA, "linearisation lane event");
  for (int g = 0; g < kLaneGroups; ++g)
    if ((!L.st[g] && cudaStreamCreateWithFlags(&L.st[g], cudaStreamNonBlocking) != cudaSuccess) ||
        (!L.done[g] && cudaEventCreateWithFlags(&L.done[g], cudaEventDisableTiming) != cudaSuccess))
      return ctx_fail(ctx, HYMOR_ERR_CUDA, "linearisation lane stream");
  double* mem = nullptr;
  int groups = 0, per = 0;
  size_t bytes = 0;
  const int plans[][2] = {{kLaneGroups, lanes_per_group(N)}, {kLaneGroups, 9}, {1, 9}, {1, 3}};
  for (const auto& p : plans) {
    groups = p[0];
    per = p[1];
    bytes = sizeof(double) * total * per * groups;
    void* q = nullptr;
    if (lin_malloc(ctx, &q, bytes) == cudaSuccess) {
      mem = static_cast<double*>(q);
      break;
    }
  }
  if (!mem) return ctx_fail(ctx, HYMOR_ERR_CUDA, "linearisation lane allocation failed");
  if (cudaMemsetAsync(mem, 0, bytes, ctx_stream(ctx)) != cudaSuccess) {
    lin_free(ctx, mem, bytes);
    return ctx_fail(ctx, HYMOR_ERR_CUDA, "linearisation lane allocation failed");
  }
  L.mem = mem;
  L.stride = (long)total;
  L.groups = groups;
  L.per_group = per;
  for (int g = 0; g < groups; ++g) {
    JacLane& l = L.first[g];
    double* b = mem + total * per * g;
    auto take = [&](size_t k) {
      double* r = b;
      b += pad(k);
      return r;
    };
    double* y[4];
    for (double*& v : y) v = take(G);
    l.Y = Cons{y[0], y[1], y[2], y[3]};
    l.p = take(G);
    l.T = take(G);
    l.aY = take(G);
    for (int v = 0; v < 4; ++v) l.F[v] = take(N);
    for (double*& v : y) v = take(n);
    l.Yp = ShockPts{y[0], y[1], y[2], y[3]};
    l.spl = take(17 * n + 16);
    l.speed_x = take(n);
    l.speed_y = take(n);
    l.rel = take(n);
    l.cols = take(4 * n);
  }
  return 0;
}

// Cells x vectors below which the float-float propagation gives every output a thread: there it
// is bound by the latency of a pass, above by the loads and products, which a cell per thread
// (one vector) and the tiles (a batch) make once for four outputs. A propagation of one context
// alone, thread per output against the other, ms: one vector, 250 matvecs, 100 x 80 1.40 / 2.82,
// 200 x 150 2.81 / 3.09, 300 x 200 8.12 / 4.83, 400 x 300 13.8 / 6.6; 150 matvecs of 100 x 80
// with 4 vectors 1.72 / 2.81, 8 vectors 3.06 / 3.09, 16 vectors 5.10 / 3.79, of 200 x 100 with 2
// vectors 2.41 / 2.08, of 300 x 200 with 2 vectors 8.29 / 3.26.
constexpr long kFfOneCells = 40000;
constexpr long kResSmem = 220 * 1024;  // shared memory of the resident propagation
bool ff_one(long N, int k) { return N * k < kFfOneCells; }

// hdts, hsteps (host, k entries, hsteps non-increasing), or null: vector c is propagated
// hsteps[c] steps of hdts[c] instead of nsteps of dt.
int expm_cooperative(hymor_ctx* ctx, int k, double dt, int nsteps, int order, const double* dX, double* dY,
                     int transpose, const double* hdts = nullptr, const int* hsteps = nullptr) {
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  ExpmCache& c = expm_cache(ctx);
  const long n = 4 * d.N * (long)k;
  int r;
  if (4 * n + 2 * k > c.cap) {
    if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
    lin_free(ctx, c.buf, sizeof(double) * c.cap);
    c.buf = nullptr;
    c.cap = 0;
    void* p = nullptr;
    if ((r = cuda_check(ctx, lin_malloc(ctx, &p, sizeof(double) * (4 * n + 2 * k))))) return r;
    c.buf = static_cast<double*>(p);
    c.cap = 4 * n + 2 * k;
  }
  double* v = c.buf;
  double* t1 = c.buf + n;
  double* t2 = c.buf + 2 * n;
  double* vout = c.buf + 3 * n;
  // float-float (degree >= 2; its kernels decompose their work items in 32 bits), with the
  // blocks' float-float copy split again after each write of the blocks
  const bool ffp = d.expm_ff && order >= 2 && 4L * d.N * k < (1L << 31);
  if (ffp && (!d.coef_ff || d.coef_ff_version != d.coef_version)) {
    if (!d.coef_ff) {
      void* p = nullptr;
      if ((r = cuda_check(ctx, lin_malloc(ctx, &p, sizeof(float2) * 144 * d.N)))) return r;
      ctx_allocs(ctx).push_back(p);
      d.coef_ff = static_cast<float2*>(p);
    }
    k_coef_to_ff<<<grid_for(144 * d.N, 256), 256, 0, st>>>(d.coef, d.coef_ff, 144 * d.N);
    d.coef_ff_version = d.coef_version;
  }
  int* blocks_per_sm = linear_state(ctx).coop_blocks;
  const bool one = mv_one(d.N, k, d.sms);
  // float-float: thread per output on few cells x vectors, else a cell per thread for one vector
  // and tiles for a batch
  const int ffmode = ff_one(d.N, k) ? 1 : (k == 1 ? 2 : 0);
  const int kind = ffp ? 2 + ffmode : (one ? 1 : 0);
  const int kst = 2 * kind + coef_stream(d);
  const void* kerns[10] = {(const void*)k_expm_coop<false, false>,  (const void*)k_expm_coop<false, true>,
                           (const void*)k_expm_coop<true, false>,   (const void*)k_expm_coop<true, true>,
                           (const void*)k_expm_coop_ff<0, false>,   (const void*)k_expm_coop_ff<0, true>,
                           (const void*)k_expm_coop_ff<1, false>,   (const void*)k_expm_coop_ff<1, true>,
                           (const void*)k_expm_coop_ff<2, false>,   (const void*)k_expm_coop_ff<2, true>};
  const void* kern = kerns[kst];
  if (!blocks_per_sm[kst] &&
      (r = cuda_check(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm[kst], kern, kind == 2 ? kFfThreads : kMvThreads,
                                                                        kind == 2 ? ff_tile_smem<kVecChunk>() : 0))))
    return r;
  const long items = kind == 4 ? d.N : (kind == 3 ? 4 * d.N * k : mv_items(d.N, k, d.sms));
  const int th = kind == 2 ? kFfThreads : mv_threads(items, d.sms);
  const int nch = (k + kVecChunk - 1) / kVecChunk, chunk = (k + nch - 1) / nch;
  const long want = kind == 2 ? ff_tiles(make_wrap(d.cfg)) * ((k + chunk - 1) / chunk) : (items + th - 1) / th;
  // co-resident: blocks of th <= 256 threads need no more than a 256-thread block
  const int grid = (int)std::min<long>(want, (long)blocks_per_sm[kst] * d.sms);
  MvArgs base;
  base.acc_prev = nullptr;
  base.c_prev = 0;
  base.vscale = nullptr;
  base.coef = d.coef;
  base.nz = d.coef_nz;
  base.w = make_wrap(d.cfg);
  base.N = d.N;
  base.ld = 4 * d.N;
  base.k = k;
  base.transpose = transpose;
  base.scale = dt;
  base.X = nullptr;
  base.Y = nullptr;
  base.acc = nullptr;
  base.c_acc = 0;
  int* vsteps = nullptr;
  if (hdts && hsteps) {
    double* vscale = c.buf + 4 * n;
    vsteps = reinterpret_cast<int*>(c.buf + 4 * n + k);
    if ((r = cuda_check(ctx, cudaMemcpyAsync(vscale, hdts, sizeof(double) * k, cudaMemcpyHostToDevice, st)))) return r;
    if ((r = cuda_check(ctx, cudaMemcpyAsync(vsteps, hsteps, sizeof(int) * k, cudaMemcpyHostToDevice, st)))) return r;
    base.vscale = vscale;
    nsteps = hsteps[0];
  }
  Taylor tc = taylor_coefficients(order);
  if (ffp) {
    MvFf bf;
    bf.coef = d.coef_ff;
    bf.nz = base.nz;
    bf.X = nullptr;
    bf.Y = nullptr;
    bf.acc = nullptr;
    bf.acc_prev = nullptr;
    bf.scale = dt;
    bf.c_acc = ff{0.0f, 0.0f};
    bf.c_prev = ff{0.0f, 0.0f};
    bf.vscale = base.vscale;
    bf.w = base.w;
    bf.N = base.N;
    bf.ld = base.ld;
    bf.k = k;
    bf.transpose = transpose;
    bf.chunk = chunk;
    float2* f1 = reinterpret_cast<float2*>(t1);
    float2* f2 = reinterpret_cast<float2*>(t2);
    float2* fo = reinterpret_cast<float2*>(vout);
    ResTile rt = ffmode == 1 ? res_tiling(base.w, d.sms, k) : ResTile{};
    if (ffmode == 1 && 4 * rt.tw * rt.th <= 1024 && res_smem(rt, k) <= kResSmem) {
      bool& ready = linear_state(ctx).res_ready;
      if (!ready && (r = cuda_check(ctx, cudaFuncSetAttribute(k_expm_res_ff, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                              (int)kResSmem))))
        return r;
      ready = true;
      rt.polls = d.res_polls;
      rt.gave_up = d.res_gave_up;
      // two buffers of 16 bytes per value: the four vectors of the other paths (v .. vout); no
      // term has number 0
      if ((r = cuda_check(ctx, cudaMemsetAsync(v, 0, sizeof(double) * 4 * n, st)))) return r;
      ulonglong2 *g0 = reinterpret_cast<ulonglong2*>(v), *g1 = reinterpret_cast<ulonglong2*>(t2);
      void* rargs[] = {&bf, &rt, &tc, &nsteps, &order, &dX, &dY, &g0, &g1, &vsteps};
      return cuda_check(ctx, cudaLaunchCooperativeKernel((const void*)k_expm_res_ff, rt.tx * rt.ty,
                                                         (4 * rt.tw * rt.th * rt.groups + 31) / 32 * 32, rargs, res_smem(rt, k), st));
    }
    void* fargs[] = {&bf, &tc, &nsteps, &order, &dX, &dY, &f1, &f2, &fo, &vsteps};
    return cuda_check(ctx, cudaLaunchCooperativeKernel(kern, grid, th, fargs,
                                                       kind == 2 ? ff_tile_smem<kVecChunk>() : 0, st));
  }
  if ((r = cuda_check(ctx, cudaMemcpyAsync(v, dX, sizeof(double) * n, cudaMemcpyDeviceToDevice, st)))) return r;
  if ((r = cuda_check(ctx, cudaMemcpyAsync(vout, dX, sizeof(double) * n, cudaMemcpyDeviceToDevice, st)))) return r;
  void* args[] = {&base, &tc, &nsteps, &order, &v, &t1, &t2, &vout, &vsteps};
  if ((r = cuda_check(ctx, cudaLaunchCooperativeKernel(kern, grid, th, args, 0, st))))
    return r;
  return cuda_check(ctx, cudaMemcpyAsync(dY, vout, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
}
}  // namespace

namespace hymor {
// Gives back the fixed-point parts of the blocks, which the FP64 matvec can do without; false
// where there are none, or the context's stream is being captured.
bool linear_spare_release(hymor_ctx* ctx) {
  LinearState* s = static_cast<LinearState*>(ctx_linear_state(ctx));
  if (!s || (!s->fx_mem[0] && !s->fx_mem[1]) || stream_captured(ctx)) return false;
  DevCtx& d = ctx_dev(ctx);
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // another stream's capture may be under way
  cudaThreadExchangeStreamCaptureMode(&mode);
  cudaStreamSynchronize(ctx_stream(ctx));
  for (int t = 0; t < 2; ++t) {
    lin_free(ctx, s->fx_mem[t], s->fx_bytes);
    s->fx_mem[t] = nullptr;
    d.fx_part[t] = nullptr;
    d.fx_ex[t] = nullptr;
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  return true;
}
// The context's other device memory, in and out of stream order: what is not to be had at first
// is tried again without the fixed-point parts.
cudaError_t ctx_malloc(hymor_ctx* ctx, void** p, size_t bytes) {
  return with_spare(ctx, [&]() { return cudaMalloc(p, bytes); });
}
cudaError_t ctx_malloc_async(hymor_ctx* ctx, void** p, size_t bytes) {
  return with_spare(ctx, [&]() { return cudaMallocAsync(p, bytes, ctx_stream(ctx)); });
}

// Called by hymor_ctx_destroy after its stream has drained.
void linear_state_release(void* p) {
  if (!p) return;
  LinearState* s = static_cast<LinearState*>(p);
  for (void* q : s->fx_mem)
    if (q) cudaFree(q);
  if (s->expm.buf) cudaFree(s->expm.buf);
  for (int g = 0; g < kLaneGroups; ++g) {
    if (s->lanes.st[g]) cudaStreamDestroy(s->lanes.st[g]);
    if (s->lanes.done[g]) cudaEventDestroy(s->lanes.done[g]);
  }
  if (s->lanes.mem) cudaFree(s->lanes.mem);
  if (s->lanes.fork) cudaEventDestroy(s->lanes.fork);
  delete s;  // the Krylov buffers are context allocations, freed with the context
}
}  // namespace hymor

extern "C" {

int hymor_linearize(hymor_ctx* ctx) {
  if (!ctx) return HYMOR_ERR_INVALID;
  int r = ensure_linear(ctx);
  if (r) return r;
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  const bool shock_blocks = d.cfg.shock_enabled && d.cfg.perturb_shock;
  JacLanes* L = nullptr;
  if ((shock_blocks && (r = ensure_shock(ctx))) || (r = ensure_lanes(ctx, &L))) return r;  // before S changes
  d.sj.on = 0;
  // LINEARIZE_L.jl:43-56: flow cells and shock BC, thermo, sound speed, boundary conditions
  if (d.cfg.shock_enabled) {
    launch_flow_cells(d, st);
    launch_thermo_sound(d, st);
    launch_shock_bc_flags(d, true, false, true, false, 1, st);
  }
  launch_thermo_sound(d, st);
  launch_shock_bc_flags(d, true, false, false, true, 1, st);
  std::vector<int> rows;
  if (shock_blocks) {
    rows.resize(d.nchi);
    cudaMemcpyAsync(rows.data(), d.cell_idx, sizeof(int) * d.nchi, cudaMemcpyDeviceToHost, st);
    if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
    if ((r = check_shock_rows_for_blocks(ctx, rows.data(), d.nchi, d.neta))) return r;
  }
  launch_jacobian_assemble(d, st, *L, rows.data());
  if ((r = cuda_check(ctx, cudaGetLastError()))) return r;
  if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  d.sj.on = shock_blocks;
  return 0;
}

int hymor_set_workspace_limit(hymor_ctx* ctx, uint64_t bytes) {
  if (!ctx) return HYMOR_ERR_INVALID;
  LinearState& s = linear_state(ctx);
  s.limit = bytes;
  s.fx_refused[0] = s.fx_refused[1] = -1;
  return 0;
}

int hymor_operator_size(hymor_ctx* ctx, int64_t* n) {
  if (!ctx || !n) return HYMOR_ERR_INVALID;
  *n = op_size(ctx_dev(ctx));
  return 0;
}

int hymor_shock_blocks_get(hymor_ctx* ctx, int32_t* rows, double* a21, double* a12, double* a22) {
  if (!ctx || !rows || !a21 || !a12 || !a22) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.sj.on) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no shock blocks: linearise with perturb_shock");
  cudaStream_t st = ctx_stream(ctx);
  const long n = d.nchi;
  cudaMemcpyAsync(rows, d.sj.rows, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(a21, d.sj.a21, sizeof(double) * 8 * n, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(a12, d.sj.a12, sizeof(double) * 4 * n * n, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(a22, d.sj.a22, sizeof(double) * n * n, cudaMemcpyDeviceToHost, st);
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_shock_blocks_set(hymor_ctx* ctx, const int32_t* rows, const double* a21, const double* a12,
                           const double* a22) {
  if (!ctx) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!rows) {
    d.sj.on = 0;
    return 0;
  }
  if (!a21 || !a12 || !a22) return HYMOR_ERR_INVALID;
  if (!d.cfg.shock_enabled) return ctx_fail(ctx, HYMOR_ERR_INVALID, "shock blocks need shock fitting");
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  int r;
  if ((r = check_shock_rows_for_blocks(ctx, rows, d.nchi, d.neta))) return r;
  if ((r = ensure_shock(ctx))) return r;
  cudaStream_t st = ctx_stream(ctx);
  const long n = d.nchi;
  cudaMemcpyAsync(d.sj.rows, rows, sizeof(int) * n, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d.sj.a21, a21, sizeof(double) * 8 * n, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d.sj.a12, a12, sizeof(double) * 4 * n * n, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d.sj.a22, a22, sizeof(double) * n * n, cudaMemcpyHostToDevice, st);
  k_transpose<<<grid_for(4 * n * n, 256), 256, 0, st>>>(d.sj.a12, d.sj.a12t, 4 * n, n);
  k_transpose<<<grid_for(n * n, 256), 256, 0, st>>>(d.sj.a22, d.sj.a22t, n, n);
  if ((r = cuda_check(ctx, cudaGetLastError()))) return r;
  if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  d.sj.on = 1;
  return 0;
}

int hymor_shock_fields(hymor_ctx* ctx, double* beta, double* rel_vel) {
  if (!ctx) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  const long n = d.nchi;
  std::vector<double> sc(2 * n);
  cudaMemcpyAsync(sc.data(), d.beta, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost, st);
  if (rel_vel) cudaMemcpyAsync(rel_vel, d.rel, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  int r = cuda_check(ctx, cudaStreamSynchronize(st));
  if (r) return r;
  if (beta)
    for (long i = 0; i < n; ++i) beta[i] = std::atan2(sc[i], sc[n + i]);
  return 0;
}

int hymor_jacobian_get(hymor_ctx* ctx, double* coef) {
  if (!ctx || !coef) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  cudaStream_t st = ctx_stream(ctx);
  double* tmp = nullptr;
  int r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&tmp, sizeof(double) * 144 * d.N)))) return r;
  k_planes_to_blocks<<<grid_for(d.N * 144, 256), 256, 0, st>>>(d.coef, tmp, d.N);
  r = cuda_check(ctx, cudaMemcpyAsync(coef, tmp, sizeof(double) * 144 * d.N, cudaMemcpyDeviceToHost, st));
  cudaFreeAsync(tmp, st);
  if (r) return r;
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_jacobian_set(hymor_ctx* ctx, const double* coef) {
  if (!ctx || !coef) return HYMOR_ERR_INVALID;
  int r = ensure_linear(ctx);
  if (r) return r;
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  double* tmp = nullptr;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&tmp, sizeof(double) * 144 * d.N)))) return r;
  r = cuda_check(ctx, cudaMemcpyAsync(tmp, coef, sizeof(double) * 144 * d.N, cudaMemcpyHostToDevice, st));
  cudaMemsetAsync(d.coef_nz + d.N, 0, 4 * d.N, st);
  k_blocks_to_planes<<<grid_for(d.N * 144, 256), 256, 0, st>>>(tmp, d.coef, d.coef_nz + d.N, d.N);
  k_masks<<<grid_for(d.N, 256), 256, 0, st>>>(d.coef_nz, d.coef_nz + d.N, make_wrap(d.cfg), d.N);
  ++d.coef_version;
  cudaFreeAsync(tmp, st);
  if (r) return r;
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

// Whether the fixed-point matvec takes k vectors, with its parts made (their storage on first
// use, whatever another stream of the caller captures; without the memory for it, and while the
// context's stream is captured, the FP64 matvec serves: a replay reads the blocks of its time).
static bool fx_ready(hymor_ctx* ctx, int k, int transpose) {
  DevCtx& d = ctx_dev(ctx);
  const int t = transpose != 0;
  if (!fx_takes(d, k) || stream_captured(ctx)) return false;
  if (!d.fx_part[t]) {
    LinearState& s = linear_state(ctx);
    if (s.fx_refused[t] == d.coef_version || ctx_select_device(ctx)) return false;
    void* p = nullptr;
    const size_t parts = sizeof(int2) * 144 * d.N, bytes = parts + sizeof(short) * 16 * d.N;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = lin_malloc(ctx, &p, bytes, true);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
      s.fx_refused[t] = d.coef_version;  // tried again after the next write of the blocks
      return false;
    }
    s.fx_mem[t] = p;
    s.fx_bytes = bytes;
    d.fx_part[t] = static_cast<int2*>(p);
    d.fx_ex[t] = reinterpret_cast<short*>(static_cast<char*>(p) + parts);
    d.fx_version[t] = d.coef_version - 1;
  }
  launch_fx_build(d, t, ctx_stream(ctx));
  return true;
}

int hymor_matvec_dev(hymor_ctx* ctx, int k, const double* dX, double* dY, int transpose) {
  if (!ctx || k < 1 || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  launch_matvec(d, k, dX, dY, transpose, 1.0, ctx_stream(ctx), 0, fx_ready(ctx, k, transpose));
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_matvec(hymor_ctx* ctx, int k, const double* X, double* Y, int transpose) {
  if (!ctx || k < 1 || !X || !Y) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  cudaStream_t st = ctx_stream(ctx);
  const size_t bytes = sizeof(double) * op_size(d) * (size_t)k;
  double *dx = nullptr, *dy = nullptr;
  int r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&dx, bytes)))) return r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&dy, bytes)))) return r;
  cudaMemcpyAsync(dx, X, bytes, cudaMemcpyHostToDevice, st);
  launch_matvec(d, k, dx, dy, transpose, 1.0, st, 0, fx_ready(ctx, k, transpose));
  cudaMemcpyAsync(Y, dy, bytes, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(dx, st);
  cudaFreeAsync(dy, st);
  if ((r = cuda_check(ctx, cudaGetLastError()))) return r;
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_bench_matvec(hymor_ctx* ctx, int k, const double* dX, double* dY, int transpose, int per_vector,
                       int reps, float* ms) {
  if (!ctx || k < 1 || !dX || !dY || reps < 1 || !ms) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  cudaStream_t st = ctx_stream(ctx);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int r;
  if ((r = cuda_check(ctx, cudaEventCreate(&e0)))) return r;
  if ((r = cuda_check(ctx, cudaEventCreate(&e1)))) {
    cudaEventDestroy(e0);
    return r;
  }
  const long n4 = op_size(d);
  const bool fx = !per_vector && fx_ready(ctx, k, transpose);
  cudaEventRecord(e0, st);
  for (int rep = 0; rep < reps; ++rep) {
    if (per_vector) {
      for (int v = 0; v < k; ++v) launch_matvec(d, 1, dX + v * n4, dY + v * n4, transpose, 1.0, st);
    } else {
      launch_matvec(d, k, dX, dY, transpose, 1.0, st, 0, fx);
    }
  }
  cudaEventRecord(e1, st);
  r = cuda_check(ctx, cudaEventSynchronize(e1));
  if (!r) r = cuda_check(ctx, cudaEventElapsedTime(ms, e0, e1));
  if (!r) r = cuda_check(ctx, cudaGetLastError());
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return r;
}

int hymor_expm_apply_dev(hymor_ctx* ctx, int k, double dt, int nsteps, int order, const double* dX, double* dY,
                         int transpose) {
  if (!ctx || k < 1 || nsteps < 0 || order < 1 || order > 20 || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  cudaStream_t st = ctx_stream(ctx);
  // the stencil operator in one cooperative launch, and with the shock blocks the extended one
  // (launch_expm); else each term is a launch sequence (launch_expm_body)
  if (!d.sj.on && (long)nsteps * (order + 1) >= kExpmCoopMinLaunches)
    return expm_cooperative(ctx, k, dt, nsteps, order, dX, dY, transpose);
  const size_t n = op_size(d) * (size_t)k;
  double* work = nullptr;
  int r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&work, 3 * n * sizeof(double))))) return r;
  launch_expm(d, k, dt, nsteps, order, dX, dY, transpose, work, st);
  cudaFreeAsync(work, st);
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_expm_apply_multi_dev(hymor_ctx* ctx, int k, const double* dts, const int32_t* nsteps, int order,
                               const double* dX, double* dY, int transpose) {
  if (!ctx || k < 1 || !dts || !nsteps || order < 1 || order > 20 || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  for (int c = 0; c < k; ++c)
    if (nsteps[c] < 0 || (c > 0 && nsteps[c] > nsteps[c - 1]))
      return ctx_fail(ctx, HYMOR_ERR_INVALID, "per-vector step counts must be non-negative and non-increasing");
  if (d.sj.on) {
    // the shock-position operator has no cooperative propagator: one vector at a time
    const long n = op_size(d);
    for (int c = 0; c < k; ++c) {
      const int r = hymor_expm_apply_dev(ctx, 1, dts[c], nsteps[c], order, dX + c * n, dY + c * n, transpose);
      if (r) return r;
    }
    return 0;
  }
  return expm_cooperative(ctx, k, 0.0, nsteps[0], order, dX, dY, transpose, dts, nsteps);
}

int hymor_expm_apply(hymor_ctx* ctx, int k, double dt, int nsteps, int order, const double* X, double* Y,
                     int transpose) {
  if (!ctx || k < 1 || !X || !Y) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  const size_t bytes = sizeof(double) * op_size(d) * (size_t)k;
  double *dx = nullptr, *dy = nullptr;
  int r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&dx, bytes)))) return r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&dy, bytes)))) return r;
  cudaMemcpyAsync(dx, X, bytes, cudaMemcpyHostToDevice, st);
  r = hymor_expm_apply_dev(ctx, k, dt, nsteps, order, dx, dy, transpose);
  if (!r) cudaMemcpyAsync(Y, dy, bytes, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(dx, st);
  cudaFreeAsync(dy, st);
  if (r || (r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  return ctx_check_waits(ctx);
}

}  // extern "C"

namespace {
KrylovScratch& kscratch(hymor_ctx* ctx) { return linear_state(ctx).kry; }
int ensure_scratch(hymor_ctx* ctx, int cols, long tmp_n) {
  KrylovScratch& k = kscratch(ctx);
  if (cols > k.cols) {
    void* p;
    if (lin_malloc(ctx, &p, sizeof(double) * (long)kDotBlocks * cols) != cudaSuccess)
      return ctx_fail(ctx, HYMOR_ERR_CUDA, "Krylov scratch allocation failed");
    ctx_allocs(ctx).push_back(p);
    k.partial = static_cast<double*>(p);
    if (lin_malloc(ctx, &p, sizeof(double) * (2 * cols + 4)) != cudaSuccess)
      return ctx_fail(ctx, HYMOR_ERR_CUDA, "Krylov scratch allocation failed");
    ctx_allocs(ctx).push_back(p);
    k.h = static_cast<double*>(p);
    k.cols = cols;
  }
  if (tmp_n > k.tmp_n) {
    void* p;
    if (lin_malloc(ctx, &p, sizeof(double) * tmp_n) != cudaSuccess)
      return ctx_fail(ctx, HYMOR_ERR_CUDA, "Krylov scratch allocation failed");
    ctx_allocs(ctx).push_back(p);
    k.tmp = static_cast<double*>(p);
    k.tmp_n = tmp_n;
  }
  return 0;
}
void dots(const double* A, long lda, int m, const double* w, long n, double* out, int mode, double* partial,
          cudaStream_t st) {
  k_dot_stage1<<<dim3(kDotBlocks, m), kDotThreads, 0, st>>>(A, lda, w, n, partial);
  k_dot_stage2<<<m, 32, 0, st>>>(partial, out, mode);
}
}  // namespace

extern "C" {

int hymor_dot_dev(hymor_ctx* ctx, int64_t n, int m, const double* dA, int64_t lda, const double* dw, double* out) {
  if (!ctx || n < 1 || m < 1 || !dA || !dw || !out) return HYMOR_ERR_INVALID;
  int r = ensure_scratch(ctx, m + 1, 0);
  if (r) return r;
  KrylovScratch& k = kscratch(ctx);
  cudaStream_t st = ctx_stream(ctx);
  dots(dA, lda, m, dw, n, k.h, 0, k.partial, st);
  cudaMemcpyAsync(out, k.h, sizeof(double) * m, cudaMemcpyDeviceToHost, st);
  if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  return ctx_check_waits(ctx);
}

int hymor_krylov_orthogonalize(hymor_ctx* ctx, int64_t n, int m, double* dV, int64_t ldv, double* dw, double* h,
                               int out_col) {
  if (!ctx || n < 1 || m < 0 || !dV || !dw || !h) return HYMOR_ERR_INVALID;
  int r = ensure_scratch(ctx, 2 * (m + 1), 0);
  if (r) return r;
  KrylovScratch& k = kscratch(ctx);
  cudaStream_t st = ctx_stream(ctx);
  const int gb = grid_for(n, 256);
  double* h1 = k.h;           // m
  double* nrm = k.h + 2 * (m + 1) - 1;
  if (m > 0) {
    for (int pass = 0; pass < 2; ++pass) {  // classical Gram-Schmidt, twice
      double* hp = pass == 0 ? h1 : h1 + m;
      dots(dV, ldv, m, dw, n, hp, 0, k.partial, st);
      k_gemv_sub<<<gb, 256, sizeof(double) * m, st>>>(dV, ldv, n, m, hp, dw);
    }
  }
  dots(dw, n, 1, dw, n, nrm, 0, k.partial, st);
  if (out_col >= 0) k_normalize<<<gb, 256, 0, st>>>(dw, dV + (long)out_col * ldv, n, nrm);
  std::vector<double> hh(2 * m + 1);
  if (m > 0) cudaMemcpyAsync(hh.data(), h1, sizeof(double) * 2 * m, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(hh.data() + 2 * m, nrm, sizeof(double), cudaMemcpyDeviceToHost, st);
  if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  if ((r = ctx_check_waits(ctx))) return r;  // the vector came from a propagation that gave up
  for (int j = 0; j < m; ++j) h[j] = hh[j] + hh[m + j];
  h[m] = std::sqrt(hh[2 * m]);
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_krylov_rotate(hymor_ctx* ctx, int64_t n, int m, int kk, double* dV, int64_t ldv, const double* Q) {
  if (!ctx || n < 1 || m < 1 || kk < 1 || kk > m || !dV || !Q) return HYMOR_ERR_INVALID;
  int r = ensure_scratch(ctx, 1, n * kk + (long)m * kk);
  if (r) return r;
  KrylovScratch& k = kscratch(ctx);
  cudaStream_t st = ctx_stream(ctx);
  double* dQ = k.tmp + n * kk;
  cudaMemcpyAsync(dQ, Q, sizeof(double) * m * kk, cudaMemcpyHostToDevice, st);
  k_rotate<<<grid_for(n, 128), 128, 0, st>>>(dV, ldv, n, m, kk, dQ, k.tmp, n);
  for (int c = 0; c < kk; ++c)
    cudaMemcpyAsync(dV + (long)c * ldv, k.tmp + (long)c * n, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
  if ((r = cuda_check(ctx, cudaGetLastError()))) return r;
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_linearize_b(hymor_ctx* ctx) {
  if (!ctx) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.cfg.shock_enabled) return ctx_fail(ctx, HYMOR_ERR_INVALID, "the upstream-boundary operator needs shock fitting");
  int r = ensure_linear(ctx);
  if (r || (r = ensure_b(ctx))) return r;
  cudaStream_t st = ctx_stream(ctx);
  std::vector<int> rows(d.nchi);
  cudaMemcpyAsync(rows.data(), d.cell_idx, sizeof(int) * d.nchi, cudaMemcpyDeviceToHost, st);
  if ((r = cuda_check(ctx, cudaStreamSynchronize(st)))) return r;
  if ((r = check_b_rows(ctx, rows.data(), d.nchi, d.neta))) return r;
  JacLanes* L = nullptr;
  if ((r = ensure_lanes(ctx, &L))) return r;
  launch_b_assemble(d, st, *L);
  if ((r = cuda_check(ctx, cudaGetLastError()))) return r;
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_b_get(hymor_ctx* ctx, int32_t* rows, double* bq, double* bs) {
  if (!ctx || !rows || !bq) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.bq) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no upstream-boundary operator: call hymor_linearize_b");
  cudaStream_t st = ctx_stream(ctx);
  cudaMemcpyAsync(rows, d.brows, sizeof(int) * d.nchi, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(bq, d.bq, sizeof(double) * 48 * d.nchi, cudaMemcpyDeviceToHost, st);
  if (bs) cudaMemcpyAsync(bs, d.bs, sizeof(double) * 12 * d.nchi, cudaMemcpyDeviceToHost, st);
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_b_set(hymor_ctx* ctx, const int32_t* rows, const double* bq, const double* bs) {
  if (!ctx || !rows || !bq || !bs) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  int r;
  if ((r = check_b_rows(ctx, rows, d.nchi, d.neta)) || (r = ensure_b(ctx))) return r;
  cudaStream_t st = ctx_stream(ctx);
  cudaMemcpyAsync(d.brows, rows, sizeof(int) * d.nchi, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d.bq, bq, sizeof(double) * 48 * d.nchi, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(d.bs, bs, sizeof(double) * 12 * d.nchi, cudaMemcpyHostToDevice, st);
  return cuda_check(ctx, cudaStreamSynchronize(st));
}

int hymor_recept_size(hymor_ctx* ctx, int nw, int64_t* n) {
  if (!ctx || nw < 0 || !n) return HYMOR_ERR_INVALID;
  *n = recept_size(ctx_dev(ctx), nw);
  return 0;
}

// the frequencies on the device for one call (freed in stream order)
static int recept_prep(hymor_ctx* ctx, int k, int nw, const double* w, const double* dX, double* dY, double** dw) {
  if (!ctx || k < 1 || nw < 1 || !w || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  if (!d.coef) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no Jacobian: call hymor_linearize or hymor_jacobian_set");
  if (!d.bq) return ctx_fail(ctx, HYMOR_ERR_NOT_READY, "no upstream-boundary operator: call hymor_linearize_b");
  cudaStream_t st = ctx_stream(ctx);
  int r;
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)dw, sizeof(double) * nw)))) return r;
  return cuda_check(ctx, cudaMemcpyAsync(*dw, w, sizeof(double) * nw, cudaMemcpyHostToDevice, st));
}

int hymor_recept_apply_dev(hymor_ctx* ctx, int k, int nw, const double* w, double scale, const double* dX, double* dY,
                           int adjoint) {
  double* dw = nullptr;
  int r = recept_prep(ctx, k, nw, w, dX, dY, &dw);
  if (r) return r;
  cudaStream_t st = ctx_stream(ctx);
  launch_recept_apply(ctx_dev(ctx), k, nw, dw, dX, dY, adjoint, scale, st);
  cudaFreeAsync(dw, st);
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_recept_expm_dev(hymor_ctx* ctx, int k, int nw, const double* w, double dt, int nsteps, int order,
                          const double* dX, double* dY, int adjoint) {
  if (nsteps < 0 || order < 1 || order > 20) return HYMOR_ERR_INVALID;
  double* dw = nullptr;
  int r = recept_prep(ctx, k, nw, w, dX, dY, &dw);
  if (r) return r;
  DevCtx& d = ctx_dev(ctx);
  cudaStream_t st = ctx_stream(ctx);
  // (k_expm_ext counts its items in 32 bits)
  if (expm_ext_fits(d, 2 * k, nsteps, order, kExtRecept) && 8L * k * d.nchi * nw < (1L << 30)) {
    ExtArgs a = ext_args(d, 2 * k, dt);
    a.bq = d.bq;
    a.bs = d.bs;
    a.w = dw;
    a.brows = d.brows;
    a.ld = recept_size(d, nw);
    a.nw = nw;
    a.divide = 1;
    double* work = nullptr;
    if (!(r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&work, sizeof(double) * 2 * a.ld * a.k)))) {
      r = cuda_check(ctx, launch_expm_ext(d, a, adjoint, nsteps, order, dX, dY, work, st));
      cudaFreeAsync(work, st);
    }
    cudaFreeAsync(dw, st);
    return r;
  }
  double* work = nullptr;
  const long n = 2L * k * recept_size(d, nw);
  if ((r = cuda_check(ctx, ctx_malloc_async(ctx, (void**)&work, sizeof(double) * 2 * n)))) return r;
  launch_recept_expm(d, k, nw, dw, dt, nsteps, order, dX, dY, adjoint, work, st);
  cudaFreeAsync(work, st);
  cudaFreeAsync(dw, st);
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_block4_apply_ext_dev(hymor_ctx* ctx, int k, int64_t ntail, const double* dB, const double* dTail,
                               const double* dX, double* dY) {
  if (!ctx || k < 1 || ntail < 0 || !dB || (ntail && !dTail) || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  k_block4_tail<<<grid_for(d.N * k, 256), 256, 0, ctx_stream(ctx)>>>(dB, dTail, dX, dY, d.N, ntail, k);
  return cuda_check(ctx, cudaGetLastError());
}

int hymor_block4_apply_dev(hymor_ctx* ctx, int k, const double* dB, const double* dX, double* dY) {
  if (!ctx || k < 1 || !dB || !dX || !dY) return HYMOR_ERR_INVALID;
  DevCtx& d = ctx_dev(ctx);
  k_block4<<<grid_for(d.N * k, 256), 256, 0, ctx_stream(ctx)>>>(dB, dX, dY, d.N, k);
  return cuda_check(ctx, cudaGetLastError());
}

}  // extern "C"
