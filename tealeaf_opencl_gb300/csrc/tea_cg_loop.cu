// The device-resident CG loop as one cooperative launch: tea_solve.f90:270-330
// with w = A p, the u/r/z update and p = z + beta p of tea_leaf_cg_cl.cl
// folded into two passes per iteration.
//
//   pass A  p' = z + beta p formed where w = A p' needs it (own cells and the
//           cells around them), u += alpha p of the iteration before, w and
//           the tile sums of p'.w
//   pass B  r -= alpha w, z = M^-1 r, the tile sums of r.z
//
// Every value is computed by the expressions of the per-call kernels (calc_w,
// calc_ur, calc_p) from the same operands, and every sum takes the fixed order
// of tea_device.cuh, so the results are theirs bit for bit.  The same passes as
// kernels of their own, for larger grids, are at the end of the file.
#include <string.h>

#include <algorithm>

#include "tea_cg.cuh"
#include "tea_device.cuh"
#include "tea_loop.cuh"
#include "tea_resident_launch.h"

namespace tea {

namespace {

// One block of 512 threads with 128 registers per SM: four rows of a tile's 33
// loads are in flight at once, and 16 warps keep the FP64 pipe busy while some
// wait (1024 threads with 64 registers, row by row: 480 us per iteration at
// 4096^2 against 417, 18.8 against 16.4 at 512^2 in the same state of the
// kernel).  Small grids are bound by latency: of 31 thousand cycles per
// iteration at 512^2 pass A takes 14, pass B 6, the two barriers and sums 11.
// Middle ones by the FP64 pipe, 59 % busy at 1501x1203 block Jacobi (the last
// round of supertiles is half full, and all loads of a round start together).
constexpr int kLoopThreads = 512;
constexpr int kLoopWarps = kLoopThreads / 32;
constexpr int kLoopSlots = kLoopWarps / kTilesPerSuper;  // supertiles in flight
constexpr int kLoopBatch = 4;                   // rounds whose tile sums share a sweep

// why the loop left
enum { kStopConverged = 1, kStopLoopMax, kStopSwitch, kStopLaunch, kStopPw, kStopRz };

struct LoopShared {
  double lanes[kLoopBatch * kLoopThreads];  // lane sums of a batch of rounds
  double tiles[kLoopBatch * kLoopWarps];    // its tile sums, supertile by supertile
  double alpha, beta;
  int go;      // barrier passed
  int stop;    // the loop ends after this iteration
};

// The least non-negative x with sqrt(x) >= t, so that sqrt(x) < t can be
// tested without the square root (monotonic), or -1 where t^2 leaves the
// normal range and the root must be taken.
__device__ __forceinline__ double square_limit(double t) {
  double x = t * t;
  if (!(x > 1e-290 && x < 1e290)) return -1.0;
  for (int k = 0; k < 16 && sqrt(x) >= t; k++)
    x = __longlong_as_double(__double_as_longlong(x) - 1);
  for (int k = 0; k < 32 && sqrt(x) < t; k++)
    x = __longlong_as_double(__double_as_longlong(x) + 1);
  return sqrt(x) >= t && sqrt(__longlong_as_double(__double_as_longlong(x) - 1)) < t ? x : -1.0;
}

// Runs body(x, y0) -> lane sum over the block's supertiles and stores the
// supertile partials.  A warp writes its lane sums to shared memory and
// whole warps then sum four tiles each (bfly4) and four supertiles each
// (the steps of supertile_partials4): 1.5 FP64 instructions per tile however
// few tiles the block has.
template <int TH, bool SUM, class Body>
__device__ __forceinline__ void loop_pass(const Dev& d, double* partials, LoopShared& sh,
                                          Body body) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = warp / kTilesPerSuper, tile = warp % kTilesPerSuper;
  const int nb = gridDim.x, b = blockIdx.x;
  const int mine = b < d.ns ? (d.ns - 1 - b) / nb + 1 : 0;  // supertiles b, b+nb, ...
  const int rounds = (mine + kLoopSlots - 1) / kLoopSlots;
  for (int r0 = 0; r0 < rounds; r0 += kLoopBatch) {
    const int nr = min(kLoopBatch, rounds - r0);
    for (int k = 0; k < nr; k++) {
      const long long s = b + (long long)nb * ((r0 + k) * kLoopSlots + slot);
      double acc = 0.0;
      if (s < d.ns) {
        const int sy = (int)s / d.nsx, sx = (int)s - sy * d.nsx;
        const int tx = sx * kTilesPerSuper + tile;
        if (tx < d.ntx) acc = body(tx * kTileW + lane, sy * TH);
      }
      if (SUM) sh.lanes[k * kLoopThreads + threadIdx.x] = acc;
    }
    if (!SUM) continue;
    __syncthreads();
    if (warp < nr * (kLoopWarps / 4)) {
      const double* a = sh.lanes + warp * 128 + lane;
      const double t = bfly4(a[0], a[32], a[64], a[96]);
      if ((lane & 7) == 0) sh.tiles[warp * 4 + bfly4_slot(lane)] = t;
    }
    __syncthreads();
    if (warp * 4 < nr * kLoopSlots) {
      double t = plus_zero(sh.tiles[warp * 32 + lane]);
#pragma unroll
      for (int off = 4; off >= 1; off >>= 1) t = t + __shfl_xor_sync(0xffffffffu, t, off);
      const int q = warp * 4 + (lane >> 3);  // supertile of the batch
      const long long s = b + (long long)nb * (r0 * kLoopSlots + q);
      if ((lane & 7) == 0 && q < nr * kLoopSlots && s < d.ns) __stcg(partials + s, t);
    }
  }
}

template <int TH, int F, bool EMU>
__global__ void __launch_bounds__(kLoopThreads, 1)
    k_cg_loop(Dev d, double* p2, Red red, ResState* st, unsigned int* bar, int* err,
              long long spin_limit, unsigned int extra, int iters) {
  __shared__ LoopShared sh;
  double* const pw_parts = red.partials;
  double* const rz_parts = red.partials + red.stride;
  const double* zsrc = d.prec != PREC_NONE ? d.z : d.r;
  const unsigned int arrivals = gridDim.x + extra;
  unsigned int target = 0;
  double* const alphas = st->alphas;
  double* const betas = st->betas;
  double rro = st->rro;  // kept up to date by thread 0
  int n = st->n;
  const int loop_max = st->loop_max, check = st->check;
  const double eps_target = st->eps_target, switch_eps = st->switch_eps;
  const int switch_n = st->switch_n;
  const double rr_limit = threadIdx.x == 32 ? square_limit(eps_target) : 0.0;
  double alpha = 0.0, beta = 0.0;
  int it = 0, stop = 0;
  for (;; it++, n++) {
    // p alternates between d.p and p2; the first iteration finds it in d.p
    const double* pin = (it & 1) || !it ? d.p : p2;
    double* pout = (it & 1) ? p2 : d.p;
    const bool first = it == 0;
    loop_pass<TH, true>(d, pw_parts, sh, [&](int x, int y0) {
      return loop_w_tile<TH, F, false, EMU>(d, pin, pout, zsrc, x, y0, alpha, beta, first);
    });
    target += arrivals;
    if (!loop_barrier(bar, err, &st->timed_out, target, spin_limit, &sh.go)) return;
    const double pw = loop_total(pw_parts, d.ns, sh.lanes, sh.tiles);
    if (threadIdx.x == 0) sh.alpha = rro / pw;
    __syncthreads();
    alpha = sh.alpha;
    loop_pass<TH, true>(d, rz_parts, sh, [&](int x, int y0) {
      double acc[1] = {0.0};
      loop_r_tile<TH, F, 1, EMU>(d, x, y0, alpha, acc);
      return acc[0];
    });
    target += arrivals;
    if (!loop_barrier(bar, err, &st->timed_out, target, spin_limit, &sh.go)) return;
    const double rrn = loop_total(rz_parts, d.ns, sh.lanes, sh.tiles);
    // the host steps of the iteration (cg_scalar_step): beta by thread 0, the
    // exit test beside it by thread 32
    if (threadIdx.x == 0) {
      const double bt = rrn / rro;
      sh.beta = bt;
      if (blockIdx.x == 0) {
        if (alphas) {
          alphas[n] = alpha;
          betas[n] = bt;
        }
      }
      rro = rrn;
    }
    if (threadIdx.x == 32) {
      const bool done = rr_limit > 0.0 ? rrn < rr_limit && rrn >= 0.0 : sqrt(rrn) < eps_target;
      const bool sw = switch_n > 0 && n + 1 >= switch_n && sqrt(rrn) <= switch_eps;
      int s = done              ? kStopConverged
              : n >= loop_max   ? kStopLoopMax
              : sw              ? kStopSwitch
              : it + 1 >= iters ? kStopLaunch
                                : 0;
      if (check) {
        if (!(pw > 0.0) || isinf(pw))
          s = kStopPw;
        else if (!isfinite(rrn))
          s = kStopRz;
      }
      if (blockIdx.x == 0 && s && s < kStopPw) st->error = sqrt(rrn);
      sh.stop = s;
    }
    __syncthreads();
    beta = sh.beta;
    stop = sh.stop;
    if (stop) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (stop >= kStopPw) {
      st->breakdown = stop == kStopPw ? 1 : 2;
      st->breakdown_n = n;
    } else {
      st->alpha = alpha;
      st->beta = beta;
      st->rro = st->rrn = rro;
      st->converged = stop == kStopConverged;
    }
    st->n = stop == kStopLaunch ? n + 1 : n;
    st->stop = stop != kStopLaunch;
    st->p_pending = 0;
  }
  // u and p of the last iteration (p stays as it is after a breakdown)
  const double* pc = (it & 1) ? p2 : d.p;
  loop_pass<TH, false>(d, pw_parts, sh, [&](int x, int y0) {
    if (x >= d.x_max) return 0.0;
    const int rows = min(TH, d.y_max - y0);
    for (int j = 0; j < rows; j++) {
      const long long c = cidx(d, x, y0 + j);
      const double po = __ldcg(pc + c), uv = d.u[c];
      d.u[c] = F ? __fma_rn(alpha, po, uv) : uv + alpha * po;
      if (stop < kStopPw) d.p[c] = p_next<F>(beta, po, __ldcg(zsrc + c));
    }
    return 0.0;
  });
}

// Jacobi sweeps until the exit test ends them, at most `iters` (even): u
// alternates between d.u and u2 (whose halo ring becomes u's), one grid barrier
// per sweep, the old u of the last one into un.  A sweep through the per-call
// path costs a launch and a host round trip, about 20 us on small grids.
template <bool EMU>
__global__ void __launch_bounds__(kLoopThreads, 1)
    k_jacobi_loop(Dev d, double* u2, Red red, ResState* st, unsigned int* bar, int* err,
                  long long spin_limit, unsigned int extra, int iters) {
  constexpr int TH = 4;  // jacobi_loop_fits
  __shared__ LoopShared sh;
  const unsigned int arrivals = gridDim.x + extra;
  unsigned int target = 0;
  int n = st->n, it = 0, stop = 0;
  const int loop_max = st->loop_max;
  const double eps_target = st->eps_target;
  const double rr_limit = threadIdx.x == 32 ? square_limit(eps_target) : 0.0;
  copy_halo_ring(d, d.u, u2);
  for (;; it++, n++) {
    const double* cur = (it & 1) ? u2 : d.u;
    double* nxt = (it & 1) ? d.u : u2;
    // partials alternate too: a block may still read the last sweep's
    double* parts = red.partials + (it & 1) * red.stride;
    loop_pass<TH, true>(d, parts, sh, [&](int x, int y0) {
      return x < d.x_max ? jacobi_tile<TH, true, EMU>(d, cur, nxt, nullptr, x, y0) : 0.0;
    });
    target += arrivals;
    if (!loop_barrier(bar, err, &st->timed_out, target, spin_limit, &sh.go)) return;
    const double sum = loop_total(parts, d.ns, sh.lanes, sh.tiles);
    if (threadIdx.x == 32) {
      const bool done = rr_limit > 0.0 ? sum < rr_limit && sum >= 0.0 : sqrt(sum) < eps_target;
      const int s = done              ? kStopConverged
                    : n >= loop_max   ? kStopLoopMax
                    : it + 1 >= iters ? kStopLaunch
                                      : 0;
      if (blockIdx.x == 0 && s) st->error = sqrt(sum);
      sh.stop = s;
    }
    __syncthreads();
    stop = sh.stop;
    if (stop) break;
  }
  const double* old = (it & 1) ? u2 : d.u;
  loop_pass<TH, false>(d, red.partials, sh, [&](int x, int y0) {
    if (x < d.x_max)
      for (int y = y0; y < min(y0 + TH, d.y_max); y++) d.un[cidx(d, x, y)] = old[cidx(d, x, y)];
    return 0.0;
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->converged = stop == kStopConverged;
    st->n = stop == kStopLaunch ? n + 1 : n;
    st->stop = stop != kStopLaunch;
  }
}

// ---- the two passes as separate kernels, for grids whose passes are long
// beside a launch (replayed from a graph) ----

// Blocks per SM by measurement.  Pass A at 128 registers: 391 us per iteration
// at 4096^2 diagonal, 474 and 504 at three and four blocks; pass B streams at
// four (392, 412 at three, two).  The exact form's pass B needs more registers
// (its strip divides): three blocks, 3000^2 block Jacobi 468 -> 458 us.
//
// In the exact form, bound by the FP64 pipe throughout, the two passes fell
// behind three kernels on large grids until the products by alpha and beta moved
// to the integer pipes (PE), but for few supertiles, where the FP64 pipe's own
// are quicker (few_supertiles).  us per iteration, three kernels / two passes
// before / after: 3000x2900 none 355 / 374 / 334, block 430 / 447 / 410;
// 1800x1700 none 160 / 164 / 154, block 192 / 194 / 184; with the true-residual
// exit 3000x2900 none 399 / 416 / 374, 1800x1700 none 169 / 182 / 170.

// Pass A.  An iteration whose predecessor has run (p_pending) forms p' and
// finishes u; the first one copies p, so that p alternates between the two
// buffers whatever happens.
template <int TH, int F, bool PE>
__global__ void __launch_bounds__(kBlock, 2)
    k_cg_pass_w(Dev d, Red red, ResState* st, const double* pin, double* pout) {
  if (*(volatile int*)&st->stop) return;
  const bool first = !*(volatile int*)&st->p_pending;
  const double alpha = st->alpha, beta = st->beta;
  const double* zsrc = d.prec != PREC_NONE ? d.z : d.r;
  const bool last = tile_driver<TH, 1>(d, red, [&](int x, int y0, bool, double* acc) {
    acc[0] = loop_w_tile<TH, F, true, true, PE>(d, pin, pout, zsrc, x, y0, alpha, beta, first);
  });
  if (last && threadIdx.x == 0) {
    const double pw = red.result[0];
    st->pw = pw;
    st->alpha = st->rro / pw;
  }
}

// Pass B and the scalar step; with NV = 2 also r.r for the exit test on the
// unpreconditioned residual.
template <int TH, int F, int NV, bool PE>
__global__ void __launch_bounds__(kBlock, F ? 4 : 3) k_cg_pass_r(Dev d, Red red, ResState* st) {
  if (*(volatile int*)&st->stop) return;
  const double alpha = st->alpha;
  const bool last = tile_driver<TH, NV>(d, red, [&](int x, int y0, bool, double* acc) {
    loop_r_tile<TH, F, NV, true, PE>(d, x, y0, alpha, acc);
  });
  if (last && threadIdx.x == 0) cg_scalar_step<NV>(st, alpha, red.result);
}

// u and p of the iteration that stopped the loop, p to d.p: it is in p2
// after an odd number of iterations.
template <int TH, int F>
__global__ void __launch_bounds__(kBlock)
    k_cg_pass_end(Dev d, Red red, ResState* st, const double* p2, unsigned int* counter) {
  if (!*(volatile int*)&st->stop || st->ended) return;
  const bool odd = ((st->n - st->n_first + 1) & 1) != 0;
  const bool brk = st->breakdown != 0;
  const double* pc = odd ? p2 : d.p;
  const double alpha = st->alpha, beta = st->beta;
  const double* z = d.prec != PREC_NONE ? d.z : d.r;
  tile_driver<TH, 0>(d, red, [&](int x, int y0, bool xin, double*) {
    if (!xin) return;
    const int rows = min(TH, d.y_max - y0);
    for (int j = 0; j < rows; j++) {
      const long long c = cidx(d, x, y0 + j);
      const double po = pc[c], uv = d.u[c];
      d.u[c] = F ? __fma_rn(alpha, po, uv) : uv + alpha * po;
      if (!brk) d.p[c] = p_next<F>(beta, po, z[c]);
    }
  });
  if (last_block(counter) && threadIdx.x == 0) {
    st->ended = 1;
    st->p_pending = 0;
  }
}

template <class... KArgs>
int pass_grid(const LaunchCtx& l, const Dev& d, void (*kernel)(KArgs...)) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  return (int)std::max<long long>(1, std::min<long long>(d.ns, (long long)l.num_sms * per_sm));
}

template <int TH, int F, int NV>
void enqueue_passes_t(const LaunchCtx& l, const Dev& d, double* p2, const Red& red,
                      ResState* st, unsigned int* counter, int iters) {
  auto* pass_w = k_cg_pass_w<TH, F, F == 0>;
  auto* pass_r = k_cg_pass_r<TH, F, NV, F == 0>;
  if constexpr (F == 0 && TH == 4)
    if (few_supertiles(d, l.num_sms)) {
      pass_w = k_cg_pass_w<TH, F, false>;
      pass_r = k_cg_pass_r<TH, F, NV, false>;
    }
  const int gw = pass_grid(l, d, pass_w);
  const int gr = pass_grid(l, d, pass_r);
  const int ge = pass_grid(l, d, k_cg_pass_end<TH, F>);
  for (int i = 0; i < iters; i += 2) {
    pass_w<<<gw, kBlock, 0, l.stream>>>(d, red, st, d.p, p2);
    pass_r<<<gr, kBlock, 0, l.stream>>>(d, red, st);
    pass_w<<<gw, kBlock, 0, l.stream>>>(d, red, st, p2, d.p);
    pass_r<<<gr, kBlock, 0, l.stream>>>(d, red, st);
  }
  k_cg_pass_end<TH, F><<<ge, kBlock, 0, l.stream>>>(d, red, st, p2, counter);
}

// A loop kernel on a block per SM, or per supertile where there are fewer.
cudaError_t launch_loop_blocks(const LaunchCtx& l, const Dev& d, const void* fn, void** args) {
  return launch_resident(std::max(1, std::min(d.ns, l.num_sms)), [&](int blocks) {
    return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(kLoopThreads), args, 0, l.stream);
  });
}

template <int TH, int F>
bool launch_loop_t(const LaunchCtx& l, Dev d, double* p2, Red red, ResState* st,
                   unsigned int* bar, long long spin_limit, unsigned int extra, int iters) {
  int* err = (int*)(bar + 1);
  void* args[] = {&d, &p2, &red, &st, &bar, &err, &spin_limit, &extra, &iters};
  const void* fn = (const void*)k_cg_loop<TH, F, true>;
  if constexpr (TH == 4)
    if (few_supertiles(d, l.num_sms)) fn = (const void*)k_cg_loop<TH, F, false>;
  return check_cuda(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned int), l.stream),
                    "CG loop barrier reset") &&
         check_cuda(launch_loop_blocks(l, d, fn, args), "CG loop launch");
}

}  // namespace

bool launch_jacobi_loop(const LaunchCtx& l, const Dev& d_, double* u2, const Red& red_,
                        ResState* st, unsigned int* bar, long long spin_limit,
                        unsigned int extra) {
  Dev d = d_;
  Red red = red_;
  int iters = kLoopLaunchIters;
  int* err = (int*)(bar + 1);
  void* args[] = {&d, &u2, &red, &st, &bar, &err, &spin_limit, &extra, &iters};
  const void* fn = few_supertiles(d, l.num_sms) ? (const void*)k_jacobi_loop<false>
                                                : (const void*)k_jacobi_loop<true>;
  count_launch("resident_jacobi_loop");
  return check_cuda(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned int), l.stream),
                    "Jacobi loop barrier reset") &&
         check_cuda(launch_loop_blocks(l, d, fn, args), "Jacobi loop launch");
}

// The line between the one launch and separate kernels, in supertiles of 4 rows
// per SM (one of 16 rows is the work of four).  A launch boundary costs a pass
// 8-10 us (start, drain, the last block's sum), a grid barrier with the sum in
// every block 2.5 us; but the cooperative kernel's passes share one register
// budget (16 warps per SM), so long passes run at 0.8-0.95 of the rate of their
// own kernels, and a block takes supertiles two at a time, so its time steps up
// where a further round begins.  us per CG iteration, graph / one launch, at 1501
// columns (2 per SM are a round):
//   per SM, within 0.2      9.0         10.0        11.1        12.0        12.2        13.9
//   diagonal, chain     50.3 / 49.4 55.1 / 53.6 60.7 / 61.2 62.7 / 63.2 65.5 / 69.5 69.7 / 71.5
//   block, chain        56.6 / 54.7 61.3 / 59.0 67.6 / 67.2 69.2 / 69.4 72.6 / 76.1
//   block, fused        57.8 / 56.8 62.9 / 61.1 69.2 / 69.6 71.1 / 71.8 74.8 / 79.1 79.4 / 81.6
//   none, chain         47.9 / 42.0 50.3 / 45.0 55.5 / 52.6 59.9 / 56.8             66.9 / 65.7
//   block, exact        84.5 / 81.5 91.4 / 88.6  101 / 98.3  104 / 104   111 / 113   121 / 119
// So the line is where the seventh round begins; without a preconditioner and in
// the exact form it is where the eighth does (14.2 per SM: none fused 71.3 / 74.2,
// block exact 124 / 127).  In 16-row tiles, 32 per SM and more, the graph is ahead
// throughout: diagonal fused 2176^2 143 / 149, 2500^2 172 / 186, 2800^2 208 / 219.
static int rows4_supertiles(const Dev& d) { return d.ns * (d.th / 4); }
bool cg_loop_fits(const Dev& d, int num_sms, int arith) {
  const int per_sm = arith != 0 && d.prec != PREC_NONE ? 12 : 14;
  return rows4_supertiles(d) <= per_sm * num_sms;
}

// Jacobi: one barrier per sweep in place of a launch and a host round trip.  us
// per sweep, per call / one launch: 64^2 16.0 / 9.3, 512^2 20.9 / 14.3; at 1501
// columns 9.9 per SM 60.1 / 54.1, 13.9 79.9 / 73.1, 15.9 89.4 / 83.9, 17.9 99.9 /
// 98.5; 1600^2 (18.4) 94.4 / 100.2, 2048^2 145 / 152, 2500^2 222 / 234.
bool jacobi_loop_fits(const Dev& d, int num_sms) { return rows4_supertiles(d) <= 18 * num_sms; }

void enqueue_cg_passes(const LaunchCtx& l, const Dev& d, double* p2, const Red& red,
                       ResState* st, unsigned int* counter, int iters, bool true_exit) {
#define TEA_PASSES(TH, NV)                                                           \
  (l.arith == 2   ? enqueue_passes_t<TH, 2, NV>(l, d, p2, red, st, counter, iters) \
   : l.arith == 1 ? enqueue_passes_t<TH, 1, NV>(l, d, p2, red, st, counter, iters) \
                  : enqueue_passes_t<TH, 0, NV>(l, d, p2, red, st, counter, iters))
  if (d.th == 16)
    true_exit ? TEA_PASSES(16, 2) : TEA_PASSES(16, 1);
  else
    true_exit ? TEA_PASSES(4, 2) : TEA_PASSES(4, 1);
#undef TEA_PASSES
}

bool launch_cg_loop(const LaunchCtx& l, const Dev& d, double* p2, const Red& red, ResState* st,
                    unsigned int* bar, long long spin_limit, unsigned int extra) {
  const int iters = kLoopLaunchIters;
  count_launch("resident_cg_loop");
  if (d.th == 16)
    return l.arith == 2 ? launch_loop_t<16, 2>(l, d, p2, red, st, bar, spin_limit, extra, iters)
         : l.arith == 1 ? launch_loop_t<16, 1>(l, d, p2, red, st, bar, spin_limit, extra, iters)
                        : launch_loop_t<16, 0>(l, d, p2, red, st, bar, spin_limit, extra, iters);
  return l.arith == 2 ? launch_loop_t<4, 2>(l, d, p2, red, st, bar, spin_limit, extra, iters)
       : l.arith == 1 ? launch_loop_t<4, 1>(l, d, p2, red, st, bar, spin_limit, extra, iters)
                      : launch_loop_t<4, 0>(l, d, p2, red, st, bar, spin_limit, extra, iters);
}

}  // namespace tea
