// GB300 (sm_103a) kernels of one NSW6 microphysics step, FP64.
//
// Four kernels per step:
//
//  nsw6_cell_kernel    one CTA = a tile of consecutive interior cells of one
//                      region.  Per cell: negative filter, saturation values,
//                      Bergeron parameters, the NSW6 process rates, the
//                      RHOGQ/RHOGE/TEM updates and the fall speeds.
//
//  nsw6_departure_kernel  one CTA = DEP_TG columns x all levels of one falling
//                      tracer: the sedimentation departure distances of
//                      vadv1d_prep on full and half levels and their per-level
//                      extrema, reduced over the region with exact
//                      order-preserving 64-bit atomics.
//
//  nsw6_column_kernel  one CTA = COL_TG columns x all levels, column state in
//                      shared memory.  Departure cells, the 24 flux integrals of
//                      vadv1d_getflux_new, the transport tendencies, surface
//                      precipitation, the KIN2EIN energy correction, the final
//                      thermodynamic state and the closing negative filter; the
//                      cells the saturation adjustment finds saturated are
//                      listed instead.
//
//  nsw6_satadj_kernel  one thread per listed cell: its Newton iteration on T
//                      (the saturation adjustment) and its final state.
//
// The only coupling between columns, the per-level max/min of the departure
// distance over a region (mod_vadv1d.cpp:316-353), is what separates the cell
// phase (the first two kernels) from the column phase.
#include <cfloat>
#include <cuda_runtime.h>

#include "nsw6_cell.cuh"
#include "nsw6_common.cuh"
#include "nsw6_fastmath.cuh"

namespace nsw6 {

// ------------------------------------------------------------------ kernel 1
template <class M>
__device__ __forceinline__ M make_math(const double* tab);
template <>
__device__ __forceinline__ FastMath make_math<FastMath>(const double* tab) {
  return FastMath(tab);
}
template <>
__device__ __forceinline__ LibMath make_math<LibMath>(const double*) {
  return LibMath{};
}
template <>
__device__ __forceinline__ FloatMath make_math<FloatMath>(const double*) {
  return FloatMath{};
}

// Cells of one CTA at most: the shared-memory keys and order take 3 B each.
constexpr int CELL_TILE_MAX = 4096;

// Fall speeds go from the cell kernel to the departure kernel in the 8-byte
// words of the departure distances' own rows (row t of tracer t); FP32 speeds
// as their bits.
__device__ __forceinline__ double vt_word(double v) { return v; }
__device__ __forceinline__ double vt_word(float v) { return __longlong_as_double((long long)__float_as_uint(v)); }
template <class R>
__device__ __forceinline__ R vt_value(double w) {
  if constexpr (sizeof(R) == sizeof(float)) return __uint_as_float((unsigned)__double_as_longlong(w));
  else return w;
}

// Counts v (< 64; 64: cells to leave out) into bucket[] and returns the cell's
// position in its bucket; one shared-memory atomic for each value that a warp
// holds, not one a cell.
__device__ __forceinline__ int bucket_add(int* bucket, int v) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(__activemask(), v);
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if ((int)lane == leader) base = atomicAdd(&bucket[v], __popc(peers));
  return __shfl_sync(peers, base, leader) + __popc(peers & ((1u << lane) - 1u));
}

// One CTA: `tile` consecutive interior cells of one region in [k][g] order, the
// cell physics and nothing that couples cells.  Bound by the FP64 pipe: what
// helps is to leave work out, so the FP64 tile's cells are grouped by their
// side of 0 C and by the hydrometeors they hold (a counting sort in shared
// memory), in Gray-code order, so that a warp that straddles two groups does
// the work of the larger one only.  A tile of many columns by few levels has
// larger groups than one of 32 columns by all levels (the layout before, with
// the departure distances in the same kernel).  The order only decides which
// thread computes which cell.  One 16900 x 42 region, FP64, with the departure
// kernel: 0.90 -> 0.67 ms; 48 columns, which had two CTAs here, 0.47 -> 0.29 ms
// for the whole step.  What is left out is branched around since: this kernel
// then took 0.45 -> 0.34 ms (6.1 M -> 3.7 M FP64 warp instructions; its FP64
// pipe is 60 % busy, next to it come waits for instructions).
//
// OPT: the kernel with the scheme switches: the switched branches of nsw6_cell
// and the CCN input.
template <class M, class R, bool OPT = false>
__global__ void __launch_bounds__(CELL_THREADS, sizeof(R) == 4 ? 3 : 2) nsw6_cell_kernel(Problem P, ConstsT<R> C, int tile) {
  constexpr bool kMixed = sizeof(R) == sizeof(float);
  const int ntr = OPT ? P.ntr : 3;          // sedimenting tracers of this call
  extern __shared__ double sm[];
  const int G = P.gall, kmin = P.kmin, kmax = P.kmax;
  const int l = blockIdx.y;
  const int first = blockIdx.x * tile;                 // of the region's interior cells
  const int n = min(tile, (kmax - kmin + 1) * G - first);
  const size_t KG = (size_t)P.kall * G;
  const size_t off = (size_t)l * KG + (size_t)kmin * G + first;          // the tile's first cell
  const size_t offq = (size_t)l * NQ * KG + (size_t)kmin * G + first;
  const size_t offv = (size_t)l * 2 * ntr * KG + (size_t)kmin * G + first;
  double* stab = sm;                                                     // [FM_TABLE_DOUBLES], FP64 only
  unsigned short* perm = reinterpret_cast<unsigned short*>(stab + FM_TABLE_DOUBLES);   // [tile], FP64 only
  unsigned char* key = reinterpret_cast<unsigned char*>(perm + tile);
  __shared__ int bucket[64];

  // the departure kernel's extrema and the column kernel's list start empty
  {
    const unsigned nkey = (unsigned)P.lall * 2 * ntr * P.kall;
    const unsigned nthread = gridDim.x * gridDim.y * blockDim.x;
    for (unsigned e = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; e < nkey; e += nthread) {
      P.zmax[e] = 0ull;
      P.zmin[e] = ~0ull;
      if (e == 0) P.satq[0] = 0u;
    }
  }
  if (!kMixed) {
    for (int c = threadIdx.x; c < FM_TABLE_DOUBLES; c += blockDim.x) stab[c] = P.fmtab[c];
    for (int c = threadIdx.x; c < 64; c += blockDim.x) bucket[c] = 0;
    __syncthreads();
#pragma unroll 1
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
      const double* rq = P.rhogq + offq + c;
      int kk = (lt_c(P.tem[off + c], TEM00) ? 32 : 0) | (gt_z(rq[(size_t)I_QS * KG]) ? 16 : 0) |
               (gt_z(rq[(size_t)I_QR * KG]) ? 8 : 0) | (gt_z(rq[(size_t)I_QG * KG]) ? 4 : 0) |
               (gt_z(rq[(size_t)I_QI * KG]) ? 2 : 0) | (gt_z(rq[(size_t)I_QC * KG]) ? 1 : 0);
      kk ^= kk >> 1;   // the key's place in Gray-code order
      kk ^= kk >> 2;
      kk ^= kk >> 4;
      key[c] = (unsigned char)kk;
      bucket_add(bucket, kk);
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // exclusive prefix sums of the 64 counts
      const int b0 = bucket[2 * threadIdx.x], b1 = bucket[2 * threadIdx.x + 1];
      int run = b0 + b1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, run, o);
        if ((int)threadIdx.x >= o) run += v;
      }
      bucket[2 * threadIdx.x] = run - b0 - b1;
      bucket[2 * threadIdx.x + 1] = run - b1;
    }
    __syncthreads();
#pragma unroll 1
    for (int c = threadIdx.x; c < n; c += blockDim.x) perm[bucket_add(bucket, key[c])] = (unsigned short)c;
    __syncthreads();
  }
  const M mth = make_math<M>(stab);
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += blockDim.x) {
    // FP64: the CTA's warps go through neighbouring groups together, so that
    // they run the same parts of the code (its 120 KB do not fit the
    // instruction caches)
    if (!kMixed) __syncthreads();
    const int j = j0 + threadIdx.x;
    if (j >= n) continue;
    const int c = kMixed ? j : perm[j];
    const size_t i = off + c;
    const size_t iq = offq + c;
    CellIn in;
    in.rhog = P.rhog[i];
    in.tem = P.tem[i];
    in.gsgam2 = P.gsgam2[i];
    in.q0 = P.q[iq];
#pragma unroll
    for (int n = 0; n < 6; ++n) in.rhogq[n] = P.rhogq[iq + (size_t)n * KG];
    in.unccn = (OPT && P.unccn) ? P.unccn[i] : 0.0;   // required only with the aerosol switch
    CellOut o;
    nsw6_cell<M, R, double, OPT>(C, mth, P.dt, P.rdt, in, o);
    P.rhog[i] = o.rhog;
    P.rhoge[i] = o.rhoge;
    P.tem[i] = o.tem;
#pragma unroll
    for (int n = 0; n < 6; ++n) P.rhogq[iq + (size_t)n * KG] = o.rhogq[n];
#pragma unroll
    for (int n = 1; n < 6; ++n) P.q[iq + (size_t)n * KG] = o.q[n];
    P.re_liquid[i] = o.rceff;
    P.re_cld[i] = o.rceff_cld;
    // fall speeds in the tracer order of the transport: QR, (QI,) QS, QG
    double* vt = P.zdis + offv + c;
    vt[0] = vt_word(R(o.Vtr));
    if (ntr == 4) vt[KG] = vt_word(R(o.Vti));
    vt[(size_t)(ntr - 2) * KG] = vt_word(R(o.Vts));
    vt[(size_t)(ntr - 1) * KG] = vt_word(R(o.Vtg));
    const int top = first + c - (kmax - kmin) * G;
    if (top >= 0) {
      // The reference writes the cloud-top scalars from every level in parallel
      // (mod_mp_nsw6.cpp:1579-1592); the sequential order, in which the top
      // interior level is written last, is used.  TagUpdateCLD, :710-726.
      const size_t ic = (size_t)l * G + top;
      P.rctop[ic] = o.rctop;
      P.tctop[ic] = o.tctop;
      const double sw = (0.5 + copysign(0.5, o.tctop - TEM00));
      P.rwtop[ic] = (sw)*o.rctop + (1.0 - sw) * UNDEF;
    }
  }
}

// ------------------------------------------------------- departure distances
// 0.5 x: the exponent one lower, where that is all there is to it
NSW6_SLOW double soft_slow_half(double x) { return 0.5 * x; }
__device__ __forceinline__ float half_of(float x) { return 0.5f * x; }
__device__ __forceinline__ double half_of(double x) {
  const long long b = __double_as_longlong(x);
  if ((unsigned)(((b >> 52) & 0x7FF) - 2) < 2045u) return __longlong_as_double(b - (1ll << 52));
  return fp_is_zero(x) ? x : soft_slow_half(x);
}
// the largest (smallest) key of a warp's lanes
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
  return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) { return ~warp_max(~v); }

// Departure distances (vadv1d_prep, mod_vadv1d.cpp:262-302) of one tracer on
// full and half levels for DEP_TG columns, and their per-level extrema over the
// region (order-preserving keys, exact atomics, so the order does not matter).
// Row t of zdis holds the tracer's fall speeds on entry, the full-level
// distances on return, row ntr + t the half-level ones.  One CTA reads all of
// its columns' speeds before it writes.  Bound by the FP64 pipe (82 % busy): a
// half-level velocity is the mean of two full-level ones, formed once, the
// halvings are integer operations, a warp walks consecutive levels and forms
// their differences once, and levels without the tracer are branched around.
// One 16900 x 42 region, FP64: 0.165 -> 0.118 ms (2.5 M -> 1.75 M FP64 warp
// instructions), with the extrema's keys by words 0.083 (1.04 M).
constexpr int DEP_TG = 32;
constexpr int DEP_THREADS = 256;

template <class R>
__host__ __device__ constexpr size_t departure_smem_bytes(int K) {
  return (size_t)K * sizeof(R) * (3 * DEP_TG + 8);
}

template <class R>
__global__ void __launch_bounds__(DEP_THREADS) nsw6_departure_kernel(Problem P) {
  extern __shared__ double sm[];
  constexpr bool kMixed = sizeof(R) == sizeof(float);
  const int G = P.gall, K = P.kall, kmin = P.kmin, kmax = P.kmax, ntr = P.ntr;
  const int g0 = blockIdx.x * DEP_TG, t = blockIdx.y, l = blockIdx.z;
  const size_t KG = (size_t)K * G;
  R* vt = reinterpret_cast<R*>(sm);     // [K][DEP_TG] fall speeds, zero outside the interior
  R* wf = vt + K * DEP_TG;              // [K][DEP_TG] velocities on the full levels' interfaces
  R* wh = wf + K * DEP_TG;              // [K][DEP_TG] and on the half levels'
  // 1 / dz, 1 / (dz- + dz) and, FP32, twice that or, FP64, twice that over dz and over dz-, of full and half levels
  R* grid = wh + K * DEP_TG;
  double* z0 = P.zdis + ((size_t)l * 2 * ntr + t) * KG;
  double* z1 = z0 + (size_t)ntr * KG;

  for (int c = threadIdx.x; c < 2 * K; c += blockDim.x) {
    const int half = c / K, k = c % K;
    const double* rdz = P.grid + (half ? GF_RDGZH : GF_RDGZ) * K;
    const double* rdzs = P.grid + (half ? GF_RDZSH : GF_RDZS) * K;
    R* row = grid + 4 * half * K + k;
    row[0] = R(rdz[k]);
    row[K] = R(rdzs[k]);
    const R s2 = R(2.0) * R(rdzs[k]);
    row[2 * K] = kMixed ? s2 : s2 * R(rdz[k]);
    row[3 * K] = (kMixed || k == 0) ? R(0.0) : s2 * R(rdz[k - 1]);
  }
  const int gx = threadIdx.x % DEP_TG, g = g0 + gx, kw = threadIdx.x / DEP_TG, nw = blockDim.x / DEP_TG;
#pragma unroll 4
  for (int k = kw; k < K; k += nw)
    vt[k * DEP_TG + gx] = (k >= kmin && k <= kmax && g < G) ? vt_value<R>(z0[(size_t)k * G + g]) : R(0.0);
  __syncthreads();
  // wh of vadv1d_prep from the speeds (full levels: mkmin = kmin)
#pragma unroll 1
  for (int k = kw; k < K; k += nw) {
    const int c = k * DEP_TG + gx;
    wf[c] = k > kmin && k <= kmax ? half_of(vt[c - DEP_TG] + vt[c]) : k == kmax + 1 ? vt[c - DEP_TG] : vt[c];
  }
  __syncthreads();
  // half levels (mkmin = kmin + 1): the speeds there, Vtermh (mod_precip_transport.cpp:847-861), are the
  // means just formed on [kmin + 1, kmax - 1] and zero elsewhere
  auto vh = [&](int k) { return k > kmin && k < kmax ? wf[k * DEP_TG + gx] : R(0.0); };
#pragma unroll 1
  for (int k = kw; k < K; k += nw)
    wh[k * DEP_TG + gx] = k > kmin + 1 && k <= kmax ? half_of(vh(k - 1) + vh(k)) : k == kmax + 1 ? vh(kmax) : vh(k);
  __syncthreads();

  const R dt = R(P.dt), hdt2 = R(P.hdt2), sdt3 = R(P.sdt3);
  // a warp: consecutive levels of one of the two rows, so that a difference of
  // two levels is formed once
  const int share = (2 * K + nw - 1) / nw;
  const bool valid = g < G;
  R w0 = R(0.0), w1 = R(0.0), dn = R(0.0);   // w at k and k + 1, w(k) - w(k - 1)
  int at = -1;                               // the row those are of
#pragma unroll 1
  for (int row = kw * share; row < min((kw + 1) * share, 2 * K); ++row) {
    const int half = row >= K ? 1 : 0, k = row - half * K, mkmin = kmin + half;
    if (k < mkmin || k > kmax) continue;
    const R* w = (half ? wh : wf) + gx;
    const R* gr = grid + 4 * half * K;
    double z;
    if constexpr (kMixed) {
      auto wp = [&](int j) { return w[j * DEP_TG]; };
      z = soft_f2d(vadv_zdis_f<R>(wp, gr, gr + K, [&](int j) { return gr[2 * K + j]; }, k, mkmin, dt, hdt2, sdt3));
    } else {
      const R wm = k > mkmin ? w[(k - 1) * DEP_TG] : R(0.0);
      if (at == row - 1) {
        w0 = w1;
      } else {
        w0 = w[k * DEP_TG];
        dn = w0 - wm;
      }
      w1 = w[(k + 1) * DEP_TG];
      at = row;
      z = w0;
      if (__any_sync(0xffffffffu, !(fp_is_zero(wm) && fp_is_zero(w0) && fp_is_zero(w1)))) {
        soft_branch();   // (levels without the tracer are branched around)
        const R up = w1 - w0;
        if (k == mkmin) {
          soft_branch();
          z = fmaR(-hdt2 * w0, up * gr[k], dt * w0);
        } else {
          soft_branch();
          z = vadv_zdis_d<R, R>(w0, up, dn, w1 - wm, gr[K + k], gr[2 * K + k], gr[3 * K + k], dt, hdt2, sdt3);
        }
        dn = up;
      } else {
        dn = R(0.0);
      }
    }
    if (valid) (half ? z1 : z0)[(size_t)k * G + g] = z;
    // NaN never wins the reference's comparisons, so it is left out
    const bool use = valid && !is_nan_bits(z);
    const unsigned long long kmx = warp_max(use ? order_key(z) : 0ull);
    const unsigned long long kmn = warp_min(use ? order_key(z) : ~0ull);
    if (gx == 0) {
      const size_t e = ((size_t)l * 2 * ntr + half * ntr + t) * K + k;
      if (kmx != 0ull) atomicMax(&P.zmax[e], kmx);
      if (kmn != ~0ull) atomicMin(&P.zmin[e], kmn);
    }
  }
}

// ------------------------------------------------------------------ math check
// Evaluates the step's table-driven transcendentals on n inputs:
// fn 0 exp(x), 1 log(x), 2 pow(x, y).
__global__ void nsw6_math_kernel(int fn, const double* x, const double* y, double* out, int n, const double* fmtab) {
  __shared__ double tab[FM_TABLE_DOUBLES];
  for (int c = threadIdx.x; c < FM_TABLE_DOUBLES; c += blockDim.x) tab[c] = fmtab[c];
  __syncthreads();
  const FastMath m = make_math<FastMath>(tab);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = x[i];
    out[i] = fn == 0 ? m.exp(v) : fn == 1 ? m.log(v) : m.pow(v, y[i]);
  }
}

cudaError_t launch_math(int fn, const double* x, const double* y, double* out, int n, const double* fmtab,
                        cudaStream_t stream) {
  const int blocks = n <= 0 ? 1 : (n + 255) / 256 > 1024 ? 1024 : (n + 255) / 256;
  nsw6_math_kernel<<<blocks, 256, 0, stream>>>(fn, x, y, out, n, fmtab);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ launchers
// Tile and threads of the cell kernel for `cells` interior cells of each of
// lall regions.  Two CTAs of 256 threads fit an SM (128 registers); the tiles
// share the cells out evenly over whole waves of them, so that no last wave is
// nearly empty, and a call too small for that gets a cell a thread on as many
// SMs as it has warps (a lone warp issues an FP64 instruction every 64 cycles,
// four warps of an SM one every 16 to 19: fewer warps an SM cost nothing).
struct CellShape {
  int tile, threads, blocks;
};
static CellShape cell_shape(int cells, int lall, bool mixed) {
  // CTAs the chip holds: in mixed precision, 80 registers a thread without
  // spills, three an SM (ten regions 4.46 -> 4.41 ms a step; FP64 at 80 spills)
  const int slots = (mixed ? 3 : 2) * 152;
  CellShape s;
  const long long total = (long long)cells * lall;
  if (total <= (long long)slots * CELL_THREADS) {
    const long long warps = (total + 31) / 32;
    s.threads = (int)((warps + slots - 1) / slots) * 32;
    s.tile = s.threads;
  } else {
    // whole waves of `slots` CTAs, each region's cells shared out alike
    const int tile_goal = 2304;
    const long long waves = (total + (long long)slots * tile_goal - 1) / ((long long)slots * tile_goal);
    long long per = (waves * slots) / lall;   // CTAs of a region
    if (per < 1) per = 1;
    int tile = (int)((cells + per - 1) / per);
    tile = (tile + 31) / 32 * 32;
    if (tile > CELL_TILE_MAX) tile = CELL_TILE_MAX;
    const int passes = (tile + CELL_THREADS - 1) / CELL_THREADS;
    s.threads = ((tile + passes - 1) / passes + 31) / 32 * 32;
    s.tile = tile;
  }
  s.blocks = (cells + s.tile - 1) / s.tile;
  return s;
}
static size_t cell_smem_bytes(const CellShape& s, bool mixed) {
  return mixed ? 0 : sizeof(double) * FM_TABLE_DOUBLES + 3 * (size_t)s.tile;
}

cudaError_t launch_prepare();

// The cell phase: the cell kernel and the departure distances.
static cudaError_t launch_cells(const Problem& P, const Consts& C, cudaStream_t stream) {
  const CellShape s = cell_shape((P.kmax - P.kmin + 1) * P.gall, P.lall, P.mixed != 0);
  const size_t sm = cell_smem_bytes(s, P.mixed != 0);
  const dim3 g1(s.blocks, P.lall);
  const int nt = s.threads;
  if (P.opt && P.mixed) nsw6_cell_kernel<FloatMath, float, true><<<g1, nt, sm, stream>>>(P, consts_to_float(C), s.tile);
  else if (P.opt) nsw6_cell_kernel<FastMath, double, true><<<g1, nt, sm, stream>>>(P, C, s.tile);
  else if (P.mixed) nsw6_cell_kernel<FloatMath, float><<<g1, nt, sm, stream>>>(P, consts_to_float(C), s.tile);
  else if (P.math_lib) nsw6_cell_kernel<LibMath, double><<<g1, nt, sm, stream>>>(P, C, s.tile);
  else nsw6_cell_kernel<FastMath, double><<<g1, nt, sm, stream>>>(P, C, s.tile);
  const dim3 g2((P.gall + DEP_TG - 1) / DEP_TG, P.ntr, P.lall);
  if (P.mixed) nsw6_departure_kernel<float><<<g2, DEP_THREADS, departure_smem_bytes<float>(P.kall), stream>>>(P);
  else nsw6_departure_kernel<double><<<g2, DEP_THREADS, departure_smem_bytes<double>(P.kall), stream>>>(P);
  return cudaGetLastError();
}

// The cell phase alone (FP64): used on a copy of a state to obtain the
// region extrema of the departure distances for the derivative kernels.
cudaError_t launch_cell_only(const Problem& P, const Consts& C, cudaStream_t stream) {
  const cudaError_t e = launch_prepare();
  if (e != cudaSuccess) return e;
  Problem F = P;
  F.mixed = F.math_lib = 0;
  return launch_cells(F, C, stream);
}

// The column phase's translation units (nsw6_column_*.cu).
cudaError_t prepare_column_fp64(int optin);
cudaError_t launch_column_fp64(const Problem& P, const Consts& C, cudaStream_t stream);
cudaError_t prepare_column_fp64_switches(int optin);
cudaError_t launch_column_fp64_switches(const Problem& P, const Consts& C, cudaStream_t stream);
cudaError_t prepare_column_mixed(int optin);
cudaError_t launch_column_mixed(const Problem& P, const Consts& C, cudaStream_t stream);
cudaError_t prepare_column_mixed_switches(int optin);
cudaError_t launch_column_mixed_switches(const Problem& P, const Consts& C, cudaStream_t stream);

// Opt-in shared-memory limits of the step kernels (once per process; before
// any stream capture of a step).
cudaError_t launch_prepare() {
  static cudaError_t done = cudaErrorNotReady;
  if (done == cudaErrorNotReady) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const cudaError_t r[] = {
        e,
        cudaFuncSetAttribute(nsw6_departure_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin),
        cudaFuncSetAttribute(nsw6_departure_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin),
        prepare_column_fp64(optin), prepare_column_fp64_switches(optin), prepare_column_mixed(optin),
        prepare_column_mixed_switches(optin)};
    done = cudaSuccess;
    for (cudaError_t x : r)
      if (x != cudaSuccess) done = x;
  }
  return done;
}

// before_column (may be null): an event the column kernel waits for (inputs
// that only it reads may still be arriving while the cell kernel runs).
cudaError_t launch_step(const Problem& P, const Consts& C, cudaStream_t stream, cudaEvent_t* ev,
                        cudaEvent_t before_column) {
  cudaError_t e = launch_prepare();
  if (e != cudaSuccess) return e;
  const bool opt = P.opt != 0;
  if (ev) cudaEventRecord(ev[0], stream);
  if ((e = launch_cells(P, C, stream)) != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[1], stream);
  if (before_column && (e = cudaStreamWaitEvent(stream, before_column, 0)) != cudaSuccess) return e;
  if (opt && P.mixed) e = launch_column_mixed_switches(P, C, stream);
  else if (opt) e = launch_column_fp64_switches(P, C, stream);
  else if (P.mixed) e = launch_column_mixed(P, C, stream);
  else e = launch_column_fp64(P, C, stream);
  if (e != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[2], stream);
  return cudaGetLastError();
}

}  // namespace nsw6
