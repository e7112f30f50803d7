// phx_flux.cu -- fluid::CalculateFluxes (fluid.cpp:659-773) as fused
// reconstruction + Riemann kernels, one launch per direction.
//
// The reference reconstructs every variable into ql/qr arrays (K1) and then
// solves one Riemann problem per face (K2).  Here a thread produces and
// consumes each face's two states:
//   X1: a CTA stages one to four (k, j) pencils' primitive rows in shared
//       memory with one tiled TMA copy per pencil
//       (cp.async.bulk.tensor through a 5-D tensor map of the primitive
//       array: i split in S rows of n1t/S, j, k, variable), completing on an
//       mbarrier (1-D cp.async.bulk per row, or plain loads, where the block
//       shape does not admit the map); lanes reconstruct consecutive cells and
//       the left state of face i (the upper-face value of cell i-1) moves to
//       lane i with __shfl_up_sync.
//   X2, X3: a thread sweeps a segment of faces along the direction, one
//       variable's stencil at a time; consecutive lanes are consecutive i
//       (coalesced), and the cells a stencil shares with its neighbours come
//       from L1.
// The face states pass from the reconstruction to the Riemann solver through
// shared memory (FaceStates).
// Faces computed, per direction d: along d [s, e+1]; transverse active
// directions [s-1, e+1].  These are all the faces FluxDivergence, FluxCT and
// EstimateTimestep read.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdlib>
#include <cstring>
#include <mutex>

#include "phx_kernels.cuh"
#include "phx_bulk.cuh"

namespace phx {

constexpr unsigned FULL = 0xffffffffu;

// Riemann solve + store for one face (riemann.hpp:256-301).
// col: the face's floor_point when the caller holds it (a sweep across X1
// faces' constant X1 when the floors depend on X1 alone), else null.
template <bool MINK, int DIR>
__device__ __forceinline__ void face_flux(const Par &p, const BView &b, int k, int j, int i,
                                          const double ql[PHX_NRECON], const double qr[PHX_NRECON],
                                          const FloorPt *col = nullptr) {
  Face f;
  if constexpr (!MINK) {
    load_pt(b, DIR == 0 ? 1 : (DIR == 1 ? 2 : 0), j, i, f.g);
    f.gdet = f.g.alpha * f.g.detgam;
    f.gammadet = f.g.detgam;
    f.gdd = f.g.gamcon[DIR][DIR];
  }
  const double2 *flr = DIR == 0 ? floor_face1(b, i) : nullptr;
  if (col) {
    f.fl = *col;
  } else if (flr) {
    f.fl = floor_load(flr);
  } else {
    f.fl = floor_point(p, DIR == 0 ? b.Xf(0, i) : b.Xc(0, i), DIR == 1 ? b.Xf(1, j) : b.Xc(1, j),
                       DIR == 2 ? b.Xf(2, k) : b.Xc(2, k));
  }
  const double gdet = MINK ? 1.0 : f.gdet;
  const double gammadet = MINK ? 1.0 : f.gammadet;
  const long long id = b.idx(k, j, i);
  double *fx = b.flux + (long long)DIR * PHX_NCONS * b.vs + id;
  const int ncons = p.mhd ? PHX_NCONS : 5;
  double sig;
#ifndef PHX_EXACT
  // both solvers as F = kl F_l + kr F_r + kc (U_r - U_l), with the states'
  // F = U vtil + G
  FluxState l, r;
  flux_state<MINK, DIR>(p, f, ql, l);
  flux_state<MINK, DIR>(p, f, qr, r);
  double kl, kr, kc;
  if (p.riemann == PHX_RIEMANN_LLF) {
    sig = max_num(max_num(-l.vm, l.vp), max_num(-r.vm, r.vp));
    kl = kr = 0.5 * gdet;
    kc = -0.5 * sig * gammadet;
  } else {
    const double cl = min_num(min_num(l.vm, r.vm), 0.0);
    const double cr = max_num(max_num(l.vp, r.vp), 0.0);
    const double dc = cr - cl;
    const int e = dexp(dc);
    const double idc = (e >= 16 && e <= 2030) ? rcp_nr(dc) : ratio_p(1.0, dc);
    const double gi = gdet * idc;
    kl = cr * gi;
    kr = -cl * gi;
    kc = cr * cl * (MINK ? idc : gammadet * idc);
    sig = max_num(-cl, cr);
  }
  // U_r - U_l formed first: equal states then carry no rounding of c U
  const double al = kl * l.vtil, ar = kr * r.vtil;
#pragma unroll
  for (int m = 0; m < PHX_NCONS; m++) {
    if (m >= ncons) continue;
    double F = kc * (r.U[m] - l.U[m]);
    if (m != PHX_CB + DIR) {  // B^d v^d - B^d v^d is 0 in both states
      F = fma(al, l.U[m], fma(ar, r.U[m], F));
      if (m != PHX_CRHO) F = fma(kl, l.G[m], fma(kr, r.G[m], F));
    }
    fx[m * b.vs] = F;
  }
#else
  const double gam_max = p.g0, sie_max = p.smax0;
  double Ul[PHX_NCONS], Fl[PHX_NCONS], Ur[PHX_NCONS], Fr[PHX_NCONS];
  double vml, vpl, vmr, vpr;
  prim_to_flux<MINK, DIR>(p, f, ql, vml, vpl, Ul, Fl, sie_max, gam_max);
  prim_to_flux<MINK, DIR>(p, f, qr, vmr, vpr, Ur, Fr, sie_max, gam_max);
  if (p.riemann == PHX_RIEMANN_LLF) {
    const double cmax = rmax(rmax(-vml, vpl), rmax(-vmr, vpr));
#pragma unroll
    for (int m = 0; m < PHX_NCONS; m++)
      if (m < ncons) fx[m * b.vs] = 0.5 * ((Fl[m] + Fr[m]) * gdet - cmax * ((Ur[m] - Ul[m]) * gammadet));
    sig = cmax;
  } else {
    const double cl = rmin(rmin(vml, vmr), 0.0);
    const double cr = rmax(rmax(vpl, vpr), 0.0);
    const double crcl = cr * cl;
    const double inv_cr_cl = ratio(1.0, cr - cl);
#pragma unroll
    for (int m = 0; m < PHX_NCONS; m++)
      if (m < ncons)
        fx[m * b.vs] = ((cr * Fl[m] - cl * Fr[m]) * gdet + crcl * (Ur[m] - Ul[m]) * gammadet) * inv_cr_cl;
    sig = rmax(-cl, cr);
  }
#endif
  b.face_sig[(long long)DIR * b.vs + id] = sig;
}

// Reconstructed states between the loop over the variables and the Riemann
// solve: one double per thread, variable and slot in shared memory (thread
// private, no barrier).  With the loop rolled the reconstruction's code is
// there once -- unrolled over nine variables it no longer fits the
// instruction cache beside the Riemann solver -- and a thread holds one
// variable's stencil in registers instead of all of them, which leaves room
// for the resident warps that hide the integer instructions' latency.
constexpr int FLUX_THREADS = 128;
// PLM and constant reconstruction are short enough to unroll (their loads
// then overlap).  256^3 WENO5-Z, three directions: unrolled with the stencils in
// registers (228 registers, 12% of the warps resident) 69.6 ms, rolled 56.6 ms.
template <int RECON>
constexpr int flux_unroll() {
  return RECON == PHX_RECON_WENO5Z || RECON == PHX_RECON_MP5 ? 1 : kReconLoad;
}
struct FaceStates {
  double q[kReconLoad][FLUX_THREADS];
  __device__ __forceinline__ void load(double out[PHX_NRECON]) const {
#pragma unroll
    for (int v = 0; v < kReconLoad; v++) out[v] = q[v][threadIdx.x];
  }
};

// Resident CTAs per SM the register allocation is bounded for.
#ifdef PHX_EXACT
constexpr int flux_minb(bool) { return 1; }
#else
constexpr int flux_minb(bool mink) { return mink ? 4 : 3; }
#endif

// ------------------------------------------------------------------ X1
constexpr int X1_WARPS = FLUX_THREADS / 32;  // warps per CTA
constexpr int X1_PENCILS = 4;                // at most this many (k, j) pencils staged per CTA

// A CTA stages np pencils (kReconLoad primitive rows each) in shared memory
// with TMA copies completing on one mbarrier.  Its warps then walk the pencils'
// cells as one flattened list [pencil][cell is-1 .. ie+1] in chunks of 32
// cells that overlap by one: lane L reconstructs its cell, takes the
// upper-face state of the cell on its left from lane L-1 (__shfl_up_sync) and
// solves the Riemann problem of its lower face; lane 0 only supplies its
// state to lane 1 (its own face belongs to the previous chunk's lane 31).

// X1 face ranges of a block: pencils (k, j) over k in [ks-dk, ke+dk],
// j in [js-dj, je+dj]; pencil pen is (klo + pen / nj, jlo + pen % nj).
struct X1Range {
  int jlo, nj, klo, npencil;
};
__host__ __device__ __forceinline__ X1Range x1_range(const BView &b) {
  const int dk = b.ndim == 3 ? 1 : 0, dj = b.ndim > 1 ? 1 : 0;
  const int js = dj ? b.ng : 0, je = dj ? b.ng + b.nx2 - 1 : 0;
  const int ks = dk ? b.ng : 0, ke = dk ? b.ng + b.nx3 - 1 : 0;
  X1Range r;
  r.jlo = js - dj;
  r.nj = je - js + 1 + 2 * dj;
  r.klo = ks - dk;
  r.npencil = r.nj * (ke - ks + 1 + 2 * dk);
  return r;
}
__host__ __device__ __forceinline__ bool x1_tma_ok(const BView &b) {
  return (b.n1t % 2 == 0) && (b.vs % 2 == 0) && ((reinterpret_cast<uintptr_t>(b.prim) & 15) == 0);
}
// Staging modes of the X1 kernels.
enum X1Mode { X1_LOADS = 0, X1_BULK = 1, X1_TENSOR = 2 };

// Shared-memory doubles per staged pencil: its kReconLoad rows of n1t,
// rounded up to 128 bytes (the alignment of a tiled TMA destination).
__host__ __device__ __forceinline__ long long x1_pencil_stride(const BView &b) {
  return ((long long)kReconLoad * b.n1t + 15) / 16 * 16;
}

// One tiled TMA copy: box {n1t/S, S, 1, 1, kReconLoad} of the 5-D map at
// (0, 0, j, k, 0) -> a pencil's kReconLoad rows, contiguous in shared memory.
__device__ __forceinline__ void tensor_g2s_5d(void *dst, const CUtensorMap *map, int j, int k, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5, %6}], [%7];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(0), "r"(j), "r"(k), "r"(0), "r"(smem_u32(bar))
      : "memory");
}

// Stage pencils p0 .. p0+np-1 into rows (pencil pp at rows + pp * pencil
// stride; mbarrier phase parity `phase` for the TMA modes).  Returns false,
// with ERR_TIMEOUT set, when the bounded wait gave up; every thread returns
// the same value.
__device__ __forceinline__ bool x1_stage(const BView &b, const X1Range &xr, int p0, int np, int mode,
                                         const CUtensorMap *map, double *rows, uint64_t *bar, unsigned phase,
                                         unsigned int *err) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n1t = b.n1t;
  const long long pst = x1_pencil_stride(b);
  if (mode == X1_TENSOR && (smem_u32(rows) & 127u) != 0) mode = X1_BULK;  // tiled TMA wants 128-byte rows
  if (mode == X1_TENSOR) {
    if (threadIdx.x == 0) {
      mbar_expect_tx(bar, (unsigned)(n1t * sizeof(double)) * kReconLoad * np);
      for (int pp = 0; pp < np; pp++) {
        const int pen = p0 + pp;
        tensor_g2s_5d(rows + pp * pst, map, xr.jlo + pen % xr.nj, xr.klo + pen / xr.nj, bar);
      }
    }
    return mbar_wait_block(bar, phase, MBAR_SPIN_LIMIT, err);
  }
  if (mode == X1_BULK) {
    const unsigned bytes = (unsigned)(n1t * sizeof(double));
    if (threadIdx.x == 0) mbar_expect_tx(bar, bytes * kReconLoad * np);
    __syncthreads();
    // one bulk copy per (pencil, variable) row; a CTA may stage more rows
    // than it has threads
    for (int r = threadIdx.x; r < np * kReconLoad; r += blockDim.x) {
      const int pp = r / kReconLoad, v = r % kReconLoad;
      const int pen = p0 + pp;
      const long long base = b.idx(xr.klo + pen / xr.nj, xr.jlo + pen % xr.nj, 0);
      bulk_g2s(rows + pp * pst + (long long)v * n1t, b.prim + v * b.vs + base, bytes, bar);
    }
    return mbar_wait_block(bar, phase, MBAR_SPIN_LIMIT, err);
  }
  for (int r = warp; r < np * kReconLoad; r += (int)(blockDim.x >> 5)) {
    const int pp = r / kReconLoad, v = r % kReconLoad;
    const int pen = p0 + pp;
    const long long base = b.idx(xr.klo + pen / xr.nj, xr.jlo + pen % xr.nj, 0);
    for (int i = lane; i < n1t; i += 32) rows[pp * pst + (long long)v * n1t + i] = b.prim[v * b.vs + base + i];
  }
  __syncthreads();
  return true;
}

template <int RECON, bool MINK>
__device__ __forceinline__ void x1_compute(const Par &p, const BView &b, const X1Range &xr, int p0, int np,
                                           const double *rows, FaceStates *fs) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = (int)(blockDim.x >> 5);
  const int n1t = b.n1t;
  const int c0 = b.is() - 1;
  const int ncell = b.ie() + 1 - c0 + 1;  // cells is-1 .. ie+1 per pencil
  const int nslot = np * ncell;
  const int nchunk = (nslot - 1 + 30) / 31;
  for (int ch = warp; ch < nchunk; ch += nwarps) {
    const int slot = ch * 31 + lane;
    const bool have = slot < nslot;
    const int pp = have ? slot / ncell : 0;
    const int c = c0 + (have ? slot % ncell : 0);  // lanes past the end repeat the first cell
    const double *r = rows + pp * x1_pencil_stride(b) + c;
#pragma unroll(flux_unroll<RECON>())
    for (int v = 0; v < kReconLoad; v++, r += n1t) {
      double ql, qr;
      if constexpr (RECON == PHX_RECON_WENO5Z || RECON == PHX_RECON_MP5)
        recon<RECON>(r[-2], r[-1], r[0], r[1], r[2], ql, qr);
      else if constexpr (RECON == PHX_RECON_LINEAR)
        recon<RECON>(0.0, r[-1], r[0], r[1], 0.0, ql, qr);
      else
        recon<RECON>(0.0, 0.0, r[0], 0.0, 0.0, ql, qr);
      fs[0].q[v][threadIdx.x] = __shfl_up_sync(FULL, ql, 1);  // from cell c-1 (same pencil when c > is-1)
      fs[1].q[v][threadIdx.x] = qr;
    }
    if (have && lane > 0 && c > c0) {  // the face of cell c
      const int pen = p0 + pp;
      double left[PHX_NRECON], right[PHX_NRECON];
      fs[0].load(left);
      fs[1].load(right);
      recon_gamma1(p, left, right);
      face_flux<MINK, 0>(p, b, xr.klo + pen / xr.nj, xr.jlo + pen % xr.nj, c, left, right);
    }
    __syncwarp();
  }
}

template <int RECON, bool MINK>
__global__ void __launch_bounds__(FLUX_THREADS, flux_minb(MINK))
    k_flux_x1(Par p, BView b, int mode, int pencils, const __grid_constant__ CUtensorMap map, unsigned int *err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ FaceStates fs[2];
  __shared__ __align__(8) uint64_t bar;
  double *rows = reinterpret_cast<double *>(smem_raw);
  const X1Range xr = x1_range(b);
  const int p0 = blockIdx.x * pencils;
  const int np = min(pencils, xr.npencil - p0);
  if (mode != X1_LOADS && threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (!x1_stage(b, xr, p0, np, mode, &map, rows, &bar, 0u, err)) return;
  x1_compute<RECON, MINK>(p, b, xr, p0, np, rows, fs);
}

// Batched X1: a persistent CTA walks the work list; item = (block, first
// pencil, pencil count).  The mbarrier is reused with alternating phase.
// maps[b] / modes[b]: block b's tensor map and staging mode.
template <int RECON, bool MINK>
__global__ void __launch_bounds__(FLUX_THREADS, flux_minb(MINK))
    kb_flux_x1(Par p, const BView *views, const WorkItem *items, int nitems, const CUtensorMap *maps, const int *modes,
               unsigned int *err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ FaceStates fs[2];
  __shared__ __align__(8) uint64_t bar;
  double *rows = reinterpret_cast<double *>(smem_raw);
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  unsigned phase = 0;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const WorkItem w = items[it];
    const BView &b = views[w.block];
    const X1Range xr = x1_range(b);
    const int mode = modes[w.block];
    if (!x1_stage(b, xr, (int)w.first, (int)(w.last - w.first), mode, maps + w.block, rows, &bar, phase, err))
      return;
    if (mode != X1_LOADS) phase ^= 1u;
    x1_compute<RECON, MINK>(p, b, xr, (int)w.first, (int)(w.last - w.first), rows, fs);
    __syncthreads();  // rows are rewritten by the next item
  }
}

// ------------------------------------------------------ X1 tensor maps
// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;  // callers on several host threads look it up once
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

// The 5-D map of a block's reconstructed primitive planes: dimensions
// (n1t / S, S, n2t, n3t, kReconLoad) with byte strides (8, 8 n1t / S, 8 n1t,
// 8 n1t n2t, 8 vs), box (n1t / S, S, 1, 1, kReconLoad): one copy moves one
// (k, j) pencil's rows.  S is the smallest split with n1t / S <= 256 (the
// box limit) and n1t / S even (16-byte rows).  False (mode falls back) when
// no split fits, the strides are not multiples of 16 bytes, the base is not
// 16-byte aligned, or the encode is refused.
bool x1_encode_map(const BView &b, CUtensorMap *map) {
  if (!x1_tma_ok(b)) return false;
  int S = 0;
  for (int s = 1; s <= 8 && !S; s++)
    if (b.n1t % s == 0 && (b.n1t / s) % 2 == 0 && b.n1t / s <= 256) S = s;
  if (!S) return false;
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t h = (cuuint64_t)(b.n1t / S);
  const cuuint64_t dim[5] = {h, (cuuint64_t)S, (cuuint64_t)b.n2t, (cuuint64_t)b.n3t, (cuuint64_t)kReconLoad};
  const cuuint64_t stride[4] = {h * 8, (cuuint64_t)b.n1t * 8, (cuuint64_t)b.n1t * b.n2t * 8, (cuuint64_t)b.vs * 8};
  const cuuint32_t box[5] = {(cuuint32_t)h, (cuuint32_t)S, 1, 1, (cuuint32_t)kReconLoad};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, b.prim, dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// PHX_X1_STAGING=loads or =bulk in the environment forces a simpler mode
// (read at every call; the three modes give identical fluxes).
int x1_mode(const BView &b, CUtensorMap *map) {
  const char *force = getenv("PHX_X1_STAGING");
  if (force && strcmp(force, "loads") == 0) return X1_LOADS;
  if (!(force && strcmp(force, "bulk") == 0) && x1_encode_map(b, map)) return X1_TENSOR;
  return x1_tma_ok(b) ? X1_BULK : X1_LOADS;
}

// The failure path of the bounded waits above, driven on purpose: one CTA
// arms an mbarrier for 16 bytes and issues no copy, so the phase never
// completes and nothing is in flight; mbar_wait_block gives up after `limit`
// polls, sets ERR_TIMEOUT and the CTA returns.
__global__ void __launch_bounds__(128) k_wait_probe(long long limit, unsigned int *err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_expect_tx(&bar, 16u);
  mbar_wait_block(&bar, 0u, limit, err);
  __syncthreads();
  if (threadIdx.x == 0) mbar_inval(&bar);
}

void launch_wait_probe(long long limit, unsigned int *err, cudaStream_t s) {
  k_wait_probe<<<1, 128, 0, s>>>(limit, err);
}

// ------------------------------------------------------------- sweeps
// Thread = (transverse a, transverse c, segment).  DIR 1: a = i, c = k;
// DIR 2: a = i, c = j; DIR 0 (fallback for X1): a = j, c = k.
template <int RECON, bool MINK, int DIR>
__device__ __forceinline__ void sweep_at(const Par &p, const BView &b, int alo, int na, int clo, int nc, int f0,
                                         int nface, int seg, int nseg, long long t, FaceStates *fs) {
  const int a = alo + (int)(t % na);
  const long long q = t / na;
  const int s = (int)(q % nseg);
  const int cc = clo + (int)(q / nseg);
  const int fbeg = f0 + s * seg;
  const int fend = min(f0 + nface - 1, fbeg + seg - 1);
  if (fbeg > fend) return;
  // position along the sweep direction -> (k, j, i)
  auto kji = [&](int x, int &k, int &j, int &i) {
    if constexpr (DIR == 0) {
      i = x;
      j = a;
      k = cc;
    } else if constexpr (DIR == 1) {
      i = a;
      j = x;
      k = cc;
    } else {
      i = a;
      j = cc;
      k = x;
    }
  };
  long long stride;
  if constexpr (DIR == 0)
    stride = 1;
  else if constexpr (DIR == 1)
    stride = b.n1t;
  else
    stride = (long long)b.n1t * b.n2t;
  int k0, j0, i0;
  kji(fbeg - 1, k0, j0, i0);
  const double *pc = b.prim + b.idx(k0, j0, i0);  // cell fbeg-1
  const long long vs = b.vs;
  // X2 and X3 faces of this column share X1 (= the cell centre of column a)
  FloorPt col{};
  const bool use_col = DIR != 0 && floors_x1_only(p);
  if (use_col) col = b.flr ? floor_load(floor_cell(b, a)) : floor_point(p, b.Xc(0, a), 0.0, 0.0);
  // states: fs[0] and fs[1] the upper-face values of the previous and this
  // cell in turn, fs[2] the lower-face values of this cell
  int cur = 0;
  for (int x = fbeg - 1; x <= fend; x++, cur ^= 1, pc += stride) {
    const double *pn = pc;
#pragma unroll(flux_unroll<RECON>())
    for (int v = 0; v < kReconLoad; v++, pn += vs) {
      double ql, qr;
      if constexpr (RECON == PHX_RECON_WENO5Z || RECON == PHX_RECON_MP5)
        recon<RECON>(pn[-2 * stride], pn[-stride], pn[0], pn[stride], pn[2 * stride], ql, qr);
      else if constexpr (RECON == PHX_RECON_LINEAR)
        recon<RECON>(0.0, pn[-stride], pn[0], pn[stride], 0.0, ql, qr);
      else
        recon<RECON>(0.0, 0.0, pn[0], 0.0, 0.0, ql, qr);
      fs[cur].q[v][threadIdx.x] = ql;
      fs[2].q[v][threadIdx.x] = qr;
    }
    if (x >= fbeg) {
      int k, j, i;
      kji(x, k, j, i);
      double left[PHX_NRECON], right[PHX_NRECON];
      fs[cur ^ 1].load(left);
      fs[2].load(right);
      recon_gamma1(p, left, right);
      face_flux<MINK, DIR>(p, b, k, j, i, left, right, use_col ? &col : nullptr);
    }
  }
}

template <int RECON, bool MINK, int DIR>
__global__ void __launch_bounds__(FLUX_THREADS, flux_minb(MINK))
    k_flux_sweep(Par p, BView b, int alo, int na, int clo, int nc, int f0, int nface, int seg, int nseg) {
  __shared__ FaceStates fs[3];
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)na * nc * nseg) sweep_at<RECON, MINK, DIR>(p, b, alo, na, clo, nc, f0, nface, seg, nseg, t, fs);
}

// Sweep geometry of a block for DIR 1 (X2 faces: j in [js, je+1], i in
// [is-1, ie+1], k in [ks-dk, ke+dk]) and DIR 2 (X3 faces: k in [ks, ke+1],
// i in [is-1, ie+1], j in [js-1, je+1]); threads per block na * nc * nseg.
struct SweepRange {
  int alo, na, clo, nc, f0, nface, seg, nseg;
};
__host__ __device__ __forceinline__ SweepRange sweep_range(const BView &b, int dir, int seg_target) {
  const int dk = b.ndim == 3 ? 1 : 0;
  const int is = b.ng, ie = b.ng + b.nx1 - 1;
  const int js = b.ng, je = b.ng + b.nx2 - 1;
  const int ks = dk ? b.ng : 0, ke = dk ? b.ng + b.nx3 - 1 : 0;
  SweepRange r;
  r.alo = is - 1;
  r.na = ie - is + 3;
  if (dir == 1) {
    r.clo = ks - dk;
    r.nc = ke - ks + 1 + 2 * dk;
    r.f0 = js;
    r.nface = je - js + 2;
  } else {
    r.clo = js - 1;
    r.nc = je - js + 3;
    r.f0 = ks;
    r.nface = ke - ks + 2;
  }
  r.nseg = (r.nface + seg_target - 1) / seg_target;
  r.seg = (r.nface + r.nseg - 1) / r.nseg;
  return r;
}

template <int RECON, bool MINK, int DIR>
__global__ void __launch_bounds__(FLUX_THREADS, flux_minb(MINK))
    kb_flux_sweep(Par p, const BView *views, const WorkItem *items, int nitems, int seg_target) {
  __shared__ FaceStates fs[3];
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const WorkItem w = items[it];
    const long long t = w.first + threadIdx.x;
    if (t < w.last) {
      const BView &b = views[w.block];
      const SweepRange r = sweep_range(b, DIR, seg_target);
      sweep_at<RECON, MINK, DIR>(p, b, r.alo, r.na, r.clo, r.nc, r.f0, r.nface, r.seg, r.nseg, t, fs);
    }
  }
}

// Faces per thread of a sweep over columns of nface faces.  A segment of seg
// faces reconstructs seg + 1 cells, so long segments do less work, but a
// launch of few long segments leaves SMs idle.  The launch takes about
// (CTAs on the busiest SM) (seg (F + R) + R), F and R the FP64 work of a
// face and of a cell's reconstruction; below two CTAs an SM's FP64 pipe is
// not kept busy, so fewer count as two.  Against 32 faces throughout: 64^3 PLM
// 1.02 -> 0.64 ms per call (69 CTAs of 33 faces before), 97 x 66 x 35 FMKS
// WENO5-Z 1.80 -> 1.18 ms.
static int sweep_segment(int recon, long long columns, int nface) {
  const int nsm = sm_count();
  const double R = recon == PHX_RECON_WENO5Z ? 1.0 : recon == PHX_RECON_MP5 ? 1.5 : 0.3;
  int best = nface;
  double cost = 0.0;
  for (int seg = nface < 64 ? nface : 64; seg >= 2 || seg == nface; seg--) {
    const long long nseg = (nface + seg - 1) / seg;
    const long long ctas = (columns * nseg + FLUX_THREADS - 1) / FLUX_THREADS;
    const long long busiest = (ctas + nsm - 1) / nsm;
    const double c = (double)(busiest > 2 ? busiest : 2) * (seg * (1.0 + R) + R);
    if (cost == 0.0 || c < cost) {
      cost = c;
      best = seg;
    }
    if (seg == 1) break;
  }
  return best;
}

template <int RECON, bool MINK, int DIR>
static void launch_sweep(const Par &p, const BView &b, int alo, int na, int clo, int nc, int f0,
                         int nface, cudaStream_t s) {
  const int target = sweep_segment(RECON, (long long)na * nc, nface);
  const int nseg = (nface + target - 1) / target;
  const int seg = (nface + nseg - 1) / nseg;
  const long long total = (long long)na * nc * nseg;
  const int T = FLUX_THREADS;
  k_flux_sweep<RECON, MINK, DIR><<<(unsigned)((total + T - 1) / T), T, 0, s>>>(p, b, alo, na, clo, nc,
                                                                            f0, nface, seg, nseg);
}

template <int RECON, bool MINK>
static void launch_fluxes_t(const Par &p, const BView &b, unsigned int *err, cudaStream_t s) {
  const int ndim = b.ndim;
  const int dk = ndim == 3 ? 1 : 0, dj = ndim > 1 ? 1 : 0;
  const int is = b.ng, ie = b.ng + b.nx1 - 1;
  const int js = dj ? b.ng : 0, je = dj ? b.ng + b.nx2 - 1 : 0;
  const int ks = dk ? b.ng : 0, ke = dk ? b.ng + b.nx3 - 1 : 0;
  // X1 faces: i in [is, ie+1]; j in [js-dj, je+dj]; k in [ks-dk, ke+dk]
  {
    const X1Range xr = x1_range(b);
    const int jlo = xr.jlo, nj = xr.nj, klo = xr.klo, nk = xr.npencil / xr.nj;
    // as many pencils as leave room for the resident CTAs the registers allow
    // (228 KB per SM, 1 KB of it per CTA); 256^3, three directions: with four
    // pencils (two CTAs per SM) 57.6 ms, with two (four CTAs) 56.6 ms
    const size_t pst = (size_t)x1_pencil_stride(b) * sizeof(double);
    const size_t room = (228 * 1024) / flux_minb(MINK) - 1024 - 64 - 2 * sizeof(FaceStates);
    const int pencils = (int)(room < pst ? 1 : (room / pst < (size_t)X1_PENCILS ? room / pst : (size_t)X1_PENCILS));
    const size_t smem = pencils * pst;
    if (smem <= 200 * 1024) {
      auto kern = k_flux_x1<RECON, MINK>;
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      CUtensorMap map;
      memset(&map, 0, sizeof(map));
      const int mode = x1_mode(b, &map);
      kern<<<(xr.npencil + pencils - 1) / pencils, 32 * X1_WARPS, smem, s>>>(p, b, mode, pencils, map, err);
    } else {
      launch_sweep<RECON, MINK, 0>(p, b, jlo, nj, klo, nk, is, ie - is + 2, s);
    }
  }
  if (ndim >= 2) {  // X2 faces: j in [js, je+1]; i in [is-1, ie+1]; k in [ks-dk, ke+dk]
    launch_sweep<RECON, MINK, 1>(p, b, is - 1, ie - is + 3, ks - dk, ke - ks + 1 + 2 * dk, js,
                                 je - js + 2, s);
  }
  if (ndim >= 3) {  // X3 faces: k in [ks, ke+1]; i in [is-1, ie+1]; j in [js-1, je+1]
    launch_sweep<RECON, MINK, 2>(p, b, is - 1, ie - is + 3, js - 1, je - js + 3, ks, ke - ks + 2, s);
  }
}

void launch_fluxes_err(const Par &p, const BView &b, unsigned int *err, cudaStream_t s) {
  const bool mink = !b.fmks;
  switch (p.recon) {
  case PHX_RECON_WENO5Z:
    mink ? launch_fluxes_t<PHX_RECON_WENO5Z, true>(p, b, err, s)
         : launch_fluxes_t<PHX_RECON_WENO5Z, false>(p, b, err, s);
    break;
  case PHX_RECON_MP5:
    mink ? launch_fluxes_t<PHX_RECON_MP5, true>(p, b, err, s) : launch_fluxes_t<PHX_RECON_MP5, false>(p, b, err, s);
    break;
  case PHX_RECON_LINEAR:
    mink ? launch_fluxes_t<PHX_RECON_LINEAR, true>(p, b, err, s)
         : launch_fluxes_t<PHX_RECON_LINEAR, false>(p, b, err, s);
    break;
  default:
    mink ? launch_fluxes_t<PHX_RECON_CONSTANT, true>(p, b, err, s)
         : launch_fluxes_t<PHX_RECON_CONSTANT, false>(p, b, err, s);
    break;
  }
}

// ------------------------------------------------------------- batched
int x1_npencil(const BView &b) { return x1_range(b).npencil; }
bool x1_tma_ok_host(const BView &b) { return x1_tma_ok(b); }
long long x1_pencil_stride_host(const BView &b) { return x1_pencil_stride(b); }
long long sweep_threads(const BView &b, int dir, int seg_target) {
  const SweepRange r = sweep_range(b, dir, seg_target);
  return (long long)r.na * r.nc * r.nseg;
}

template <int RECON, bool MINK>
static void x1_prepare_t(size_t smem) {
  static size_t set = 0;  // largest dynamic shared memory already allowed
  if (smem > set) {
    cudaFuncSetAttribute(kb_flux_x1<RECON, MINK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    set = smem;
  }
}

template <int RECON, bool MINK>
static void x1_batched_t(const Par &p, const BView *views, const WorkItem *items, int nitems, int grid, size_t smem,
                         const CUtensorMap *maps, const int *modes, unsigned int *err, cudaStream_t s) {
  auto kern = kb_flux_x1<RECON, MINK>;
  x1_prepare_t<RECON, MINK>(smem);
  kern<<<persistent_grid(kern, 32 * X1_WARPS, smem, nitems, grid), 32 * X1_WARPS, smem, s>>>(
      p, views, items, nitems, maps, modes, err);
}

template <int RECON, bool MINK>
static void sweep_batched_t(const Par &p, int dir, const BView *views, const WorkItem *items, int nitems, int grid,
                            int seg_target, cudaStream_t s) {
  if (dir == 1)
    kb_flux_sweep<RECON, MINK, 1><<<persistent_grid(kb_flux_sweep<RECON, MINK, 1>, 128, 0, nitems, grid), 128, 0, s>>>(
        p, views, items, nitems, seg_target);
  else
    kb_flux_sweep<RECON, MINK, 2><<<persistent_grid(kb_flux_sweep<RECON, MINK, 2>, 128, 0, nitems, grid), 128, 0, s>>>(
        p, views, items, nitems, seg_target);
}

#define PHX_RECON_DISPATCH(FN, ...)                                                         \
  switch (p.recon) {                                                                        \
  case PHX_RECON_WENO5Z:                                                                    \
    mink ? FN<PHX_RECON_WENO5Z, true>(__VA_ARGS__) : FN<PHX_RECON_WENO5Z, false>(__VA_ARGS__); \
    break;                                                                                  \
  case PHX_RECON_MP5:                                                                       \
    mink ? FN<PHX_RECON_MP5, true>(__VA_ARGS__) : FN<PHX_RECON_MP5, false>(__VA_ARGS__);     \
    break;                                                                                  \
  case PHX_RECON_LINEAR:                                                                    \
    mink ? FN<PHX_RECON_LINEAR, true>(__VA_ARGS__) : FN<PHX_RECON_LINEAR, false>(__VA_ARGS__); \
    break;                                                                                  \
  default:                                                                                  \
    mink ? FN<PHX_RECON_CONSTANT, true>(__VA_ARGS__) : FN<PHX_RECON_CONSTANT, false>(__VA_ARGS__); \
    break;                                                                                  \
  }

void launch_flux_x1_batched(const Par &p, bool mink, const BView *views, const WorkItem *items, int nitems, int grid,
                            size_t smem, const CUtensorMap *maps, const int *modes, unsigned int *err,
                            cudaStream_t s) {
  if (nitems <= 0) return;
  PHX_RECON_DISPATCH(x1_batched_t, p, views, items, nitems, grid, smem, maps, modes, err, s)
}

void prepare_flux_x1_batched(const Par &p, bool mink, size_t smem) {
  PHX_RECON_DISPATCH(x1_prepare_t, smem)
}

void launch_flux_sweep_batched(const Par &p, bool mink, int dir, const BView *views, const WorkItem *items,
                               int nitems, int grid, int seg_target, cudaStream_t s) {
  if (nitems <= 0) return;
  PHX_RECON_DISPATCH(sweep_batched_t, p, dir, views, items, nitems, grid, seg_target, s)
}

}  // namespace phx
