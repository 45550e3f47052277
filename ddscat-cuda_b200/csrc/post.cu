// EVALQ and far-field (SCAT) kernels (sm_100a).
//
// EVALQ restates ddscat_cuda_unified/cuda/ddscat_matvec_cuda.cu:770-783 and
// :939-950: q = (CXADIA + i (2/3) k^3) P + CXAOFF block terms, then FP64
// products P^H q and E^H P.
//
// The far-field sums S_d = sum_j P_j exp(-i k_d . r_j), r_j = ((i+1)+x0)*dx
// (cu:793-822), use a separable phase: exp(-i k.r) = ex_d[ix] * ey_d[iy] *
// ez_d[iz], three 1-D tables per direction built in FP64.  The x rows are
// contracted first, as a register-tiled complex matrix product (k_ff_rows);
// partial sums are combined in a fixed order (deterministic).
#include <algorithm>
#include <vector>
#include "solvers.h"

namespace ddb {

template <typename C>
__global__ void k_evalq_q(const C* p, C* q, const C* ad, const C* ao, const int* occ, int nat, int nat0, int a_full,
                          double rabs_im) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nat0) return;
  const size_t jf = a_full ? (size_t)occ[j] : (size_t)j;
  const size_t st = a_full ? (size_t)nat : (size_t)nat0;
  const C p1 = p[j], p2 = p[j + nat0], p3 = p[j + 2 * (size_t)nat0];
  C d1 = ad[jf], d2 = ad[jf + st], d3 = ad[jf + 2 * st];
  const float ri = (float)rabs_im;  // the reference stores i*(2/3)k^3 as a float
  d1.y += ri; d2.y += ri; d3.y += ri;
  C q1 = cmul(d1, p1), q2 = cmul(d2, p2), q3 = cmul(d3, p3);
  if (ao) {
    const C a23 = ao[jf], a31 = ao[jf + st], a12 = ao[jf + 2 * st];
    q1 = cadd(q1, cadd(cmul(a31, p3), cmul(a12, p2)));
    q2 = cadd(q2, cadd(cmul(a12, p1), cmul(a23, p3)));
    q3 = cadd(q3, cadd(cmul(a23, p2), cmul(a31, p1)));
  }
  q[j] = q1;
  q[j + nat0] = q2;
  q[j + 2 * (size_t)nat0] = q3;
}

template <typename T>
int evalq_compute(Engine<T>& eng, VecOps<T>& ops, const cplx<T>* e, const cplx<T>* p, const cplx<T>* adia,
                  const cplx<T>* aoff, int a_full, cplx<T>* qbuf, double ak3, double2* zabs, double2* zep) {
  const int nat0 = eng.g.nat0;
  k_evalq_q<<<(unsigned)ceil_div(nat0, 256), 256, 0, ops.stream>>>(p, qbuf, adia, aoff, eng.occ, eng.g.nat, nat0, a_full,
                                                                   ak3 / 1.5);
  note_launch();
  if (check_launch("GPU EVALQ local alpha^-1 P")) return 306;
  const cplx<T>* A[2] = {p, e};
  const cplx<T>* B[2] = {qbuf, p};
  const int cj[2] = {1, 1};
  double2 o[2];
  if (ops.dots(3 * nat0, 2, A, B, cj, o)) return 307;
  *zabs = o[0];
  *zep = o[1];
  return 0;
}

// ---------------------------------------------------------------- far field
// S_d = sum over x rows of ey_d[iy] ez_d[iz] (sum_ix ex_d[ix] P[ix]): the inner
// sums are a complex matrix product, directions x columns x (rows, components),
// and only the row sums meet the y and z phases.  12 multiply-adds per site,
// component triple and direction instead of the 30 operations and three
// gathered table reads of a per-site phase.
//   block: FF_WARPS warps share one tile of ex, FF_COLS columns x 64 directions,
//     in shared memory; a lane holds two adjacent directions;
//   warp: takes pairs of x rows (strided over the grid of row blocks), packs the
//     columns where either row is occupied into records in shared memory
//     (vacuum costs nothing), and accumulates the pair's row sums in registers;
//   per pair: row sums times the y and z phases, accumulated in FP64.
// Bound by the FMA pipes: a record is 48 multiply-adds per lane against 8
// wavefronts of shared-memory reads (32 cycles for the SM's four schedulers).
// Packed fma.rn.f32x2 was measured slower (it runs at half the rate of a scalar
// FMA and needs separate real and imaginary accumulators).
// Precision (FP32): neighbouring sites of a row add up coherently, so a plain
// FP32 chain over the row rounds larger partial sums than a per-site form whose
// threads add sites 256 apart.  Chains stop after FF_CHAIN products and meet in
// a compensated (Kahan) sum, and the y and z phases multiply the row sums in
// FP64: off-peak amplitudes (below 5 % of the peak) of 33^3 to 111^3
// spheres are 5.1e-8 to 9.3e-8 off in norm against 6.0e-8 to 1.0e-7 for the
// per-site form; plain chains of 32 gave 9.2e-8 to 1.8e-7.
// Measured, 96^3 sphere, FP32: 2.62 ms against 5.73 for the per-site
// form (7,500 directions; 1.1 ms at the FMA peak); 64^3, FP64, 8 polarisations:
// 4.93 against 9.97 ms.
constexpr int FF_WARPS = 12;
constexpr int FF_COLS = 64;
constexpr int FF_CHAIN = 8;
constexpr int FF_ND = 2;            // directions per lane
constexpr int FF_TILE = 32 * FF_ND;  // directions per block

// y and z phases tabulated per direction: yz[u][d], u < ny: exp(-i ky (iy+1+x0y) dy),
// then nz entries, in FP64; ex[u][d] = exp(-i kx (ix+1+x0x) dx) in FP64, stored as
// complex float (SCAT) or complex double (the all-FP64 amplitudes); zero for the
// padding directions ndir <= d < pitch
template <typename TC>
__global__ void k_ff_tables(const double* dirs, int ndir, int pitch, int nx, int ny, int nz, double dx0, double dx1,
                            double dx2, double x00, double x01, double x02, TC* ex, double2* yz) {
  const size_t tot = (size_t)pitch * (nx + ny + nz);
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
    const int d = (int)(t % pitch), u = (int)(t / pitch);
    double s = 0.0, c = 0.0;
    if (d < ndir) {
      double ph;
      if (u < nx) ph = dirs[3 * d] * ((u + 1) + x00) * dx0;
      else if (u < nx + ny) ph = dirs[3 * d + 1] * ((u - nx + 1) + x01) * dx1;
      else ph = dirs[3 * d + 2] * ((u - nx - ny + 1) + x02) * dx2;
      sincos(ph, &s, &c);
    }
    if (u < nx) ex[t] = mk<TC>(c, -s);
    else yz[t - (size_t)pitch * nx] = make_double2(c, -s);
  }
}

// Site position r_j = ((i+1) + x0) * dx of the far-field sums, per axis
struct SitePos {
  float x0[3], dx[3];
};

// acc += p * e
template <typename C> __device__ __forceinline__ void cfma(C& acc, C p, C e) {
  acc.x = fma(p.x, e.x, acc.x);
  acc.y = fma(p.x, e.y, acc.y);
  acc.x = fma(-p.y, e.y, acc.x);
  acc.y = fma(p.y, e.x, acc.y);
}
// n (even for 8-byte elements) elements by 16-byte loads
template <int N, typename C> __device__ __forceinline__ void load_vec(C (&v)[N], const C* src) {
  if constexpr (sizeof(C) == 8) {
    static_assert(N % 2 == 0, "pairs");
#pragma unroll
    for (int k = 0; k < N; k += 2) {
      const float4 q = *reinterpret_cast<const float4*>(src + k);
      v[k] = mk<C>(q.x, q.y);
      v[k + 1] = mk<C>(q.z, q.w);
    }
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = src[k];
  }
}

// shared memory of k_ff_rows: ex tile | records | column offsets
template <typename TR> constexpr size_t ff_smem() {
  return (size_t)FF_COLS * FF_TILE * sizeof(cplx<TR>) +
         (size_t)FF_WARPS * FF_COLS * (6 * sizeof(cplx<TR>) + sizeof(int));
}

// s[c][d] += sum over the records [j0, j1) of record component c times ex
template <typename TC>
__device__ __forceinline__ void ff_chain(TC (&s)[6][FF_ND], const TC* rec, const int* col, const TC* ex, int j0, int j1) {
#pragma unroll 2
  for (int j = j0; j < j1; ++j) {
    TC x[FF_ND], r[6];
    load_vec(x, ex + col[j]);
    load_vec(r, rec + 6 * j);
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int d = 0; d < FF_ND; ++d) cfma(s[c][d], r[c], x[d]);
  }
}
template <typename TC> __device__ __forceinline__ void ff_clear(TC (&s)[6][FF_ND]) {
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int d = 0; d < FF_ND; ++d) s[c][d] = mk<TC>(0, 0);
}
// Kahan step: sum += v with the running compensation k
__device__ __forceinline__ void kahan(float& sum, float& k, float v) {
  const float y = v - k, t = sum + y;
  k = (t - sum) - y;
  sum = t;
}

// Partial sums of one direction tile (blockIdx.y), column chunk (blockIdx.z)
// and share of the row pairs (blockIdx.x) into partials[part][3*d + c], part =
// blockIdx.z * gridDim.x + blockIdx.x.  wt = 0: weight 1; 1..3: each site
// weighted by its x, y or z position (the moments U of the torque).
template <typename C, typename TR>
__global__ void __launch_bounds__(32 * FF_WARPS, 1) k_ff_rows(const C* p, const int* inv, int nat0, int nrows, int pitch, int nx,
                                                              int ny,
                                                              const cplx<TR>* tab, const double2* yz,
                                                              double2* partials, int wt, SitePos pos) {
  using TC = cplx<TR>;
  constexpr int ND = FF_ND, TILE = FF_TILE, H = FF_COLS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TC* ext = reinterpret_cast<TC*>(smem_raw);  // [FF_COLS][TILE]
  TC* recs = ext + FF_COLS * TILE;            // [FF_WARPS][FF_COLS][6]: 2 rows x 3 components
  int* cols = reinterpret_cast<int*>(recs + FF_WARPS * FF_COLS * 6);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int d0 = blockIdx.y * TILE, k0 = blockIdx.z * FF_COLS, ncol = min(FF_COLS, nx - k0);
  {
    // 16-byte moves: TILE and pitch are even in elements
    constexpr int V = 16 / (int)sizeof(TC), W = TILE / V;
    for (int u = threadIdx.x; u < ncol * W; u += 32 * FF_WARPS) {
      const int k = u / W, v = u - k * W;
      reinterpret_cast<float4*>(ext)[u] = reinterpret_cast<const float4*>(tab + (size_t)(k0 + k) * pitch + d0)[v];
    }
  }
  __syncthreads();
  TC* myrec = recs + wid * FF_COLS * 6;
  int* mycol = cols + wid * FF_COLS;
  const TC* mye = ext + ND * lane;
  double2 acc[3][ND];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < ND; ++d) acc[c][d] = make_double2(0.0, 0.0);
  const int npair = (nrows + 1) / 2, stride = gridDim.x * FF_WARPS;
  // compact indices of the lane's columns in both rows of a pair, -1 for
  // vacuum; those of the next pair load while this one is summed
  int q[2][H];
  auto load_q = [&](int pr) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int row = 2 * pr + r, k = 32 * h + lane;
        q[r][h] = pr < npair && row < nrows && k < ncol ? inv[(size_t)row * nx + k0 + k] : -1;
      }
  };
  load_q(blockIdx.x * FF_WARPS + wid);
  for (int pr = blockIdx.x * FF_WARPS + wid; pr < npair; pr += stride) {
    const int rows[2] = {2 * pr, min(2 * pr + 1, nrows - 1)};
    int cnt = 0;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int k = 32 * h + lane;
      const bool occ = q[0][h] >= 0 || q[1][h] >= 0;
      const unsigned m = __ballot_sync(0xffffffffu, occ);
      if (occ) {
        const int j = cnt + __popc(m & ((1u << lane) - 1u));
        mycol[j] = k * TILE;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          TR w = (TR)1;
          if (wt) {
            const int i = wt == 1 ? k0 + k : (wt == 2 ? rows[r] % ny : rows[r] / ny);
            w = ((TR)(i + 1) + (TR)pos.x0[wt - 1]) * (TR)pos.dx[wt - 1];
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            TC v = mk<TC>(0, 0);
            if (q[r][h] >= 0) v = p[(size_t)c * nat0 + q[r][h]];
            myrec[6 * j + 3 * r + c] = wt ? cscale(v, w) : v;
          }
        }
      }
      cnt += __popc(m);
    }
    __syncwarp();
    load_q(pr + stride);
    if (cnt) {
      TC s[6][ND];
      ff_clear(s);
      if constexpr (sizeof(TR) == 8) {
        ff_chain(s, myrec, mycol, mye, 0, cnt);
      } else {
        ff_chain(s, myrec, mycol, mye, 0, min(cnt, FF_CHAIN));
        TC k[6][ND];
        ff_clear(k);
        for (int j0 = FF_CHAIN; j0 < cnt; j0 += FF_CHAIN) {
          TC v[6][ND];
          ff_clear(v);
          ff_chain(v, myrec, mycol, mye, j0, min(cnt, j0 + FF_CHAIN));
#pragma unroll
          for (int c = 0; c < 6; ++c)
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              kahan(s[c][d].x, k[c][d].x, v[c][d].x);
              kahan(s[c][d].y, k[c][d].y, v[c][d].y);
            }
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const double2* ey = yz + (size_t)(rows[r] % ny) * pitch + d0 + ND * lane;
        const double2* ez = yz + (size_t)(ny + rows[r] / ny) * pitch + d0 + ND * lane;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const double2 e = cmul(ey[d], ez[d]);
#pragma unroll
          for (int c = 0; c < 3; ++c) cfma(acc[c][d], to_d(s[3 * r + c][d]), e);
        }
      }
    }
    __syncwarp();  // the records are consumed before the next pair overwrites them
  }
  // the warps' sums meet in shared memory (fixed order), one partial per block
  __syncthreads();
  double2* red = reinterpret_cast<double2*>(smem_raw);  // [FF_WARPS][3 * TILE]
  static_assert((size_t)FF_WARPS * 3 * TILE * sizeof(double2) <= ff_smem<TR>(), "block reduction space");
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < ND; ++d) red[wid * 3 * TILE + 3 * (ND * lane + d) + c] = acc[c][d];
  __syncthreads();
  double2* out = partials + (size_t)(blockIdx.z * gridDim.x + blockIdx.x) * 3 * pitch + (size_t)3 * d0;
  for (int t = threadIdx.x; t < 3 * TILE; t += 32 * FF_WARPS) {
    double2 v = red[t];
#pragma unroll
    for (int w = 1; w < FF_WARPS; ++w) v = cadd(v, red[w * 3 * TILE + t]);
    out[t] = v;
  }
}

// sums[d][base + step*c] = the parts' partials in part order
__global__ void k_ff_final(const double2* partials, int nparts, int rows, int part_stride, int ns, int base, int step,
                           double2* sums) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  double2 s = make_double2(0, 0);
  for (int b = 0; b < nparts; ++b) s = cadd(s, partials[(size_t)b * part_stride + r]);
  const int d = r / 3, c = r - 3 * d;
  sums[(size_t)d * ns + base + step * c] = s;
}

// Far-field sums of a compact polarisation p (device) over ndir directions,
// phases and row sums in TR; NS sums per direction (3: S, 12: S and the position
// moments U_ab = sum_j P_ja r_jb exp(-i k.r_j), a-major), sums_host[dir][NS].
template <typename C, typename TR, int NS = 3>
static int ff_sums_impl(const int* inv, int nx, int ny, int nz, int nat0, const C* p,
                        const double* dirs_host, int ndir, const double dx[3], const double x0[3], double2* sums_host,
                        cudaStream_t s) {
  using TC = cplx<TR>;
  if (nx > 2047 || ny > 2047 || nz > 1023) { set_error("GPU SCAT", "grid too large for the far-field sums"); return 322; }
  constexpr int TILE = FF_TILE;
  const int chunk = std::min(4096, (int)ceil_div(std::max(ndir, 1), TILE) * TILE);  // directions per launch
  const int nrows = ny * nz, npair = (nrows + 1) / 2, kch = (int)ceil_div(nx, FF_COLS), ntab = nx + ny + nz;
  // row blocks: at least 4 waves of one block per SM where each warp still
  // gets two row pairs (the ex tile is loaded once per block)
  auto row_blocks = [&](int tiles) {
    const size_t want = ceil_div((size_t)4 * 148, (size_t)tiles * kch);
    return (int)std::max<size_t>(1, std::min<size_t>(want, ceil_div((size_t)npair, 2 * FF_WARPS)));
  };
  size_t npartial = 0;
  for (int off = 0; off < ndir; off += chunk) {
    const int tiles = (int)ceil_div(std::min(chunk, ndir - off), TILE);
    npartial = std::max(npartial, (size_t)row_blocks(tiles) * kch * 3 * tiles * TILE);
  }
  double* d_dirs = nullptr;
  TC* tab = nullptr;
  double2 *yz = nullptr, *partials = nullptr, *sums = nullptr;
  int rc = 0;
  cudaError_t e = dev_alloc((void**)&d_dirs, (size_t)3 * chunk * sizeof(double));
  if (e == cudaSuccess) e = dev_alloc((void**)&tab, (size_t)chunk * nx * sizeof(TC));
  if (e == cudaSuccess) e = dev_alloc((void**)&yz, (size_t)chunk * (ny + nz) * sizeof(double2));
  if (e == cudaSuccess) e = dev_alloc((void**)&partials, npartial * sizeof(double2));
  if (e == cudaSuccess) e = dev_alloc((void**)&sums, (size_t)chunk * NS * sizeof(double2));
  if (e != cudaSuccess) { set_cuda_error("SCAT workspace", e); rc = 322; }
  if (!rc) {
    raise_smem_limit((const void*)k_ff_rows<C, TR>);
    SitePos pos;
    for (int k = 0; k < 3; ++k) { pos.x0[k] = (float)x0[k]; pos.dx[k] = (float)dx[k]; }
    for (int off = 0; off < ndir && !rc; off += chunk) {
      const int cnt = std::min(chunk, ndir - off), tiles = (int)ceil_div(cnt, TILE), pitch = tiles * TILE;
      const int nb = row_blocks(tiles);
      cudaMemcpyAsync(d_dirs, dirs_host + (size_t)3 * off, (size_t)3 * cnt * sizeof(double), cudaMemcpyHostToDevice, s);
      k_ff_tables<TC><<<(unsigned)std::min<size_t>(ceil_div((size_t)pitch * ntab, 256), 4096), 256, 0, s>>>(
          d_dirs, cnt, pitch, nx, ny, nz, dx[0], dx[1], dx[2], x0[0], x0[1], x0[2], tab, yz);
      note_launch();
      for (int wt = 0; wt <= (NS == 12 ? 3 : 0); ++wt) {
        k_ff_rows<C, TR><<<dim3((unsigned)nb, (unsigned)tiles, (unsigned)kch), 32 * FF_WARPS, ff_smem<TR>(), s>>>(
            p, inv, nat0, nrows, pitch, nx, ny, tab, yz, partials, wt, pos);
        note_launch();
        k_ff_final<<<(unsigned)ceil_div((size_t)cnt * 3, 128), 128, 0, s>>>(partials, nb * kch, cnt * 3, 3 * pitch, NS,
                                                                            wt ? 2 + wt : 0, wt ? 3 : 1, sums);
        note_launch();
      }
      if (check_launch("SCAT far-field sums")) { rc = 325; break; }
      e = cudaMemcpyAsync(sums_host + (size_t)NS * off, sums, (size_t)NS * cnt * sizeof(double2), cudaMemcpyDeviceToHost,
                          s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) { set_cuda_error("SCAT sums D2H", e); rc = 329; }
    }
  }
  if (rc) cudaStreamSynchronize(s);
  dev_free(d_dirs); dev_free(tab); dev_free(yz); dev_free(partials); dev_free(sums);
  return rc;
}

template <typename T>
int farfield_sums(Engine<T>& eng, const cplx<T>* p, const float* dirs_host, int ndir, const float dx[3], const float x0[3],
                  double2* sums_host, cudaStream_t s) {
  std::vector<double> hd((size_t)3 * std::max(ndir, 0));
  for (size_t i = 0; i < hd.size(); ++i) hd[i] = (double)dirs_host[i];
  const double dxd[3] = {dx[0], dx[1], dx[2]}, x0d[3] = {x0[0], x0[1], x0[2]};
  return ff_sums_impl<cplx<T>, float>(eng.inv, eng.g.nx, eng.g.ny, eng.g.nz, eng.g.nat0, p, hd.data(), ndir,
                                      dxd, x0d, sums_host, s);
}

template <typename T>
int farfield_torque_sums(Engine<T>& eng, const cplx<T>* p, const double* dirs_host, int ndir, const float dx[3],
                         const float x0[3], double2* sums_host, cudaStream_t s) {
  const double dxd[3] = {dx[0], dx[1], dx[2]}, x0d[3] = {x0[0], x0[1], x0[2]};
  return ff_sums_impl<cplx<T>, float, 12>(eng.inv, eng.g.nx, eng.g.ny, eng.g.nz, eng.g.nat0, p, dirs_host,
                                          ndir, dxd, x0d, sums_host, s);
}

// Torque of the incident field E on the dipoles P (compact), per block:
// sum_j 1/2 Re(P_j x conj(E_j)) and sum_j (k/2) Im(P_j . conj(E_j)) r_j x k-hat*|k|,
// six FP64 partials per block, folded in block order by k_torque_final.
template <typename C>
__global__ void __launch_bounds__(256) k_torque_inc(const C* p, const C* e, const int* occ, int nat0, int nx, int ny,
                                                    SitePos pos, double kx, double ky, double kz, double* partials) {
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nat0; q += gridDim.x * blockDim.x) {
    const int j = occ[q];
    const double r0 = ((j % nx) + 1 + (double)pos.x0[0]) * pos.dx[0];
    const double r1 = (((j / nx) % ny) + 1 + (double)pos.x0[1]) * pos.dx[1];
    const double r2 = ((j / (nx * ny)) + 1 + (double)pos.x0[2]) * pos.dx[2];
    const double2 p0 = to_d(p[q]), p1 = to_d(p[q + nat0]), p2 = to_d(p[q + 2 * (size_t)nat0]);
    const double2 e0 = to_d(e[q]), e1 = to_d(e[q + nat0]), e2 = to_d(e[q + 2 * (size_t)nat0]);
    // Re(a conj(b)) and Im(a conj(b))
    auto rc = [](double2 a, double2 b) { return a.x * b.x + a.y * b.y; };
    auto ic = [](double2 a, double2 b) { return a.y * b.x - a.x * b.y; };
    acc[0] += 0.5 * (rc(p1, e2) - rc(p2, e1));
    acc[1] += 0.5 * (rc(p2, e0) - rc(p0, e2));
    acc[2] += 0.5 * (rc(p0, e1) - rc(p1, e0));
    const double w = 0.5 * (ic(p0, e0) + ic(p1, e1) + ic(p2, e2));
    acc[3] += w * (r1 * kz - r2 * ky);
    acc[4] += w * (r2 * kx - r0 * kz);
    acc[5] += w * (r0 * ky - r1 * kx);
  }
  __shared__ double red[8][6];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = acc[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w][threadIdx.x];
    partials[(size_t)blockIdx.x * 6 + threadIdx.x] = v;
  }
}

__global__ void k_torque_final(const double* partials, int nblocks, double* out) {
  const int k = threadIdx.x;
  if (k >= 6) return;
  double v = 0.0;
  for (int b = 0; b < nblocks; ++b) v += partials[(size_t)b * 6 + k];
  out[k] = v;
}

// gamma[0..2]: spin part, gamma[3..5]: orbital part of the incident-field torque
template <typename T>
int incident_torque(Engine<T>& eng, const cplx<T>* p, const cplx<T>* e, const float dx[3], const float x0[3],
                    const double k[3], double gamma[6], cudaStream_t s) {
  const int nat0 = eng.g.nat0;
  const int nblocks = (int)std::min<size_t>(ceil_div((size_t)nat0, 256), 1184);
  double* d = nullptr;
  cudaError_t e1 = dev_alloc((void**)&d, ((size_t)nblocks * 6 + 6) * sizeof(double));
  if (e1 != cudaSuccess) { set_cuda_error("torque workspace", e1); return 341; }
  SitePos pos;
  for (int i = 0; i < 3; ++i) { pos.x0[i] = x0[i]; pos.dx[i] = dx[i]; }
  k_torque_inc<<<(unsigned)nblocks, 256, 0, s>>>(p, e, eng.occ, nat0, eng.g.nx, eng.g.ny, pos, k[0], k[1], k[2], d + 6);
  note_launch();
  k_torque_final<<<1, 32, 0, s>>>(d + 6, nblocks, d);
  note_launch();
  int rc = 0;
  if (check_launch("torque sums")) rc = 342;
  if (!rc) {
    e1 = cudaMemcpyAsync(gamma, d, 6 * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e1 == cudaSuccess) e1 = cudaStreamSynchronize(s);
    if (e1 != cudaSuccess) { set_cuda_error("torque sums D2H", e1); rc = 343; }
  }
  if (rc) cudaStreamSynchronize(s);
  dev_free(d);
  return rc;
}

template int farfield_torque_sums<float>(Engine<float>&, const float2*, const double*, int, const float*, const float*,
                                         double2*, cudaStream_t);
template int incident_torque<float>(Engine<float>&, const float2*, const float2*, const float*, const float*,
                                    const double*, double*, cudaStream_t);

int farfield_sums_f64(const Engine<float>& eng, const double2* p, const double* dirs_host, int ndir,
                      const double dx[3], const double x0[3], double2* sums_host, cudaStream_t s) {
  return ff_sums_impl<double2, double>(eng.inv, eng.g.nx, eng.g.ny, eng.g.nz, eng.g.nat0, p, dirs_host, ndir,
                                       dx, x0, sums_host, s);
}

// --------------------------------------------------------------------------
// Amplitude matrix (S1..S4) and Mueller matrix (S_ij) per scattering direction,
// the step DDSCAT's GETMUELLER performs after SCAT (not in the reference).
// Definitions of Bohren & Huffman (1983), section 3.2 and eq. 3.16; f_ml as
// ddscat_cuda_scat_f32 returns them (k times the physical amplitude), so
// S = -i f.  DDSCAT's basis has EM2 = n x EM1 (phi-hat); Bohren & Huffman's
// perpendicular vector is -EM2 for scattered and incident light, and
// e_par,i = khat x e_perp,i.  With g_1l = f_1l and g_2l = -f_2l:
//   S2 = -i sum_l g_1l conj(e0l).e_par   S3 = -i sum_l g_1l conj(e0l).e_perp
//   S4 = -i sum_l g_2l conj(e0l).e_par   S1 = -i sum_l g_2l conj(e0l).e_perp
struct MuellerIn {
  double kh[3];
  double2 e0c[2][3];  // conj(e01), conj(e02)
};

__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) { return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }  // a conj(b)

template <typename R>
__global__ void k_mueller(int ndir, MuellerIn in, const R* em2, const cplx<R>* f11, const cplx<R>* f21,
                          const cplx<R>* f12, const cplx<R>* f22, cplx<R>* s_out, double* m_out) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= ndir) return;
  const double ep[3] = {-(double)em2[3 * d], -(double)em2[3 * d + 1], -(double)em2[3 * d + 2]};  // e_perp = -EM2
  const double ea[3] = {in.kh[1] * ep[2] - in.kh[2] * ep[1], in.kh[2] * ep[0] - in.kh[0] * ep[2],
                        in.kh[0] * ep[1] - in.kh[1] * ep[0]};
  double2 cpar[2], cperp[2];
  for (int l = 0; l < 2; ++l) {
    cpar[l] = make_double2(0.0, 0.0);
    cperp[l] = make_double2(0.0, 0.0);
    for (int k = 0; k < 3; ++k) {
      cpar[l].x += ea[k] * in.e0c[l][k].x; cpar[l].y += ea[k] * in.e0c[l][k].y;
      cperp[l].x += ep[k] * in.e0c[l][k].x; cperp[l].y += ep[k] * in.e0c[l][k].y;
    }
  }
  const double2 a11 = to_d(f11[d]), a12 = to_d(f12[d]);
  const double2 a21 = make_double2(-(double)f21[d].x, -(double)f21[d].y);  // g_2l = -f_2l
  const double2 a22 = make_double2(-(double)f22[d].x, -(double)f22[d].y);
  using C = cplx<R>;
  auto mi = [](double2 z) { return make_double2(z.y, -z.x); };  // -i z
  auto add = [](double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); };
  const double2 S2 = mi(add(zmul(a11, cpar[0]), zmul(a12, cpar[1])));
  const double2 S3 = mi(add(zmul(a11, cperp[0]), zmul(a12, cperp[1])));
  const double2 S4 = mi(add(zmul(a21, cpar[0]), zmul(a22, cpar[1])));
  const double2 S1 = mi(add(zmul(a21, cperp[0]), zmul(a22, cperp[1])));
  if (s_out) {
    s_out[4 * d] = mk<C>(S1.x, S1.y);
    s_out[4 * d + 1] = mk<C>(S2.x, S2.y);
    s_out[4 * d + 2] = mk<C>(S3.x, S3.y);
    s_out[4 * d + 3] = mk<C>(S4.x, S4.y);
  }
  const double q1 = zabs2(S1), q2 = zabs2(S2), q3 = zabs2(S3), q4 = zabs2(S4);
  const double2 s23 = zmulc(S2, S3), s14 = zmulc(S1, S4), s24 = zmulc(S2, S4), s13 = zmulc(S1, S3);
  const double2 s12 = zmulc(S1, S2), s34 = zmulc(S3, S4);
  double* M = m_out + (size_t)16 * d;
  M[0] = 0.5 * (q2 + q1 + q4 + q3);
  M[1] = 0.5 * (q2 - q1 + q4 - q3);
  M[2] = s23.x + s14.x;
  M[3] = s23.y - s14.y;
  M[4] = 0.5 * (q2 - q1 - q4 + q3);
  M[5] = 0.5 * (q2 + q1 - q4 - q3);
  M[6] = s23.x - s14.x;
  M[7] = s23.y + s14.y;
  M[8] = s24.x + s13.x;
  M[9] = s24.x - s13.x;
  M[10] = s12.x + s34.x;
  M[11] = -s12.y - s34.y;   // Im(S2 S1* + S4 S3*)
  M[12] = -s24.y + s13.y;   // Im(S4 S2* + S1 S3*)
  M[13] = -s24.y - s13.y;   // Im(S4 S2* - S1 S3*)
  M[14] = s12.y - s34.y;    // Im(S1 S2* - S3 S4*)
  M[15] = s12.x - s34.x;
}

template <typename R>
static int mueller_impl(int ndir, const R* ak, const cplx<R>* e01, const cplx<R>* e02, const R* em2, const cplx<R>* f11,
                        const cplx<R>* f21, const cplx<R>* f12, const cplx<R>* f22, cplx<R>* s_out, double* m_out) {
  using C = cplx<R>;
  MuellerIn in{};
  const double kk = std::sqrt((double)ak[0] * ak[0] + (double)ak[1] * ak[1] + (double)ak[2] * ak[2]);
  if (!(kk > 0.0)) { set_error("Mueller", "zero incident wave vector"); return 700; }
  for (int k = 0; k < 3; ++k) {
    in.kh[k] = ak[k] / kk;
    in.e0c[0][k] = make_double2(e01[k].x, -e01[k].y);
    in.e0c[1][k] = make_double2(e02[k].x, -e02[k].y);
  }
  const size_t off_f = ((size_t)ndir * 3 * sizeof(R) + 15) & ~(size_t)15;  // 16-byte aligned f block
  const size_t nb = off_f + (size_t)ndir * (8 * sizeof(C) + 16 * sizeof(double));
  unsigned char* buf = nullptr;
  cudaError_t e = dev_alloc((void**)&buf, nb);
  if (e != cudaSuccess) { set_cuda_error("Mueller workspace", e); return 701; }
  R* d_em2 = reinterpret_cast<R*>(buf);
  C* d_f = reinterpret_cast<C*>(buf + off_f);
  C* d_s = d_f + (size_t)4 * ndir;
  double* d_m = reinterpret_cast<double*>(d_s + (size_t)4 * ndir);
  const C* hf[4] = {f11, f21, f12, f22};
  e = cudaMemcpy(d_em2, em2, (size_t)ndir * 3 * sizeof(R), cudaMemcpyHostToDevice);
  for (int k = 0; k < 4 && e == cudaSuccess; ++k)
    e = cudaMemcpy(d_f + (size_t)k * ndir, hf[k], (size_t)ndir * sizeof(C), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) { dev_free(buf); set_cuda_error("Mueller H2D", e); return 702; }
  k_mueller<R><<<(unsigned)ceil_div(ndir, 128), 128>>>(ndir, in, d_em2, d_f, d_f + ndir, d_f + 2 * (size_t)ndir,
                                                       d_f + 3 * (size_t)ndir, d_s, d_m);
  note_launch();
  if (check_launch("Mueller kernel")) { dev_free(buf); return 703; }
  if (s_out) e = cudaMemcpy(s_out, d_s, (size_t)ndir * 4 * sizeof(C), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(m_out, d_m, (size_t)ndir * 16 * sizeof(double), cudaMemcpyDeviceToHost);
  dev_free(buf);
  if (e != cudaSuccess) { set_cuda_error("Mueller D2H", e); return 702; }
  return 0;
}

int mueller_compute(int ndir, const float* ak, const float2* e01, const float2* e02, const float* em2,
                    const float2* f11, const float2* f21, const float2* f12, const float2* f22, float2* s_out,
                    double* m_out) {
  return mueller_impl<float>(ndir, ak, e01, e02, em2, f11, f21, f12, f22, s_out, m_out);
}

int mueller_compute_f64(int ndir, const double* ak, const double2* e01, const double2* e02, const double* em2,
                        const double2* f11, const double2* f21, const double2* f12, const double2* f22,
                        double2* s_out, double* m_out) {
  return mueller_impl<double>(ndir, ak, e01, e02, em2, f11, f21, f12, f22, s_out, m_out);
}

template int evalq_compute<float>(Engine<float>&, VecOps<float>&, const float2*, const float2*, const float2*,
                                  const float2*, int, float2*, double, double2*, double2*);
template int evalq_compute<double>(Engine<double>&, VecOps<double>&, const double2*, const double2*, const double2*,
                                   const double2*, int, double2*, double, double2*, double2*);
template int farfield_sums<float>(Engine<float>&, const float2*, const float*, int, const float[3], const float[3],
                                  double2*, cudaStream_t);

}  // namespace ddb
