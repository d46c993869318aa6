// J/K from packed ERIs (the reference's PackedJK, csrc/packed_jk.cc:6-80):
// s8 storage (np(np+1)/2 values, np = n(n+1)/2) or s4 (np x np), any real
// density batch (nonsymmetric allowed), output (with_j + with_k, nb, n, n)
// overwritten.
//
// What the operation cannot do without is one read of the lower triangle
// (ab >= cd) per result; the arithmetic per element is two multiply-adds for J
// and four for K per symmetric density.  The previous form read it once but
// added J[c][d] to memory per element and reduced K[a][c] over a warp for
// every c: 5.82 ms for n = 168, two densities (807 MB).  Here J and K are two
// passes that read it once each: 0.77 ms at that size, three times what the two
// reads take at the copy rate.  Under ncu the J pass (0.27 ms) reads 3.0 TB/s and
// the K pass (0.50 ms) 1.6 TB/s: two warps a scheduler (176 and 168 registers)
// wait on fixed latencies and on their loads, in K with the L1 data stage 54%
// busy from the tiles' transposes and broadcast reads.
//   J: J = M x with M the symmetric pair matrix, x_cd = D_cd + D_dc.  A block
//      takes 128 rows x 1024 columns; a thread keeps its four columns' x and
//      column sums in registers (one add per column and block), and the row
//      dot products of eight rows are reduced together.
//   K: with S the triangle of row ab as a symmetric matrix over (c, d),
//      MK[a][.] += S D[b][.], MK[b][.] += S D[a][.], K = MK + MK^T for the
//      symmetric part of D and MK - MK^T for the antisymmetric part (skipped
//      on the device when it is zero).  A warp takes one row, in 32 x 32
//      tiles held in registers: once with the lanes on d, once transposed
//      through shared memory with the lanes on c, so no element needs a
//      reduction over lanes.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <stdexcept>
#include <string>

#include "b200jk.h"
#include "plan.h"

namespace b200jk {
namespace {

// i >= j with pair = i(i+1)/2 + j
__device__ __forceinline__ void unpair(long long pr, int& i, int& j) {
  long long r = (long long)((sqrt(8.0 * (double)pr + 1.0) - 1.0) * 0.5);
  while (r * (r + 1) / 2 > pr) --r;
  while ((r + 1) * (r + 2) / 2 <= pr) ++r;
  i = (int)r;
  j = (int)(pr - r * (r + 1) / 2);
}

__device__ __forceinline__ const double* eri_row(const double* eri, int layout, long long np, long long ab) {
  return layout == 1 ? eri + ab * (ab + 1) / 2 : eri + ab * np;
}

// Density batch -> x (pair-packed, for J) and the symmetric and antisymmetric
// parts (for K); anti[e] is set when density e has an antisymmetric part.
__global__ void packed_prep_kernel(const double* __restrict__ dens, int n, long long np, int nb,
                                   double* __restrict__ x, double* __restrict__ sym, double* __restrict__ asym,
                                   int* __restrict__ anti) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nn = (long long)n * n;
  if (idx >= nn * nb) return;
  const int e = (int)(idx / nn);
  const long long r = idx - e * nn;
  const int i = (int)(r / n), j = (int)(r % n);
  const double dij = dens[idx], dji = dens[e * nn + (long long)j * n + i];
  if (x && i >= j) x[e * np + (long long)i * (i + 1) / 2 + j] = i == j ? dij : dij + dji;
  if (sym) {
    const double t = dij == dji ? 0.0 : 0.5 * dij - 0.5 * dji;
    sym[idx] = 0.5 * dij + 0.5 * dji;
    asym[idx] = t;
    if (t != 0.0) anti[e] = 1;   // every writer stores the same value (a NaN counts)
  }
}

constexpr int kJRows = 128, kJCols = 4, kJThreads = 256, kJGroup = 8;

// jp[e][ab] += sum_cd M[ab][cd] x[e][cd] over both triangles, NE densities.
template <int NE>
__global__ void __launch_bounds__(kJThreads) packed_j_kernel(const double* __restrict__ eri, int layout, long long np,
                                                             const double* __restrict__ x, double* __restrict__ jp) {
  const long long c0 = (long long)blockIdx.x * (kJThreads * kJCols) + threadIdx.x;
  const long long r0 = (long long)blockIdx.y * kJRows, r1 = min(r0 + kJRows, np);
  if ((long long)blockIdx.x * (kJThreads * kJCols) >= r1) return;   // wholly above the diagonal
  const int lane = threadIdx.x & 31;
  double xc[NE][kJCols], sum[NE][kJCols];
#pragma unroll
  for (int e = 0; e < NE; ++e)
#pragma unroll
    for (int q = 0; q < kJCols; ++q) {
      const long long c = c0 + q * kJThreads;
      xc[e][q] = c < np ? x[e * np + c] : 0.0;
      sum[e][q] = 0.0;
    }
  for (long long r = r0; r < r1; r += kJGroup) {
    double v[kJGroup][kJCols];
#pragma unroll
    for (int g = 0; g < kJGroup; ++g) {
      const double* row = eri_row(eri, layout, np, r + g);
#pragma unroll
      for (int q = 0; q < kJCols; ++q) {
        const long long c = c0 + q * kJThreads;
        v[g][q] = (r + g < r1 && c <= r + g) ? __ldcs(row + c) : 0.0;
      }
    }
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      double dot[kJGroup];
#pragma unroll
      for (int g = 0; g < kJGroup; ++g) {
        const double xr = r + g < r1 ? x[e * np + r + g] : 0.0;
        dot[g] = 0.0;
#pragma unroll
        for (int q = 0; q < kJCols; ++q) {
          dot[g] += v[g][q] * xc[e][q];
          sum[e][q] += c0 + q * kJThreads < r + g ? v[g][q] * xr : 0.0;   // the diagonal element counts once
        }
      }
      // eight rows over 32 lanes: each exchange halves the rows a lane holds
#pragma unroll
      for (int h = 4, off = 16; h >= 1; h /= 2, off /= 2) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int g = 0; g < h; ++g) {
          const double give = up ? dot[g] : dot[g + h], keep = up ? dot[g + h] : dot[g];
          dot[g] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      }
      double d = dot[0];
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      const long long rr = r + ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0);
      if ((lane & 3) == 0 && rr < r1 && d != 0.0) atomicAdd(jp + e * np + rr, d);
    }
  }
#pragma unroll
  for (int e = 0; e < NE; ++e)
#pragma unroll
    for (int q = 0; q < kJCols; ++q) {
      const long long c = c0 + q * kJThreads;
      if (c < np && sum[e][q] != 0.0) atomicAdd(jp + e * np + c, sum[e][q]);
    }
}

// J[i][j] = J[j][i] = jp[pair(i, j)] for every density.
__global__ void packed_j_out_kernel(const double* __restrict__ jp, int n, long long np, int nb,
                                    double* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nn = (long long)n * n;
  if (idx >= nn * nb) return;
  const int e = (int)(idx / nn);
  const long long r = idx - e * nn;
  const int i = (int)(r / n), j = (int)(r % n);
  const long long pr = i >= j ? (long long)i * (i + 1) / 2 + j : (long long)j * (j + 1) / 2 + i;
  out[idx] = jp[(long long)e * np + pr];
}

// Shared memory of one warp of packed_k_kernel, in doubles: 2 NE rows of D
// and 2 NE result rows (padded to whole tiles) and one transposed tile.
__host__ __device__ constexpr int packed_k_pad(int n) { return (n + 31) / 32 * 32; }
__host__ __device__ constexpr size_t packed_k_warp(int n, int ne) { return (size_t)4 * ne * packed_k_pad(n) + 32 * 33; }

// mk[e] += the rows a and b of MK from every row ab, longest rows first; skipped
// when `anti` is given and says that none of the NE densities has that part.
template <int NE>
__global__ void __launch_bounds__(128) packed_k_kernel(const double* __restrict__ eri, int layout, int n, long long np,
                                                       const double* __restrict__ dens, double* __restrict__ mk,
                                                       const int* __restrict__ anti) {
  if (anti) {
    int any = 0;
#pragma unroll
    for (int e = 0; e < NE; ++e) any |= anti[e];
    if (!any) return;
  }
  extern __shared__ __align__(16) double sk[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pad = packed_k_pad(n);
  const long long ab = np - 1 - ((long long)blockIdx.x * (blockDim.x >> 5) + warp);
  if (ab < 0) return;
  double* vec = sk + warp * packed_k_warp(n, NE);   // [2 NE][pad]: D_e[b][.], D_e[a][.]
  double* out = vec + 2 * NE * pad;                 // [2 NE][pad]: rows a, rows b
  double* tile = out + 2 * NE * pad;                // [32][33]
  int a, b;
  unpair(ab, a, b);
  const long long nn = (long long)n * n;
#pragma unroll
  for (int e = 0; e < NE; ++e)
    for (int i = lane; i < pad; i += 32) {
      vec[(2 * e) * pad + i] = i < n ? dens[e * nn + (long long)b * n + i] : 0.0;
      vec[(2 * e + 1) * pad + i] = i < n ? dens[e * nn + (long long)a * n + i] : 0.0;
      out[(2 * e) * pad + i] = out[(2 * e + 1) * pad + i] = 0.0;
    }
  __syncwarp();
  const double* row = eri_row(eri, layout, np, ab);
  for (int ct = 0; ct <= a; ct += 32)
    for (int dt = 0; dt <= ct; dt += 32) {
      double v[32];
      const int d = dt + lane;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int c = ct + i;
        const bool in = c <= a && d <= (c == a ? b : c);
        v[i] = in ? __ldcs(row + (long long)c * (c + 1) / 2 + d) : 0.0;
      }
      if (dt == ct) {   // c = d counts half (both orders below add it)
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i == lane) v[i] *= 0.5;
      }
      if (a < ct + 32 && b >= dt && b < dt + 32) {   // ab = cd counts half
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (ct + i == a && d == b) v[i] *= 0.5;
      }
      // lanes on d: out[d] += sum_c v[c][d] vec[c]
#pragma unroll
      for (int y = 0; y < 2 * NE; ++y) {
        const double2* q = reinterpret_cast<const double2*>(vec + y * pad + ct);
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const double2 w = q[i];
          s0 += v[2 * i] * w.x;
          s1 += v[2 * i + 1] * w.y;
        }
        out[y * pad + d] += s0 + s1;
      }
      // lanes on c: out[c] += sum_d v[c][d] vec[d]
#pragma unroll
      for (int i = 0; i < 32; ++i) tile[i * 33 + lane] = v[i];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = tile[lane * 33 + i];
      __syncwarp();
#pragma unroll
      for (int y = 0; y < 2 * NE; ++y) {
        const double2* q = reinterpret_cast<const double2*>(vec + y * pad + dt);
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const double2 w = q[i];
          s0 += v[2 * i] * w.x;
          s1 += v[2 * i + 1] * w.y;
        }
        out[y * pad + ct + lane] += s0 + s1;
      }
    }
  // c and d run up to a; a = b counts half (rows a and b are the same row)
  const double sc = a == b ? 0.5 : 1.0;
#pragma unroll
  for (int e = 0; e < NE; ++e)
    for (int i = lane; i <= a; i += 32) {
      atomicAdd(mk + e * nn + (long long)a * n + i, sc * out[(2 * e) * pad + i]);
      atomicAdd(mk + e * nn + (long long)b * n + i, sc * out[(2 * e + 1) * pad + i]);
    }
}

// K = MK + MK^T of the symmetric part, plus MK - MK^T of the antisymmetric part.
__global__ void packed_k_out_kernel(const double* __restrict__ mks, const double* __restrict__ mka,
                                    const int* __restrict__ anti, int n, int nb, double* __restrict__ out) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nn = (long long)n * n;
  if (idx >= nn * nb) return;
  const int e = (int)(idx / nn);
  const long long r = idx - e * nn;
  const long long t = e * nn + (r % n) * n + r / n;
  double v = mks[idx] + mks[t];
  if (anti[e]) v += mka[idx] - mka[t];
  out[idx] = v;
}

template <int NE>
cudaError_t launch_j(const double* eri, int layout, long long np, const double* x, double* jp, cudaStream_t st) {
  const dim3 grid((unsigned)((np + kJThreads * kJCols - 1) / (kJThreads * kJCols)),
                  (unsigned)((np + kJRows - 1) / kJRows));
  packed_j_kernel<NE><<<grid, kJThreads, 0, st>>>(eri, layout, np, x, jp);
  return cudaGetLastError();
}

constexpr size_t kMaxShared = 200 * 1024;

template <int NE>
cudaError_t launch_k(const double* eri, int layout, int n, long long np, const double* dens, double* mk,
                     const int* anti, cudaStream_t st) {
  const size_t per_warp = packed_k_warp(n, NE) * sizeof(double);
  int warps = 4;
  while (warps > 1 && warps * per_warp > kMaxShared / 2) warps /= 2;   // two blocks an SM where that fits
  static std::atomic<uint64_t> smem_done{0};
  const cudaError_t e = smem_opt_in(packed_k_kernel<NE>, kMaxShared, smem_done);
  if (e != cudaSuccess) return e;
  packed_k_kernel<NE><<<(unsigned)((np + warps - 1) / warps), 32 * warps, warps * per_warp, st>>>(eri, layout, n, np,
                                                                                             dens, mk, anti);
  return cudaGetLastError();
}

// Workspace layout of one call, in doubles from the start.
struct PackedWs {
  size_t x, jp, sym, asym, mks, mka, anti, total;
};
PackedWs packed_ws(long long n, int nb, int with_j, int with_k) {
  const size_t np = (size_t)(n * (n + 1) / 2), nn = (size_t)n * n;
  PackedWs w{};
  size_t o = 0;
  auto take = [&](size_t c) { const size_t at = o; o += (c + 31) / 32 * 32; return at; };
  w.x = take(with_j ? nb * np : 0);
  w.sym = take(with_k ? nb * nn : 0);
  w.asym = take(with_k ? nb * nn : 0);
  // zeroed together before the passes: jp, mks, mka, anti
  w.jp = take(with_j ? nb * np : 0);
  w.mks = take(with_k ? nb * nn : 0);
  w.mka = take(with_k ? nb * nn : 0);
  w.anti = take((size_t)nb);
  w.total = o;
  return w;
}

void check_packed(const double* d_eri, int layout, int64_t eri_size, int n, const double* d_density, int nb,
                  const double* d_out, int with_j, int with_k) {
  if ((with_j != 0 && with_j != 1) || (with_k != 0 && with_k != 1) || !(with_j || with_k))
    fail_invalid("Packed J/K requires at least one selected operator");
  if (!d_eri || !d_density || !d_out || n < 1 || nb < 1 || (layout != 0 && layout != 1))
    fail_invalid("Packed J/K dimensions do not match");
  const long long np = (long long)n * (n + 1) / 2;
  if (eri_size != (layout == 1 ? np * (np + 1) / 2 : np * np))
    fail_invalid("Packed J/K dimensions do not match");  // csrc/packed_jk.cc:18-22
  // a warp's exchange sums of one density (the passes take densities one or two at a time)
  if (with_k && packed_k_warp(n, 1) * sizeof(double) > kMaxShared)
    fail_invalid("Packed J/K: n too large for one row's exchange sums");
}

#define PACKED_OK(expr)                                                   \
  do {                                                                    \
    const cudaError_t _e = (expr);                                        \
    if (_e != cudaSuccess) throw std::runtime_error(cudaGetErrorString(_e)); \
  } while (0)

void run_packed(const double* eri, int layout, int n, const double* dens, int nb, double* out, int with_j, int with_k,
                double* ws, cudaStream_t st) {
  const long long np = (long long)n * (n + 1) / 2, nn = (long long)n * n, total = nn * nb;
  const PackedWs w = packed_ws(n, nb, with_j, with_k);
  int* anti = reinterpret_cast<int*>(ws + w.anti);
  const unsigned blocks = (unsigned)((total + 255) / 256);
  PACKED_OK(cudaMemsetAsync(ws + w.jp, 0, (w.total - w.jp) * sizeof(double), st));
  packed_prep_kernel<<<blocks, 256, 0, st>>>(dens, n, np, nb, with_j ? ws + w.x : nullptr,
                                             with_k ? ws + w.sym : nullptr, with_k ? ws + w.asym : nullptr, anti);
  PACKED_OK(cudaGetLastError());
  if (with_j) {
    for (int e = 0; e < nb;) {
      const double* x = ws + w.x + (size_t)e * np;
      double* jp = ws + w.jp + (size_t)e * np;
      const int ne = nb - e >= 3 ? 3 : nb - e;
      PACKED_OK(ne == 3 ? launch_j<3>(eri, layout, np, x, jp, st)
                        : ne == 2 ? launch_j<2>(eri, layout, np, x, jp, st) : launch_j<1>(eri, layout, np, x, jp, st));
      e += ne;
    }
    packed_j_out_kernel<<<blocks, 256, 0, st>>>(ws + w.jp, n, np, nb, out);
    PACKED_OK(cudaGetLastError());
  }
  if (with_k) {
    for (int part = 0; part < 2; ++part)
      for (int e = 0; e < nb;) {
        const double* d = ws + (part ? w.asym : w.sym) + (size_t)e * nn;
        double* mk = ws + (part ? w.mka : w.mks) + (size_t)e * nn;
        const int* flag = part ? anti + e : nullptr;
        const bool two = nb - e >= 2 && packed_k_warp(n, 2) * sizeof(double) <= kMaxShared;
        PACKED_OK(two ? launch_k<2>(eri, layout, n, np, d, mk, flag, st)
                      : launch_k<1>(eri, layout, n, np, d, mk, flag, st));
        e += two ? 2 : 1;
      }
    packed_k_out_kernel<<<blocks, 256, 0, st>>>(ws + w.mks, ws + w.mka, anti, n, nb, out + (size_t)with_j * total);
    PACKED_OK(cudaGetLastError());
  }
}

}  // namespace
}  // namespace b200jk

extern "C" int b200jk_packed_jk_workspace(int32_t n, int32_t nb, int32_t with_j, int32_t with_k, int64_t* bytes) {
  return b200jk::guarded_call([&] {
    if (n < 1 || nb < 1 || !bytes) b200jk::fail_invalid("Packed J/K dimensions do not match");
    *bytes = (int64_t)(b200jk::packed_ws(n, nb, with_j != 0, with_k != 0).total * sizeof(double));
  });
}

extern "C" int b200jk_packed_jk_ws(const double* d_eri, int32_t layout, int64_t eri_size, int32_t n,
                                   const double* d_density, int32_t nb, double* d_out, int32_t with_j, int32_t with_k,
                                   void* d_workspace, int64_t workspace_bytes, void* stream) {
  return b200jk::guarded_call([&] {
    b200jk::check_packed(d_eri, layout, eri_size, n, d_density, nb, d_out, with_j, with_k);
    if (!d_workspace || (reinterpret_cast<uintptr_t>(d_workspace) & 15) != 0 ||
        workspace_bytes < (int64_t)(b200jk::packed_ws(n, nb, with_j, with_k).total * sizeof(double)))
      b200jk::fail_invalid("Packed J/K workspace too small or not 16-byte aligned");
    b200jk::run_packed(d_eri, layout, n, d_density, nb, d_out, with_j, with_k, static_cast<double*>(d_workspace),
                       (cudaStream_t)stream);
  });
}

extern "C" int b200jk_packed_jk(const double* d_eri, int32_t layout, int64_t eri_size, int32_t n,
                                const double* d_density, int32_t nb, double* d_out, int32_t with_j,
                                int32_t with_k, void* stream) {
  return b200jk::guarded_call([&] {
    b200jk::check_packed(d_eri, layout, eri_size, n, d_density, nb, d_out, with_j, with_k);
    cudaStream_t st = (cudaStream_t)stream;
    // stream-ordered workspace, freed on the stream after use
    double* ws = nullptr;
    PACKED_OK(cudaMallocAsync(reinterpret_cast<void**>(&ws), b200jk::packed_ws(n, nb, with_j, with_k).total * sizeof(double), st));
    try {
      b200jk::run_packed(d_eri, layout, n, d_density, nb, d_out, with_j, with_k, ws, st);
    } catch (...) {
      cudaFreeAsync(ws, st);
      throw;
    }
    PACKED_OK(cudaFreeAsync(ws, st));
  });
}
