// Coarsest multigrid level: dense FP64 matrix over the kept dofs, explicit inverse by a blocked symmetric
// sweep over its lower tiles (symmetric positive definite, no pivoting), applied as a GEMV in every V-cycle.
// The reference factorises the same matrix (SciPy splu, fe/gmg.py:102; cuSOLVER Cholesky,
// rb/gpusolve.py:138-161); an explicit inverse turns the per-V-cycle solve into one coalesced GEMV.
#include "dense.cuh"

namespace feb {

namespace {

constexpr int SB = 64;        // sweep block: pivot block and update tile
constexpr int SLD = SB + 1;   // row pitch of transposing tiles

__global__ void k_dense_from_stencil(const double* __restrict__ A, int nx, int ny, int nz,
                                     const int* __restrict__ cmap, double* __restrict__ M, int ld) {
  const int o = threadIdx.x;
  const int64_t n = (int64_t)nx * ny * nz;
  const int64_t J = blockIdx.x * (int64_t)blockDim.y + threadIdx.y;
  if (J >= n) return;
  int cj = cmap[J];
  if (cj < 0) return;
  int i = int(J % nx), j = int((J / nx) % ny), k = int(J / ((int64_t)nx * ny));
  int dx = o % 3 - 1, dy = (o / 3) % 3 - 1, dz = o / 9 - 1;
  if (i + dx < 0 || i + dx >= nx || j + dy < 0 || j + dy >= ny || k + dz < 0 || k + dz >= nz) return;
  int64_t K = J + dx + (int64_t)nx * (dy + (int64_t)ny * dz);
  int ck = cmap[K];
  if (ck < 0) return;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c)
      M[(size_t)(3 * cj + r) * ld + 3 * ck + c] += A[(size_t)(o * 9 + 3 * r + c) * n + J];
}

__global__ void k_dense_add_entries(int nent, const int* __restrict__ rdof, const int* __restrict__ cdof,
                                    const double* __restrict__ val, const int* __restrict__ cmap,
                                    double* __restrict__ M, int ld) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nent) return;
  int cr = cmap[rdof[e] / 3], cc = cmap[cdof[e] / 3];
  if (cr < 0 || cc < 0) return;
  atomicAdd(M + (size_t)(3 * cr + rdof[e] % 3) * ld + 3 * cc + cdof[e] % 3, val[e]);
}

// Lower tiles of (M + M^T) / 2 (a diagonal tile whole); rows and columns past nd become those of the identity,
// so the sweep needs no bounds.  One CTA per tile pair; the partner tile is transposed through shared memory.
__global__ void __launch_bounds__(256) k_symmetrize(double* __restrict__ M, int nd, int ld) {
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double B[SB][SLD];
  const int c = threadIdx.x & 63, r0 = threadIdx.x >> 6;
  for (int r = r0; r < SB; r += 4) B[r][c] = M[(size_t)(tj * SB + r) * ld + ti * SB + c];
  __syncthreads();
  for (int r = r0; r < SB; r += 4) {
    const int i = ti * SB + r, j = tj * SB + c;
    double* p = M + (size_t)i * ld + j;
    *p = (i >= nd || j >= nd) ? (i == j ? 1.0 : 0.0) : 0.5 * (*p + B[c][r]);
  }
}

// M = -S from the swept lower tiles, both triangles.
__global__ void __launch_bounds__(256) k_mirror(double* __restrict__ M, int ld) {
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  __shared__ double B[SB][SLD];
  const int c = threadIdx.x & 63, r0 = threadIdx.x >> 6;
  for (int r = r0; r < SB; r += 4) {
    double* p = M + (size_t)(ti * SB + r) * ld + tj * SB + c;
    const double v = -*p;
    *p = v;
    B[r][c] = v;
  }
  if (ti == tj) return;
  __syncthreads();
  for (int r = r0; r < SB; r += 4) M[(size_t)(tj * SB + r) * ld + ti * SB + c] = B[c][r];
}

// Symmetric sweep of a 64 x 64 block held 4 x 4 per thread (rows 4 ty + u, columns 4 tx + v): step p turns
// a_pp = d into -1/d, a_ip and a_pi into a_ip / d and a_ij into a_ij - a_ip a_pj / d; after all steps the block is
// minus its inverse.  Row p travels through a double-buffered line of shared memory (its column is the same
// numbers by symmetry), so a step costs one barrier.  A non-positive pivot sets *status and counts as 1.
__device__ __forceinline__ void sweep_block(double (&a)[4][4], double (*line)[SB], int ty, int tx, int* status) {
  for (int pb = 0; pb < SB / 4; ++pb) {
#pragma unroll
    for (int pu = 0; pu < 4; ++pu) {
      const int p = 4 * pb + pu;
      double* row = line[p & 1];
      if (ty == pb) {
#pragma unroll
        for (int v = 0; v < 4; ++v) row[4 * tx + v] = a[pu][v];
      }
      __syncthreads();
      double d = row[p];
      if (!(d > 0.0) || !isfinite(d)) {
        if (threadIdx.x == 0) atomicExch(status, FEB_ERR_COARSE);
        d = 1.0;
      }
      const double ip = 1.0 / d;
      double ci[4], cj[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) { ci[u] = row[4 * ty + u] * ip; cj[u] = row[4 * tx + u]; }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const bool pr = ty == pb && u == pu, pc = tx == pb && v == pu;
          if (pr && pc) a[u][v] = -ip;
          else if (pr) a[u][v] = cj[v] * ip;
          else if (pc) a[u][v] = ci[u];
          else a[u][v] -= ci[u] * cj[v];
        }
    }
  }
}

// Dinv = inverse of the first pivot block.
__global__ void __launch_bounds__(256)
k_sweep_first(const double* __restrict__ M, int ld, double* __restrict__ Dinv, int* __restrict__ status) {
  __shared__ double line[2][SB];
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  double a[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) a[u][v] = M[(size_t)(4 * ty + u) * ld + 4 * tx + v];
  sweep_block(a, line, ty, tx, status);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) Dinv[(4 * ty + u) * SB + 4 * tx + v] = -a[u][v];
}

// Pivot panel of step k: C_i = S_ik (from the lower triangle: S_ki^T for i < k), W_i = C_i Dinv; S_ik <- W_i,
// S_kk <- -Dinv.  C and W are left transposed (k-major rows of length ld), as the update's operands.  A CTA takes
// 16 rows of block row i: at 64 rows a CTA the panel would use a third of the SMs.
__global__ void __launch_bounds__(256)
k_sweep_panel(double* __restrict__ M, int ld, int k, const double* __restrict__ Dinv, double* __restrict__ CT,
              double* __restrict__ WT) {
  __shared__ __align__(16) double Ds[SB][SB];
  __shared__ double Cs[16][SLD];
  const int i = blockIdx.x, r0 = 16 * blockIdx.y, t = threadIdx.x;
  const int row = i * SB + r0, kc = k * SB;
  if (i == k) {
    for (int e = t; e < 16 * SB; e += 256) M[(size_t)(row + e / SB) * ld + kc + e % SB] = -Dinv[(r0 + e / SB) * SB + e % SB];
    return;
  }
  for (int e = t; e < SB * SB; e += 256) Ds[e / SB][e % SB] = Dinv[e];
  for (int e = t; e < 16 * SB; e += 256) {
    if (i > k) Cs[e / SB][e % SB] = M[(size_t)(row + e / SB) * ld + kc + e % SB];
    else Cs[e % 16][e / 16] = M[(size_t)(kc + e / 16) * ld + row + e % 16];
  }
  __syncthreads();
  for (int e = t; e < 16 * SB; e += 256) CT[(size_t)(e / 16) * ld + row + e % 16] = Cs[e % 16][e / 16];
  const int r = t >> 4, c = (t & 15) * 4;
  double w[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int q = 0; q < SB; ++q) {
    const double a = Cs[r][q];
#pragma unroll
    for (int v = 0; v < 4; ++v) w[v] += a * Ds[q][c + v];
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < 4; ++v) Cs[r][c + v] = w[v];
  __syncthreads();
  for (int e = t; e < 16 * SB; e += 256) {
    const double x = Cs[e % 16][e / 16];
    WT[(size_t)(e / 16) * ld + row + e % 16] = x;
    if (i < k) M[(size_t)(kc + e / 16) * ld + row + e % 16] = x;
    else M[(size_t)(row + e / SB) * ld + kc + e % SB] = Cs[e / SB][e % SB];
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Step k's update of the lower tiles outside the pivot panel: S_ij -= C_i W_j^T (64 x 64 x 64 a CTA, 4 x 4 a
// thread).  The CTA of the next pivot block (block 0, so that it starts first) inverts it on the spot: the serial
// part of the sweep runs beside the other tiles instead of between two steps.
//
// With 32-wide pivot blocks over the whole matrix and the pivot, row, column and finish passes as kernels of their
// own, the inverse of 3510 dofs took 13.9 ms (77.7 us an update, 2.5 TB/s of matrix traffic, 40 us of serial kernels
// a step) and that of 2457 dofs 6.3 ms; this form's times stand at launch_dense_invert.
__global__ void __launch_bounds__(256)
k_sweep_update(double* __restrict__ M, int ld, int k, const double* __restrict__ CT, const double* __restrict__ WT,
               double* __restrict__ Dinv, int* __restrict__ status) {
  extern __shared__ __align__(16) double sm[];
  double (*As)[SB] = reinterpret_cast<double (*)[SB]>(sm);
  double (*Bs)[SB] = reinterpret_cast<double (*)[SB]>(sm + SB * SB);
  const int nt = ld / SB, t = threadIdx.x;
  const bool has_next = k + 1 < nt;
  // tiles a >= b over the nt - 1 block rows without k; linear index a (a + 1) / 2 + b; the next pivot (a = b = k) first
  int lin = blockIdx.x;
  const int first = k * (k + 1) / 2 + k;
  if (has_next) { if (lin == 0) lin = first; else if (lin == first) lin = 0; }
  int a = (int)((sqrtf(8.f * lin + 1.f) - 1.f) * 0.5f);
  while ((a + 1) * (a + 2) / 2 <= lin) ++a;
  while (a * (a + 1) / 2 > lin) --a;
  const int b = lin - a * (a + 1) / 2;
  const int i0 = (a + (a >= k)) * SB, j0 = (b + (b >= k)) * SB;
  for (int e = t; e < SB * SB / 2; e += 256) {
    const int q = e / (SB / 2), c = 2 * (e % (SB / 2));
    cp_async16(&As[q][c], CT + (size_t)q * ld + i0 + c);
    cp_async16(&Bs[q][c], WT + (size_t)q * ld + j0 + c);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  const int ty = t >> 4, tx = t & 15;
  double s[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double2* p = reinterpret_cast<const double2*>(M + (size_t)(i0 + 4 * ty + u) * ld + j0 + 4 * tx);
    const double2 x = p[0], y = p[1];
    s[u][0] = x.x; s[u][1] = x.y; s[u][2] = y.x; s[u][3] = y.y;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll 4
  for (int q = 0; q < SB; ++q) {
    double av[4], bv[4];
#pragma unroll
    for (int u = 0; u < 4; u += 2) {
      const double2 x = *reinterpret_cast<const double2*>(&As[q][4 * ty + u]);
      const double2 y = *reinterpret_cast<const double2*>(&Bs[q][4 * tx + u]);
      av[u] = x.x; av[u + 1] = x.y; bv[u] = y.x; bv[u + 1] = y.y;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) s[u][v] -= av[u] * bv[v];
  }
  if (has_next && blockIdx.x == 0) {
    __syncthreads();
    sweep_block(s, reinterpret_cast<double (*)[SB]>(sm), ty, tx, status);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) Dinv[(4 * ty + u) * SB + 4 * tx + v] = -s[u][v];
    return;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    double2* p = reinterpret_cast<double2*>(M + (size_t)(i0 + 4 * ty + u) * ld + j0 + 4 * tx);
    p[0] = make_double2(s[u][0], s[u][1]);
    p[1] = make_double2(s[u][2], s[u][3]);
  }
}

// x = Minv b on the coarsest level in one launch: the first brows blocks take 8 RPW rows each (RPW rows per warp), the
// remaining blocks zero the entries of nodes outside the dense system (cmap < 0), a disjoint set.  A block gathers b
// through klist into shared memory once, so that its warps stream their rows of Minv with 16-byte loads and nothing
// else (the gather inside the row loop, one 8-byte load per value, ran 2457 dofs at 28.8 us and 1.7 TB/s from L2).
constexpr int kSolveChunk = 4096;

template <typename T, int RPW>
__global__ void __launch_bounds__(256)
k_dense_solve(const double* __restrict__ Minv, int nd, int ld, const int* __restrict__ klist,
              const int* __restrict__ cmap, int64_t n, const T* __restrict__ b, T* __restrict__ x, int brows,
              const int* __restrict__ skip) {
  if (skip && *skip) return;
  if ((int)blockIdx.x < brows) {
    __shared__ __align__(16) double bs[kSolveChunk];
    const int lane = threadIdx.x & 31, row0 = (blockIdx.x * 8 + threadIdx.x / 32) * RPW;
    double acc[RPW][2] = {};
    for (int c0 = 0; c0 < nd; c0 += kSolveChunk) {
      const int len = min(kSolveChunk, ld - c0);      // a multiple of 64
      if (c0) __syncthreads();
      for (int j = threadIdx.x; j < len; j += 256) {
        const int q = c0 + j;
        bs[j] = q < nd ? double(b[3 * (int64_t)klist[q / 3] + q % 3]) : 0.0;
      }
      __syncthreads();
      if (row0 < nd) {        // rows past nd (< ld) are the identity's
        const double2* m = reinterpret_cast<const double2*>(Minv + (size_t)row0 * ld + c0) + lane;
        const double2* bb = reinterpret_cast<const double2*>(bs) + lane;
#pragma unroll 8
        for (int j = 0; j < len / 2; j += 32) {
          const double2 v = bb[j];
#pragma unroll
          for (int r = 0; r < RPW; ++r) {
            const double2 w = m[(size_t)r * (ld / 2) + j];
            acc[r][0] += w.x * v.x;
            acc[r][1] += w.y * v.y;
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const double s = warp_sum(acc[r][0] + acc[r][1]);
      const int row = row0 + r;
      if (lane == 0 && row < nd) x[3 * (int64_t)klist[row / 3] + row % 3] = T(s);
    }
    return;
  }
  const int64_t e = (int64_t)(blockIdx.x - brows) * blockDim.x + threadIdx.x;
  if (e < 3 * n && cmap[e / 3] < 0) x[e] = T(0);
}

}  // namespace

void launch_dense_from_stencil(const double* A, int nx, int ny, int nz, const int* cmap, double* M, int ld,
                               cudaStream_t s) {
  int64_t n = (int64_t)nx * ny * nz;
  dim3 blk(27, 8);
  k_dense_from_stencil<<<div_up(n, 8), blk, 0, s>>>(A, nx, ny, nz, cmap, M, ld); note_launch();
}

// M += lam_t v_t v_t^T of every term (one block per term; entries on dropped nodes are skipped)
__global__ void k_dense_add_terms(const int* __restrict__ t_ptr, const int* __restrict__ t_dof,
                                  const double* __restrict__ t_val, const double* __restrict__ t_lam,
                                  const int* __restrict__ cmap, double* __restrict__ M, int ld) {
  const int t = blockIdx.x, eb = t_ptr[t], ne = t_ptr[t + 1] - eb;
  const double lam = t_lam[t];
  for (int q = threadIdx.x; q < ne * ne; q += blockDim.x) {
    const int a = eb + q / ne, b = eb + q % ne;
    const int ca = cmap[t_dof[a] / 3], cb = cmap[t_dof[b] / 3];
    if (ca < 0 || cb < 0) continue;
    atomicAdd(M + (size_t)(3 * ca + t_dof[a] % 3) * ld + 3 * cb + t_dof[b] % 3, lam * t_val[a] * t_val[b]);
  }
}

void launch_dense_add_terms(int nterms, const int* t_ptr, const int* t_dof, const double* t_val, const double* t_lam,
                            const int* cmap, double* M, int ld, cudaStream_t s) {
  if (nterms > 0) k_dense_add_terms<<<nterms, kThreads, 0, s>>>(t_ptr, t_dof, t_val, t_lam, cmap, M, ld); note_launch();
}

void launch_dense_add_entries(int nent, const int* rdof, const int* cdof, const double* val, const int* cmap,
                              double* M, int ld, cudaStream_t s) {
  if (nent > 0) k_dense_add_entries<<<div_up(nent, kThreads), kThreads, 0, s>>>(nent, rdof, cdof, val, cmap, M, ld); note_launch();
}

int dense_ld(int nd) { return div_up(nd, SB) * SB; }

int launch_dense_invert(double* M, int nd, double* scratch, int* status, cudaStream_t s) {
  const int ld = dense_ld(nd), nt = ld / SB;
  const int smem = 2 * SB * SB * (int)sizeof(double);
  FEB_TRY(set_dyn_smem((const void*)k_sweep_update, smem));
  k_symmetrize<<<dim3(nt, nt), 256, 0, s>>>(M, nd, ld); note_launch();
  double* Dinv = scratch;
  double* CT = scratch + SB * SB;
  double* WT = CT + (size_t)SB * ld;
  k_sweep_first<<<1, 256, 0, s>>>(M, ld, Dinv, status); note_launch();
  for (int k = 0; k < nt; ++k) {
    k_sweep_panel<<<dim3(nt, SB / 16), 256, 0, s>>>(M, ld, k, Dinv, CT, WT); note_launch();
    if (nt > 1) { k_sweep_update<<<nt * (nt - 1) / 2, 256, smem, s>>>(M, ld, k, CT, WT, Dinv, status); note_launch(); }
  }
  k_mirror<<<dim3(nt, nt), 256, 0, s>>>(M, ld); note_launch();
  return FEB_OK;
}

size_t dense_scratch_doubles(int nd) { return (size_t)SB * SB + 2 * (size_t)SB * dense_ld(nd); }

// Two rows a warp once one row a warp fills every SM twice (16 rows a block, 148 SMs): fewer gathers of b a row.
template <typename T>
void launch_dense_solve(const double* Minv, int nd, const int* klist, const int* cmap, int64_t n, const T* b, T* x,
                        const int* skip, cudaStream_t s) {
  const int ld = dense_ld(nd), zero = div_up(3 * n, 256);
  if (nd > 2 * 8 * kSmCount) {
    const int brows = div_up(nd, 16);
    k_dense_solve<T, 2><<<brows + zero, 256, 0, s>>>(Minv, nd, ld, klist, cmap, n, b, x, brows, skip);
  } else {
    const int brows = div_up(nd, 8);
    k_dense_solve<T, 1><<<brows + zero, 256, 0, s>>>(Minv, nd, ld, klist, cmap, n, b, x, brows, skip);
  }
  note_launch();
}

template void launch_dense_solve<float>(const double*, int, const int*, const int*, int64_t, const float*, float*,
                                        const int*, cudaStream_t);
template void launch_dense_solve<double>(const double*, int, const int*, const int*, int64_t, const double*, double*,
                                         const int*, cudaStream_t);

}  // namespace feb
