// Coarsest multigrid level: dense FP64 matrix over the kept dofs, explicit inverse by a blocked symmetric
// sweep over its lower tiles (symmetric positive definite, no pivoting), applied as a GEMV in every V-cycle.
// The reference factorises the same matrix (SciPy splu, fe/gmg.py:102; cuSOLVER Cholesky,
// rb/gpusolve.py:138-161); an explicit inverse turns the per-V-cycle solve into one coalesced GEMV.
#include "dense.cuh"

#include <cfloat>

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

// Symmetric sweep of a 64 x 64 block held 4 x 4 per thread (rows 4 ty + u, columns 4 tx + v): step p turns
// a_pp = d into -1/d, a_ip and a_pi into a_ip / d and a_ij into a_ij - a_ip a_pj / d; after all steps the block is
// minus its inverse.  Row p travels through a double-buffered line of shared memory (its column is the same numbers by
// symmetry), so a step costs one barrier; the line also carries the next diagonal value before the step, so that
// every thread forms the next pivot and its reciprocal while the step's update runs.  A non-positive pivot sets
// *status and counts as 1.
__device__ __forceinline__ double pivot_inverse(double d, bool& bad) {
  const bool ok = d > 0.0 && d <= DBL_MAX;
  bad |= !ok;
  return 1.0 / (ok ? d : 1.0);
}

__device__ __forceinline__ void sweep_block(double (&a)[4][4], double (*line)[SB + 2], int ty, int tx, int* status) {
  double ip = 0.0;
  bool bad = false;
#pragma unroll 1
  for (int pb = 0; pb < SB / 4; ++pb) {
#pragma unroll
    for (int pu = 0; pu < 4; ++pu) {
      const int p = 4 * pb + pu;
      double* row = line[pu & 1];
      if (ty == pb) {
        *reinterpret_cast<double2*>(row + 4 * tx) = make_double2(a[pu][0], a[pu][1]);
        *reinterpret_cast<double2*>(row + 4 * tx + 2) = make_double2(a[pu][2], a[pu][3]);
      }
      const int nb = pu < 3 ? pb : pb + 1;
      if (ty == nb && tx == nb) row[SB] = a[(pu + 1) & 3][(pu + 1) & 3];
      __syncthreads();
      if (p == 0) ip = pivot_inverse(row[0], bad);
      double ci[4], cj[4];
#pragma unroll
      for (int u = 0; u < 4; u += 2) {
        const double2 x = *reinterpret_cast<const double2*>(row + 4 * ty + u);
        const double2 y = *reinterpret_cast<const double2*>(row + 4 * tx + u);
        ci[u] = x.x * ip; ci[u + 1] = x.y * ip; cj[u] = y.x; cj[u + 1] = y.y;
      }
      double next = 1.0;
      if (p + 1 < SB) {
        const double c = row[p + 1];
        next = pivot_inverse(row[SB] - c * ip * c, bad);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) a[u][v] -= ci[u] * cj[v];
      if (ty == pb) {
#pragma unroll
        for (int v = 0; v < 4; ++v) a[pu][v] = cj[v] * ip;
      }
      if (tx == pb) {
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u][pu] = ci[u];
        if (ty == pb) a[pu][pu] = -ip;
      }
      ip = next;
    }
  }
  if (bad && threadIdx.x == 0) atomicExch(status, FEB_ERR_COARSE);
}

// Dinv = inverse of the first pivot block.
__global__ void __launch_bounds__(256)
k_sweep_first(const double* __restrict__ M, int ld, double* __restrict__ Dinv, int* __restrict__ status) {
  __shared__ __align__(16) double line[2][SB + 2];
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

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Pivot panel of step k: C_i = S_ik (from the lower triangle: S_ki^T for i < k), W_i = C_i Dinv; S_ik <- W_i,
// S_kk <- -Dinv.  -C and W are left transposed (k-major rows of length ld), as the update's operands.  A CTA takes
// 16 rows of block row i: at 64 rows a CTA the panel would use a third of the SMs.
__global__ void __launch_bounds__(256)
k_sweep_panel(double* __restrict__ M, int ld, int k, const double* __restrict__ Dinv, double* __restrict__ CT,
              double* __restrict__ WT) {
  __shared__ __align__(16) double Ds[SB][SB];
  __shared__ __align__(16) double Cs[SB][16];     // C_i^T
  const int i = blockIdx.x, r0 = 16 * blockIdx.y, t = threadIdx.x;
  const int row = i * SB + r0, kc = k * SB;
  if (i == k) {
#pragma unroll
    for (int e = t; e < 16 * SB; e += 256) M[(size_t)(row + e / SB) * ld + kc + e % SB] = -Dinv[(r0 + e / SB) * SB + e % SB];
    return;
  }
#pragma unroll
  for (int e = t; e < SB * SB / 2; e += 256) cp_async16(&Ds[0][0] + 2 * e, Dinv + 2 * e);
  if (i > k) {
    double2 v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + 256 * h;
      v[h] = *reinterpret_cast<const double2*>(M + (size_t)(row + e / 32) * ld + kc + 2 * (e % 32));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = t + 256 * h;
      Cs[2 * (e % 32)][e / 32] = v[h].x;
      Cs[2 * (e % 32) + 1][e / 32] = v[h].y;
    }
  } else {
#pragma unroll
    for (int e = t; e < 8 * SB; e += 256) cp_async16(&Cs[e / 8][2 * (e % 8)], M + (size_t)(kc + e / 8) * ld + row + 2 * (e % 8));
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int e = t; e < 8 * SB; e += 256)
    {
    const double2 x = *reinterpret_cast<const double2*>(&Cs[e / 8][2 * (e % 8)]);
    *reinterpret_cast<double2*>(CT + (size_t)(e / 8) * ld + row + 2 * (e % 8)) = make_double2(-x.x, -x.y);
  }
  // thread: row r, columns c .. c + 3 of W_i
  const int r = t & 15, c = (t >> 4) * 4;
  double w[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 16
  for (int q = 0; q < SB; ++q) {
    const double x = Cs[q][r];
    const double2 d0 = *reinterpret_cast<const double2*>(&Ds[q][c]), d1 = *reinterpret_cast<const double2*>(&Ds[q][c + 2]);
    w[0] += x * d0.x; w[1] += x * d0.y; w[2] += x * d1.x; w[3] += x * d1.y;
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) WT[(size_t)(c + v) * ld + row + r] = w[v];
  if (i < k) {
#pragma unroll
    for (int v = 0; v < 4; ++v) M[(size_t)(kc + c + v) * ld + row + r] = w[v];
  } else {
    double2* p = reinterpret_cast<double2*>(M + (size_t)(row + r) * ld + kc + c);
    p[0] = make_double2(w[0], w[1]);
    p[1] = make_double2(w[2], w[3]);
  }
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Step k's update of the lower tiles outside the pivot panel: S_ij -= C_i W_j^T (64 x 64 x 64 a CTA, 32 x 16 a
// warp).  The FP64 matrix instruction has the scalar FMA's rate (64 a clock and SM) but needs a sixth of its operand
// reads from shared memory, which bounded the scalar form (4 x 4 a thread: 12 TFLOP/s of 37).  The CTA of the next
// pivot block (block 0, so that it starts first) inverts it on the spot: the serial part of the sweep runs beside
// the other tiles instead of between two steps.
constexpr int ULD = SB + 8;   // operand pitch: the four k rows of a fragment fall on both halves of the banks

__global__ void __launch_bounds__(256)
k_sweep_update(double* __restrict__ M, int ld, int k, const double* __restrict__ CT, const double* __restrict__ WT,
               double* __restrict__ Dinv, int* __restrict__ status) {
  extern __shared__ __align__(16) double sm[];
  double (*As)[ULD] = reinterpret_cast<double (*)[ULD]>(sm);
  double (*Bs)[ULD] = reinterpret_cast<double (*)[ULD]>(sm + SB * ULD);
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
#pragma unroll
  for (int e = t; e < SB * SB / 2; e += 256) {
    const int q = e / (SB / 2), c = 2 * (e % (SB / 2));
    cp_async16(&As[q][c], CT + (size_t)q * ld + i0 + c);
    cp_async16(&Bs[q][c], WT + (size_t)q * ld + j0 + c);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  const int lane = t & 31, w = t >> 5;
  const int r = 32 * (w >> 2) + (lane >> 2), c = 16 * (w & 3) + 2 * (lane & 3);   // first row, column pair held
  double s[4][2][2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const double2 x = *reinterpret_cast<const double2*>(M + (size_t)(i0 + r + 8 * u) * ld + j0 + c + 8 * v);
      s[u][v][0] = x.x;
      s[u][v][1] = x.y;
    }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  const double* Ap = &As[lane & 3][32 * (w >> 2) + (lane >> 2)];
  const double* Bp = &Bs[lane & 3][16 * (w & 3) + (lane >> 2)];
#pragma unroll 4
  for (int q = 0; q < SB; q += 4) {
    double av[4], bv[2];
#pragma unroll
    for (int u = 0; u < 4; ++u) av[u] = Ap[q * ULD + 8 * u];
#pragma unroll
    for (int v = 0; v < 2; ++v) bv[v] = Bp[q * ULD + 8 * v];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) dmma(s[u][v], av[u], bv[v]);
  }
  if (has_next && blockIdx.x == 0) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v)
        *reinterpret_cast<double2*>(&As[r + 8 * u][c + 8 * v]) = make_double2(s[u][v][0], s[u][v][1]);
    __syncthreads();
    const int ty = t >> 4, tx = t & 15;
    double d[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) d[u][v] = As[4 * ty + u][4 * tx + v];
    sweep_block(d, reinterpret_cast<double (*)[SB + 2]>(&Bs[0][0]), ty, tx, status);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) Dinv[(4 * ty + u) * SB + 4 * tx + v] = -d[u][v];
    return;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v)
      *reinterpret_cast<double2*>(M + (size_t)(i0 + r + 8 * u) * ld + j0 + c + 8 * v) =
          make_double2(s[u][v][0], s[u][v][1]);
}

// x = -S b on the coarsest level in one launch, S the swept matrix (minus the inverse), of which the lower tiles are read:
// block (ti, tj) multiplies its 64 x 64 tile with b_tj and, off the diagonal, its transpose with b_ti, and leaves the two
// partial vectors in slots of its own; the last block to arrive at a block row adds the row's slots in their order.  The
// blocks after the tiles zero the entries of nodes outside the dense system (cmap < 0), a disjoint set.  A block has its
// tile on the way (eight 16-byte loads a thread) before it gathers the 128 values of b.
// Bound by reading the tiles, and by gather and arrivals where those come from L2.  With all of S read, a row a warp:
// 3510 dofs in a solve 21.7 -> 17.0 us, 2457 dofs between level-0 sweeps (from memory) 23.0 -> 14.0 us, alone and from L2
// 9.4 -> 10.4 us.  Runs of tiles with a sum a run, the next tile on its way, were slower (13 us; 5265 dofs 45 against 32).
template <typename T>
__global__ void __launch_bounds__(256)
k_dense_solve(const double* __restrict__ S, int nd, int ld, const int* __restrict__ klist, const int* __restrict__ cmap,
              int64_t n, const T* __restrict__ b, T* __restrict__ x, int tiles, double* part, int* arrived,
              const int* __restrict__ skip) {
  if (skip && *skip) return;
  if ((int)blockIdx.x >= tiles) {
    const int64_t e = (int64_t)(blockIdx.x - tiles) * blockDim.x + threadIdx.x;
    if (e < 3 * n && cmap[e / 3] < 0) x[e] = T(0);
    return;
  }
  __shared__ double xb[2][SB];                   // b_ti, b_tj
  __shared__ __align__(16) double col[8][SB];
  __shared__ int last[2];
  const int nt = ld / SB, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int ti = (int)((sqrtf(8.f * (float)blockIdx.x + 1.f) - 1.f) * 0.5f);
  while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
  const int tj = blockIdx.x - ti * (ti + 1) / 2;
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
    v[r] = reinterpret_cast<const double2*>(S + (size_t)(ti * SB + 8 * w + r) * ld + tj * SB)[lane];
  if (threadIdx.x < 2 * SB) {
    const int h = threadIdx.x / SB, q = (h ? tj : ti) * SB + threadIdx.x % SB, qc = min(q, nd - 1);
    const double bq = double(b[3 * (int64_t)klist[qc / 3] + qc % 3]);
    xb[h][threadIdx.x % SB] = q < nd ? bq : 0.0;
  }
  __syncthreads();
  const double x0 = xb[1][2 * lane], x1 = xb[1][2 * lane + 1];
  double p[8], c0 = 0.0, c1 = 0.0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const double xr = xb[0][8 * w + r];
    p[r] = v[r].x * x0 + v[r].y * x1;
    c0 += v[r].x * xr;
    c1 += v[r].y * xr;
  }
  reinterpret_cast<double2*>(col[w])[lane] = make_double2(c0, c1);
  // sums over the lanes of eight rows at once: after the exchanges lane l holds row 4 (l >> 4 & 1) + 2 (l >> 3 & 1) + (l >> 2 & 1)
#pragma unroll
  for (int h = 4, m = 16; h >= 1; h >>= 1, m >>= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int r = 0; r < h; ++r) {
      const double give = up ? p[r] : p[h + r], keep = up ? p[h + r] : p[r];
      p[r] = keep + __shfl_xor_sync(0xffffffffu, give, m);
    }
  }
  p[0] += __shfl_xor_sync(0xffffffffu, p[0], 2);
  p[0] += __shfl_xor_sync(0xffffffffu, p[0], 1);
  if ((lane & 3) == 0)
    part[((size_t)ti * nt + tj) * SB + 8 * w + 4 * (lane >> 4) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1)] = p[0];
  __syncthreads();
  if (ti != tj && threadIdx.x < SB) {
    double c = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) c += col[q][threadIdx.x];
    part[((size_t)tj * nt + ti) * SB + threadIdx.x] = c;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    const int row = threadIdx.x ? tj : ti;
    const bool mine = threadIdx.x == 0 || ti != tj;
    __threadfence();                             // the block's slots before its arrival, and the others' after the last one
    const bool done = mine && atomicAdd(arrived + row, 1) == nt - 1;
    if (done) arrived[row] = 0;                  // for the next launch
    __threadfence();
    last[threadIdx.x] = done;
  }
  __syncthreads();
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    if (!last[h]) continue;
    const int row = h ? tj : ti, r = threadIdx.x & (SB - 1), g = threadIdx.x / SB;
    double a = 0.0;
    const double* q = part + (size_t)row * nt * SB + r;
#pragma unroll 8
    for (int t = g; t < nt; t += 4) a += __ldcg(q + (size_t)t * SB);
    __syncthreads();                             // col is read
    col[g][r] = a;
    __syncthreads();
    const int d = row * SB + r;
    if (g == 0 && d < nd)
      x[3 * (int64_t)klist[d / 3] + d % 3] = T(-((col[0][r] + col[1][r]) + (col[2][r] + col[3][r])));
  }
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

// Two launches a step.  1890 / 2457 / 3510 / 5265 dofs take 0.86 / 1.42 / 2.5 / 6.7 ms; an update takes 72 us at 5265 dofs
// (25 TFLOP/s), and below about 3000 dofs the next pivot's chain of divisions (20 us) bounds it.  With 32-wide pivot
// blocks over the whole matrix and five launches a step the inverse of 3510 dofs took 13.9 ms and that of 2457 6.3 ms.
int launch_dense_invert(double* M, int nd, double* scratch, int* status, cudaStream_t s) {
  const int ld = dense_ld(nd), nt = ld / SB;
  const int smem = 2 * SB * ULD * (int)sizeof(double);
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
  return FEB_OK;
}

size_t dense_scratch_doubles(int nd) { return (size_t)SB * SB + 2 * (size_t)SB * dense_ld(nd); }

size_t dense_part_doubles(int nd) { const size_t nt = dense_ld(nd) / SB; return nt * nt * SB; }
int dense_tiles(int nd) { return dense_ld(nd) / SB; }

template <typename T>
void launch_dense_solve(const double* S, int nd, const int* klist, const int* cmap, int64_t n, const T* b, T* x, double* part,
                        int* arrived, const int* skip, cudaStream_t s) {
  const int nt = dense_tiles(nd), tiles = nt * (nt + 1) / 2;
  k_dense_solve<T><<<tiles + div_up(3 * n, 256), 256, 0, s>>>(S, nd, dense_ld(nd), klist, cmap, n, b, x, tiles, part, arrived,
                                                             skip);
  note_launch();
}

template void launch_dense_solve<float>(const double*, int, const int*, const int*, int64_t, const float*, float*, double*,
                                        int*, const int*, cudaStream_t);
template void launch_dense_solve<double>(const double*, int, const int*, const int*, int64_t, const double*, double*, double*,
                                         int*, const int*, cudaStream_t);

}  // namespace feb
