// Dense coarsest level (see dense.cu).
#pragma once
#include "common.cuh"
#include <algorithm>

namespace feb {

// Leading dimension of the dense matrix of nd dofs (whole 64-wide tiles); the assembly calls take it as `ld`.
int dense_ld(int nd);
void launch_dense_from_stencil(const double* A, int nx, int ny, int nz, const int* cmap, double* M, int ld,
                               cudaStream_t s);
void launch_dense_add_terms(int nterms, const int* t_ptr, const int* t_dof, const double* t_val, const double* t_lam,
                            const int* cmap, double* M, int ld, cudaStream_t s);
void launch_dense_add_entries(int nent, const int* rdof, const int* cdof, const double* val, const int* cmap,
                              double* M, int ld, cudaStream_t s);
// Lower tiles of M <- -M^-1 in place (symmetrised first; dense_ld(nd) rows of dense_ld(nd) values, identity past nd);
// scratch: dense_scratch_doubles(nd); *status = FEB_ERR_COARSE on a non-positive pivot.
int launch_dense_invert(double* M, int nd, double* scratch, int* status, cudaStream_t s);
size_t dense_scratch_doubles(int nd);
// x = -S b on the kept nodes, S from launch_dense_invert (klist: node of compact index, cmap: compact index of node or -1; x
// is zeroed on the other nodes), one launch.  part: dense_part_doubles(nd) of work space; arrived: dense_tiles(nd) counters,
// zero before the first call and after every one.  Calls that share them have to follow one another on one stream.
template <typename T>
void launch_dense_solve(const double* S, int nd, const int* klist, const int* cmap, int64_t n, const T* b, T* x, double* part,
                        int* arrived, const int* skip, cudaStream_t s);
size_t dense_part_doubles(int nd);
int dense_tiles(int nd);

}  // namespace feb
