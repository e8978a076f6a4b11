// One part of the column-first transforms: the kernels or device functions of one
// class of lengths and one precision (JRG_PART_*, set by the build), so that the
// unrolled line transforms compile in parallel.
#define JRG_CAT2(a, b) a##b
#define JRG_CAT(a, b) JRG_CAT2(a, b)
#include "k_cols.cuh"
#include "k_cube.cuh"
#define SIZES JRG_CAT(JRG_COLS_SIZES_, JRG_PART_CLASS)

namespace jrg {
namespace cols {
using R = JRG_PART_REAL;
using C = C_t<R>;
#if JRG_PART_KIND == 0
#define INST(N) template int run_columns<R, N>(const jrg_plan*, int, const fast::Args&, cudaStream_t);
#elif JRG_PART_KIND == 1
#define INST(N) template __device__ void y_inverse<C, N>(Tile<C>); template __device__ void y_forward<C, N>(Tile<C>);
#elif JRG_PART_KIND == 2
#define INST(N) template __device__ void z_apply<C, N>(Tile<C>, int, int, int, int);
#elif JRG_PART_KIND == 4
#define INST(N) template int run_cube<R, N>(const jrg_plan*, int, const fast::Args&, cudaStream_t);
#else
#define INST(N) template __device__ void z_density<C, N>(Tile<C>, int, int, int, int, int);
#endif
SIZES(INST)
}  // namespace cols
}  // namespace jrg
