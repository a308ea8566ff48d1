// Plan of the nested subspace products (internal interface of libsgpp_gb300): host part, plain C++.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <string>
#include <vector>

namespace sgmev {

// A subspace (level vector l) is a node of a tree: its active dimensions are those with l_t > 1, in
// ascending order, and its parent is the subspace without its last active dimension. The factor of
// (t, l) at a data point is entry e of the point's table,
//     tab[e][j] = h_l(x_t) / h_1(x_t)   (ModLinear: h_l(x_t)),  tab[0][j] = prod_t h_1(x_t)  (1)
// and the point's cell in dimension t at level l is xcell[t][j] >> (finest level's bits - (l - 1)).
// A factor is packed into an int: e (10 bits), t (5), l - 1 (5), the shift of xcell (5).
#ifdef __CUDACC__
#define NEST_HD __host__ __device__
#else
#define NEST_HD
#endif
NEST_HD constexpr int fac_e(int f) { return f & 1023; }
NEST_HD constexpr int fac_t(int f) { return (f >> 10) & 31; }
NEST_HD constexpr int fac_k(int f) { return (f >> 15) & 31; }
NEST_HD constexpr int fac_shift(int f) { return (f >> 20) & 31; }
constexpr int make_fac(int e, int t, int k, int shift) {
  return e | (t << 10) | (k << 15) | (shift << 20);
}
constexpr int kFacH1 = make_fac(0, 0, 0, 31);  // entry 0; a shift of 31 gives cell 0

struct alignas(8) NestOp2 { int x, y; };
struct alignas(16) NestOp4 { int x, y, z, w; };

constexpr int kNestMultThreads = 64;  // points per CTA of the mult
constexpr int kNestTile = 32;         // points per tile of the multTranspose (a warp's lanes)
constexpr int kNestSplits = 16;       // most CTAs that share the groups of one tile of points
constexpr size_t kNestSmem = 200 * 1024;
constexpr size_t kNestAccBudget = 64 * 1024;  // cell sums of a multTranspose CTA (two CTAs per SM)

// shared memory of a multTranspose CTA behind its [cells][threads] sums: per point of the tile the
// inner products, the table row (with a 1 behind it), the inner cells and the coordinates' cells; odd
// row lengths keep a warp's 32 points in different banks
struct NestTileLayout {
  int qs, es, cs, xs;  // row lengths: doubles, doubles, uint16, uint32
  NEST_HD NestTileLayout(int nq, int n_ent, int dim)
      : qs(nq | 1), es((n_ent + 1) | 1), cs(((nq + 1) / 2 | 1) * 2), xs(dim | 1) {}
  NEST_HD size_t bytes() const {
    return static_cast<size_t>(kNestTile) * (8 * qs + 8 * es + 2 * cs + 4 * xs);
  }
};

// multTranspose launches: chunks of one block size
struct NestClass {
  int threads = 0;  // subspaces per chunk, one per thread
  int cells = 0;    // most cells of a subspace
  int chunk_begin = 0, chunks = 0;
  int nq = 0;       // most inner nodes of a chunk
  size_t smem = 0;
  int64_t row_begin = 0, row_len = 0;  // positions of the class in the transposed layout
  int streams = 0;  // tile streams (rows of partial sums)
};

struct NestTables {
  int dim = 0, n_sub = 0, n_ent = 0;
  int64_t n = 0;
  std::vector<int> lmax;  // [dim] finest level per dimension
  // mult: groups (first and end inner node, first and end factor of the group's product), inner
  // nodes (position or -1, first and end leaf, factor) and leaves (position, factor)
  std::vector<NestOp4> rops, qops;
  std::vector<NestOp2> lops;
  std::vector<int> facs;
  std::vector<int> cuts;  // row s - 1 of kNestSplits + 1: boundaries of the groups among s CTAs
  std::vector<int> inv;   // grid point of a position or -1
  // multTranspose: chunks (first inner node, inner nodes, first depth boundary, depths), their inner
  // nodes (local parent, factor), depth boundaries, subspaces by thread (local parent, factor) and
  // their cell counts (0: none), grid point of a transposed position
  std::vector<NestClass> classes;
  std::vector<NestOp4> chunks;
  std::vector<NestOp2> cq, cs;
  std::vector<int> clev, ccell, tinv;
};

// False (and a reason) when the grid is not one that the kernels take: dim <= 32, levels up to 20, at
// most 512 cells per subspace (multTranspose keeps them in shared memory), a table row and a chunk
// that fit shared memory.
bool nest_plan(NestTables* p, int dim, int64_t n, const double* level_pow2, const double* index,
               std::string* err);

}  // namespace sgmev
