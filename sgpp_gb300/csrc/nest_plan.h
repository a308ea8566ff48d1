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

// The mult evaluates three common kinds of subtrees whole, with the factors of levels 2 and 3 in
// registers. For runs and trees, per cell of a node whose last active dimension is t, with k = dim - 1 - t dimensions
// after it, the coefficients lie in one row:
//   run  (the node and its level-2 leaves): the node, then the two cells of the leaf of dimension
//        t' at 1 + 2 (dim - 1 - t')
//   tree (the node, its level-2 children with their runs, its level-3 leaves): the node, then per
//        dimension t' from the last to the first, at nest_tree_at(dim - 1 - t'), the two run rows
//        of the level-2 child and the four cells of the level-3 leaf
// A section's place does not depend on t. Run rows are 2 mod 4 long and tree rows 4 mod 8: a warp's
// gathers at one place of a tree (row c, run row b, cell b': c rows + b run rows + b') then hit
// different banks for up to 8 rows (odd lengths gave 1.9 wavefronts a gather on the regression
// workload's grid).
NEST_HD constexpr int nest_run_row(int k) { return 2 * k + (k % 2 == 0 ? 2 : 4); }
NEST_HD constexpr int nest_tree_at(int k) {
  int r = 4;
  for (int i = 0; i < k; ++i) r += 2 * nest_run_row(i) + 4;
  return r;
}
NEST_HD constexpr int nest_tree_row(int k) { return (nest_tree_at(k) + 3) / 8 * 8 + 4; }
// A forest (the node, and per later dimension t' its level-2 child with its tree, its level-3 child
// with its run and its level-4 leaf) holds the node's cells (a multiple of 4) and then, per dimension
// from the last to the first, at C nest_forest_at(dim - 1 - t') for C cells of the node: the child's
// 2 C tree rows, 4 C run rows and 8 C cells.
NEST_HD constexpr int nest_forest_step(int k) { return 2 * nest_tree_row(k) + 4 * nest_run_row(k) + 8; }
NEST_HD constexpr int nest_forest_at(int k) {
  int r = 0;
  for (int i = 0; i < k; ++i) r += nest_forest_step(i);
  return r;
}
constexpr int kNestMacroDim = 16;
constexpr int kNestBlockCells = 6144;  // most coefficients of one inner node's block
constexpr int kNestLeaves = 256;       // most leaves of one inner node's record
constexpr int kNestProgram = 640;      // most words (16 bytes) of a window's program
// positions are 32-bit, and a subspace takes up to 512 of them whatever its number of grid points: 1 GB of
// coefficients in FP64 at most; and the ten lists' programs together stay below 3 GB
constexpr int64_t kNestMaxPositions = int64_t(1) << 27;
constexpr int64_t kNestMaxWords = int64_t(1) << 24;
// window lists: at most cap coefficients per window, for so many CTAs sharing a tile of points
constexpr int kNestLists = 10;
NEST_HD constexpr int nest_list_cap(int list) { return list < kNestLists / 2 ? 18432 : 6144; }
NEST_HD constexpr int nest_list_ctas(int list) { return 1 << (list % (kNestLists / 2)); }

constexpr int kNestTile = 32;         // points per tile of the multTranspose (a warp's lanes)
constexpr size_t kNestSmem = 200 * 1024;
constexpr size_t kNestMultSmem = 220 * 1024;  // the mult runs one CTA per SM
constexpr size_t kNestAccBudget = 64 * 1024;  // cell sums of a multTranspose CTA (two CTAs per SM)

// shared memory of a multTranspose CTA behind its cell sums: per point of the tile the
// inner products, the table row (with a 1 behind it), the inner cells and the coordinates' cells; odd
// row lengths keep a warp's 32 points in different banks (bytes: with values of `value` bytes)
struct NestTileLayout {
  int qs, es, cs, xs;  // row lengths: values, values, uint16, uint32
  NEST_HD NestTileLayout(int nq, int n_ent, int dim)
      : qs(nq | 1), es((n_ent + 1) | 1), cs(((nq + 1) / 2 | 1) * 2), xs(dim | 1) {}
  NEST_HD size_t bytes(int value) const {
    return static_cast<size_t>(kNestTile) * (value * (qs + es) + 2 * cs + 4 * xs);
  }
};

// multTranspose launches: chunks of one block size
struct NestClass {
  int threads = 0;  // subspaces per chunk, one per thread
  int sums = 0;     // most cell sums of a chunk
  int chunk_begin = 0, chunks = 0;
  int nq = 0;       // most inner nodes of a chunk
  size_t smem(int value, int n_ent, int dim) const {
    return static_cast<size_t>(value) * sums + NestTileLayout(nq, n_ent, dim).bytes(value);
  }
  int64_t row_begin = 0, row_len = 0;  // positions of the class in the transposed layout
};

struct NestTables {
  int dim = 0, n_sub = 0, n_ent = 0;
  int64_t n = 0;
  int64_t n_act = 0, cells = 0;  // active dimensions and cells of all subspaces
  int cmax = 0;                  // most cells of a subspace
  bool whole = false;            // one run, tree or forest is all of the grid
  std::vector<int> lmax;  // [dim] finest level per dimension
  // mult: per window list, windows (first and end word of the program, first and end position). The
  // program is a sequence of groups: a header (inner nodes, factors), the factors of the group's
  // product (four a word), and per inner node two words: position in the window or -1, leaves, -, -;
  // or for runs and trees position, -(1 + 4 (first dimension) + (0 run, 1 tree, 2 forest)), row length
  // (forest: log2 of the node's cells), -;
  // and the node's factor unpacked: e, t, l - 1, shift. Then the leaves, a word each: position,
  // e | t << 16, l - 1, shift.
  std::vector<NestOp4> windows, prog;
  std::vector<int> list_begin, list_cells, list_words;  // first window, widest, longest program
  std::vector<int> inv;   // grid point of a position or -1
  // multTranspose: chunks (first inner node, inner nodes, first depth boundary, depths), their inner
  // nodes (local parent, factor), depth boundaries, subspaces by thread (local parent, factor) and
  // their cell counts (0: none), where a warp's sums begin in shared memory and in a row (thread's
  // cell c at 32 c + lane), grid point of a transposed position
  std::vector<NestClass> classes;
  std::vector<NestOp4> chunks;
  std::vector<NestOp2> cq, cs, cwarp;
  std::vector<int> clev, ccell, tinv;
};

// False (and a reason) when the grid is not one that the kernels take: dim <= 32, levels up to 20, at
// most 512 cells per subspace (multTranspose keeps them in shared memory), a table row and a chunk
// that fit shared memory, no grid point twice, positions and words within the limits above.
bool nest_plan(NestTables* p, int dim, int64_t n, const double* level_pow2, const double* index,
               std::string* err);

}  // namespace sgmev
