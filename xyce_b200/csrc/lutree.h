// Elimination-tree plan of the sparse LU refactorization and of its triangular solves (internal to
// the library).
//
// The pivots of P A Q form a tree: pivot k's updates reach only rows and columns of its front
// struct(k) (the rows of L's column k and the columns of U's row k, closed under elimination), all
// of which are ancestors of k. Two facts about circuit factors shape the plan:
//   * the tree is a wide forest of small subtrees under a few long paths. At 200k unknowns (the
//     placed 100k-MOSFET netlist) 4,212 subtrees of at most 40 levels hang off 56 paths, the
//     longest of 2,888 pivots, in frames of 35 to 71 slots;
//   * a few pivots (a supply's branch equation and current) have an empty row of U or an empty
//     column of L and so make no updates, however long their other side is; their adjacency must
//     not be counted as a front (the rail's 90k-entry row would make one front of 90k variables).
// So the pivots are split in two: the BOTTOM subtrees, of at most kTopWork updates each, are spread
// over thread blocks that walk their levels independently; the TOP pivots are eliminated path by
// path ("chains"), one thread block per chain, with the front held densely in shared memory
// (lutree.cu). A matrix whose structure does not fit (frame over kMaxFrame, fill of the symmetrised
// pattern, an update-free pivot that others wait for) has no plan, and the level-by-level
// kernels of lu.cu and sptrsv.cu take it.
#pragma once

#include <vector>

struct XdPos2 { int x, y; };
struct XdPos4 { int x, y, z, w; };

constexpr int kMaxFrame = 128;       // largest frame (slots) of a chain
constexpr int kJoinNone = 255;       // a parent slot the child chain has no variable for
constexpr int kBlockPivots = 8;      // pivots a chain eliminates at a time
constexpr int kBlockInts = 12;       // a block's record: its pivots' slots (kNoPivot past the last), the
                                     // frame's live slots, the first and last child chain that joins
constexpr int kNoPivot = (int)0x80000000;
constexpr int kLongPairs = 32;       // updates of a bottom destination that a thread takes; more: a warp
#ifdef __CUDACC__
#define XD_TREE_FN __host__ __device__
#else
#define XD_TREE_FN
#endif
// Values per block of top pivots in V.
XD_TREE_FN constexpr long long xd_panel_size(int F) { return 2LL * kBlockPivots * F + kBlockPivots * kBlockPivots; }

// The bottom rows' sums of a triangular solve, as passes of a thread block: a pass is at most
// kPassThreads / lanes rows of one level, `lanes` threads each; the entries of a pass sit in the
// order its threads read them (round k, thread i at off + k * rows * lanes + i; absent ones have
// column -1 and value 0), so a pass reads its columns and values in whole lines and needs no row
// pointers.
constexpr int kPassThreads = 512;
struct XdPasses {
  std::vector<int> gptr;             // group g's passes [gptr[g], gptr[g + 1])
  std::vector<XdPos4> pass;          // (first row in rows, rows | log2 lanes << 16 | last of its level << 24, off, rounds)
  std::vector<int> rows;             // positions in order
  std::vector<int> col;              // column (position in order) of each entry slot, or -1
};

// Host side of the plan. Values live in one array V: the bottom rows' strict-lower entries by forward
// pass, the top rows' strict-lower entries outside the panels row by row, the bottom rows' upper
// entries by backward pass, the entries of rows that are solved last, bottom diagonals, and then per
// block of top pivots a dense panel of 2 * kBlockPivots * F values, the pivots' U rows by column slot
// (a pivot at its own slot) and their L columns by row slot, and the block's kBlockPivots x
// kBlockPivots diagonal part once more with the pivots' reciprocals on its diagonal.
struct XdTreePlan {
  int n = 0, F = 0;                  // F: slots of a frame, a multiple of 16
  int nbot = 0, ntop = 0;
  std::vector<int> order;            // [n] bottom rows by (group, level, index), then top rows by panel
  XdPasses fwd, bwd;
  std::vector<int> lptr, lcol;       // top rows' lower entries outside the panels
  std::vector<int> tail;             // positions in order of the rows that are solved last
  std::vector<int> tptr, tcol;       // their upper entries outside the panels
  int l0 = 0, u0 = 0, t0 = 0, d0 = 0, p0 = 0;  // V offsets: top rows, backward passes, last rows, diagonals, panels
  long long nv = 0;                  // length of V
  std::vector<int> pos;              // [nnz of M] position in V of each entry of M
  std::vector<int> diag;             // [n] position in V of each pivot
  // Bottom groups: group g has levels [glev[g], glev[g + 1]); level l its rows order[lrow[l] ..
  // lrow[l + 1]), its divisions and its update destinations.
  int ngroups = 0;
  std::vector<int> glev, lrow, ldiv, ldst;
  std::vector<int> llong;            // [levels] the first of a level's destinations with more than kLongPairs updates
  bool any_long = false;
  std::vector<XdPos2> div;           // (position of L(i, k), position of U(k, k))
  std::vector<XdPos4> dst, pairs;    // as in lu.cu: one update inline, or a range of pairs
  // Updates of top entries by bottom pivots: destination sdst[d], pairs (L, U) sptr[d] .. sptr[d + 1].
  std::vector<int> sdst, sptr;
  std::vector<XdPos2> spairs;
  std::vector<XdPos2> tdiv;          // divisions of top pivots' entries outside their panels
  // Chains, children before parents: chain c has panels [cptr[c], cptr[c + 1]), eliminated in blocks
  // of kBlockPivots from the first: blocks [bptr[c], bptr[c + 1]), records in blocks. A variable has
  // a slot from the first block whose pivots' fronts hold it to its own block.
  int nchains = 0;
  std::vector<int> cptr, bptr, blocks;
  std::vector<int> jchild;           // child chains in the order they join
  std::vector<unsigned char> jmap;   // [nchains * F] a chain's slot of each slot of its parent, or kJoinNone
  std::vector<int> border;           // [nchains * F] position in order of the variable left in each slot, or -1
};

// Builds the plan of M = L - I + U (CSR, columns ascending, closed under elimination; diag[k] the
// position of the pivot). Returns false when the structure does not fit.
bool xd_tree_plan(int n, const std::vector<int> &mp, const std::vector<int> &mi, const std::vector<int> &mdiag,
                  XdTreePlan *plan);

// ---- device side (lutree.cu) ---------------------------------------------------------------------
#include <cuda_runtime.h>

struct XdTree {
  bool on = false;                   // the matrix has a plan
  bool divide = false;               // V's chain pivots are divided by (their diagonal parts hold no reciprocals)
  int n = 0, F = 0, ntop = 0, ngroups = 0, nchains = 0, nsd = 0, ntdiv = 0, p0 = 0;
  long long nv = 0;
  double *d_v = nullptr;             // V
  int *d_diag = nullptr;             // [n]
  int *d_glev = nullptr, *d_ldiv = nullptr, *d_ldst = nullptr;
  int *d_llong = nullptr;            // null: no destination has more than kLongPairs updates
  int2 *d_div = nullptr;
  int4 *d_dst = nullptr, *d_pairs = nullptr;
  int *d_gptr = nullptr, *d_gpos = nullptr;  // the bottom groups' entries (positions in V) in shared memory
  size_t bottom_smem = 0;
  int *d_sdst = nullptr, *d_sptr = nullptr;
  int2 *d_spairs = nullptr, *d_tdiv = nullptr;
  int *d_cptr = nullptr, *d_bptr = nullptr, *d_blocks = nullptr, *d_jchild = nullptr;
  unsigned char *d_jmap = nullptr;
  double *d_jbuf = nullptr;          // [nchains][F * F] the fronts that chains hand to their parents
  int *d_ctl = nullptr;              // the words below; zeroed by each call
  // Solves: rows by position in the plan's order.
  int nbot = 0, ntail = 0, nchunk = 0, l0 = 0, u0 = 0, t0 = 0, d0 = 0;
  struct Passes {
    int *gptr = nullptr, *rows = nullptr, *col = nullptr;
    int4 *pass = nullptr;
  } d_fwd, d_bwd;
  int *d_grow = nullptr;             // [ngroups + 1] first row of each group
  size_t pass_smem = 0;
  bool schur_long = false, row_long = false, pass_long[2] = {};  // lists that a block takes (lutree.cu)
  int *d_lptr = nullptr, *d_lcol = nullptr, *d_tcol = nullptr;
  int4 *d_chunk = nullptr;           // chunks of the rows solved last: (row, first entry, end, chunk of the row)
  int4 *d_tail = nullptr;            // those rows: (position in order, V position of its pivot, first chunk, chunks)
  int *d_bsrc = nullptr;             // [n] right-hand side index of each row
  int *d_xdst = nullptr;             // [n] solution index, ~index for a row solved last
  int *d_joined = nullptr, *d_border = nullptr;  // whether a chain has a parent; its border's rows
  double *d_y = nullptr, *d_x = nullptr;  // [n] forward and backward solved values
  double *d_wbuf = nullptr;          // [nchains][F] the sums that chains hand to their parents
  double *d_part = nullptr;          // [nchunk]
  int *d_sctl = nullptr;             // tickets, chain flags of both directions, finished chunks per last row
};

// p, q as in (P A Q)[i][j] = A[P[i]][Q[j]].
int xd_tree_upload(XdTree *t, const XdTreePlan &plan, const int *p, const int *q);
void xd_tree_free(XdTree *t);
// Eliminates V (holding P A Q, zeros elsewhere) in place; kTreeInfo of d_ctl holds n - k for the first
// zero pivot k (0: none), kTreeExpired is nonzero when a wait between chains gave up, kTreeOdd when a
// chain met a pivot whose reciprocal is not a normal number: without t->divide the factors are then
// not to be used. (Then the chains' ticket, and a flag for each.)
constexpr int kTreeInfo = 0, kTreeExpired = 1, kTreeOdd = 2, kTreeTicket = 3, kTreeFlags = 4;
int xd_tree_factor(XdTree *t, cudaStream_t st);
// Solves A x = b in place in d_x with V's factors. Stream-ordered.
int xd_tree_solve(XdTree *t, double *d_x, cudaStream_t st);
