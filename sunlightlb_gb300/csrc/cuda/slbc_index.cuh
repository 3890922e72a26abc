// Index arithmetic that kernels and host code share, free of CUDA types, so
// that a host compiler checks it at the ends of its ranges.
#ifndef SLBC_INDEX_CUH
#define SLBC_INDEX_CUH

#ifdef __CUDACC__
#define SLBC_HD __host__ __device__ __forceinline__
#else
#define SLBC_HD inline
#endif

namespace slbc {

// f(e) for e = first, first + step, ... below count, in 32 bits: a lattice has
// fewer than 2^31 nodes and a grid fewer than 2^31 threads, so the last e +
// step stays below 2^32 and does not wrap (in int it would, to a negative
// element, for counts within one step of 2^31).
template <typename F>
SLBC_HD void grid_turns(unsigned first, unsigned step, unsigned count, F f) {
  for (unsigned e = first; e < count; e += step) f(e);
}

// The kernels over voxels walk the grid row by row (a row: W voxels times the
// 16-byte vectors of a voxel): a block of 256 threads takes one long row or
// several short ones at a time, so a thread divides once per row instead of
// four times per vector.  I: unsigned below 2^31 rows (row + step does not
// wrap), unsigned long long above.
template <typename I>
struct RowWalk {
  I row, step;  // first row of this thread, rows between its turns
  unsigned e;   // first element in the row
};

template <typename I>
SLBC_HD RowWalk<I> row_walk(unsigned block, unsigned blocks, unsigned thread, unsigned rowlen) {
  RowWalk<I> w;
  if (rowlen >= 256) {
    w.row = block;
    w.step = blocks;
    w.e = thread;
  } else {
    const unsigned per = 256 / rowlen, sub = thread / rowlen;
    w.e = thread - sub * rowlen;
    w.row = sub < per ? (I)block * per + sub : ~(I)0;  // past every row
    w.step = (I)blocks * per;
  }
  return w;
}

// Long rows of grids that have few of them are cut into pieces of whole turns of
// a block, so that blocks enough to fill the GPU have one (pooling a grid of 2 x 2
// x 20,000 with 256 channels: 689 us with a block per row, 6.6 so).
constexpr int kRowBlocks = 152 * 16;

struct RowCut {
  unsigned cuts, piece;  // pieces per row, elements of a piece
};

SLBC_HD RowCut row_cut(unsigned long long rows, unsigned rowlen) {
  if (rowlen < 512 || rows < 1 || rows >= kRowBlocks) return {1, rowlen};
  const unsigned want = (kRowBlocks + (unsigned)rows - 1) / (unsigned)rows, most = rowlen / 256;
  const unsigned per = want < most ? want : most, piece = ((rowlen + per - 1) / per + 255) / 256 * 256;
  return {(rowlen + piece - 1) / piece, piece};
}

// A thread's turns over `rows` rows of `len` elements: for (turn = first; turn <
// turns; turn += step), each the elements e, e + 256, ... below end of a row.
template <typename I>
struct RowTurns {
  I first, step, turns;
  unsigned e, len;
  RowCut cut;
  struct Piece {
    I row;
    unsigned e, end;
  };
  SLBC_HD Piece piece(I turn) const {
    if (cut.cuts == 1) return {turn, e, len};
    const I row = turn / cut.cuts;
    const unsigned from = (unsigned)(turn - row * cut.cuts) * cut.piece, left = len - from;
    return {row, from + e, from + (left < cut.piece ? left : cut.piece)};
  }
};

template <typename I>
SLBC_HD RowTurns<I> row_turns(unsigned block, unsigned blocks, unsigned thread, I rows, unsigned len) {
  const RowCut cut = row_cut(rows, len);
  const RowWalk<I> w = row_walk<I>(block, blocks, thread, cut.piece);
  return {w.row, w.step, (I)(rows * cut.cuts), w.e, len, cut};
}

// Blocks for `rows` rows of `rowlen` (>= 1) elements
inline int rows_grid(long long rows, long long rowlen) {
  const RowCut cut = row_cut((unsigned long long)rows, (unsigned)rowlen);
  const long long per = cut.piece >= 256 ? 1 : 256 / cut.piece, blocks = (rows * cut.cuts + per - 1) / per;
  return (int)(blocks < 1 ? 1 : blocks > kRowBlocks ? kRowBlocks : blocks);
}

// The sample n, plane z and line y of a row of B x D x H
template <typename I>
SLBC_HD void row_of(I row, int D, int H, int &n, int &z, int &y) {
  const I t = row / (I)H;
  y = (int)(row - t * (I)H);
  n = (int)(t / (I)D);
  z = (int)(t - (I)n * (I)D);
}

// Planes a tracer block marches over, at most `most`: the least of (waves of
// `slots` resident blocks + tail / 6) x (planes + halo) for `tiles` tiles of a
// plane, where a block costs its planes and what it does once, and `tail` sixths
// of a wave stand for blocks that take longer than the others.  Of the many counts of blocks along i
// that give the same march only the first is looked at: the rule runs at every
// update (60,000 x 4 x 4 in FP32: 351 us per update with all, 118 so).
inline int march_planes(int esi, long long tiles, long long slots, int most = 1 << 30, int halo = 2, int tail = 0) {
  long long best = 0;
  int planes = 1;
  for (long long chunks = 1; chunks <= esi;) {
    const int p = (int)((esi + chunks - 1) / chunks);
    if (p <= most) {
      const long long waves = (tiles * ((esi + p - 1) / p) + slots - 1) / slots, cost = (6 * waves + tail) * (p + halo);
      if (best == 0 || cost < best || (tail > 0 && cost == best)) {
        best = cost;
        planes = p;
      }
    }
    if (p == 1) break;
    chunks = (esi + p - 2) / (p - 1);  // the fewest with a shorter march
  }
  return planes;
}

}  // namespace slbc

#endif
