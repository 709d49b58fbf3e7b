// The default split-precision scheme: FP64 rows cut into e4m3 digits, their
// products on the fp8 tensor pipe (split8.cu).
#pragma once
#include "split.h"

namespace gi {

// The vibrational functions (dipole rows and columns) in the order of the
// digit planes.  Functions fall into classes: two functions share a class
// when every loaded basis uses them alike, i.e. the same (J, key) carry the
// same symmetries on both.  A column of Y = (initial symmetry, key) is
// non-zero on whole classes only, and the final symmetry reads rows of Z of
// whole classes only, so classes are what the half-line-strength GEMM skips.
struct VibTile {  // 128 rows of A: members [i0, i0 + rows) of a class, one component
  int comp, cls, i0, rows;
};
struct VibPlan {
  uint64_t uid = next_uid();
  uint64_t key = 0;                     // what the plan was made of (bases, N, panel)
  int N = 0, ncls = 0, ldz = 0, nk = 0;  // nk: 32-wide K slices of a whole row
  std::vector<std::vector<int32_t>> members;  // functions of a class, ascending
  std::vector<int32_t> zpos;            // row of Z of a function (-1: used by no basis)
  std::vector<int32_t> z0;              // first row of Z of a class
  std::vector<int32_t> s0;              // first K slice of a class ([ncls] = nk)
  std::vector<int32_t> vk;              // [32 nk] function at a K position, -1: padding
  // classes on which (basis uid, gamma, slot) has a non-zero coefficient
  std::map<uint64_t, std::vector<uint32_t>> support;  // [gamma * nslot + slot]
  uint32_t all() const { return ncls >= 32 ? 0xffffffffu : (1u << ncls) - 1u; }
};

// A GEMM of a launch: C[coff(tile) + n ldc + r] over its row tiles and columns.
struct Prob8 {
  const uint8_t* A;
  const uint8_t* B;
  const int32_t* ea;    // [A tile][128]
  const int32_t* eb;    // [column]
  double* C;
  long long ldc;
  const ATile* at;      // nA row tiles; null: tile i holds rows [128 i, 128 i + 128) of M
  const uint16_t* kl;   // A slice of each of the nk slices; null: the first nk
  const int32_t* za;    // [A tile][nkA] planes that are all zero from the top; null: none known
  int nkA, nkB, nk;     // slices per stored A tile, per stored B tile, contracted
  int M, nA, nB, Nc, GA, first;
  // the fused epilogue (see FusedLines)
  int nparts;
  const EpiPart* parts;
  const double* EF;
  const uint8_t* upper;
  const int32_t* lvF;
};
constexpr int kMaxProb8 = 96;

constexpr int kDigits8 = 11;    // digits per element
constexpr int kCols8 = 40;      // columns per tile
constexpr size_t kATileSlice8 = (size_t)kDigits8 * 128 * 32;     // bytes of a tile's K slice
constexpr size_t kBTileSlice8 = (size_t)kDigits8 * kCols8 * 32;
inline size_t a_bytes8(size_t tiles, size_t nk) { return tiles * nk * kATileSlice8; }
inline size_t b_bytes8(size_t cols, size_t nk) {
  return (cols + kCols8 - 1) / kCols8 * nk * kBTileSlice8;
}

// The default scheme applies: no digit count asked for, no pinned kernel or layout.
bool split8_selected(const Ctx* c);
bool split8_active(const Ctx* c);  // after split_prepare: the run uses it
// The context's plan of vibrational functions for its bases and dipole
// (a serving worker: its parent's).  Null with *st set on failure.
const VibPlan* vib_plan(Ctx* c, gi_status* st);
gi_status split8_prepare(Ctx* c);
// The plan and the device tables of its order (both precisions); a worker uses
// its parent's.  panel's first row of the row-source table.
gi_status vib_prepare(Ctx* c, const VibPlan** vp);
const int32_t* vib_rowsrc(const Ctx* c, int panel);
// Row tiles of the dipole (or of panel p of a streamed one), in stored order.
std::vector<VibTile> split8_tiles(const VibPlan& vp, int f0, int rows);
// B workspace bytes and columns of the largest launch; final blocks' digits.
gi_status split8_reserve(Ctx* c, size_t b_bytes, size_t cols, const std::vector<Block*>& finals);
// Digit products per row and column that the GEMM forms, for tile t of
// split8_tiles(vp, 0, N) and class k of the contraction: [t * ncls + k] (the
// zero planes left out, but for a streamed dipole).
const std::vector<double>& split8_products(const Ctx* c);
// The context's dipole digits as a problem's A operand.
void split8_dipole_operand(Ctx* c, Prob8* p);
uint8_t* split8_b(Ctx* c);
int32_t* split8_b_exp(Ctx* c);
// The digits of n column groups; tile_item[b / 64]: the first group of blocks
// b..b+63 (null: one group, whose first block is the launch's).
// (digits false: as doubles, out being double[column][32 nk] of the band.)
gi_status split8_build_y(Ctx* c, const YItem8* items, const int32_t* tile_item, int n,
                         long long blocks, bool digits = true);
// Rows of Z of a basis's roots for the plan (after split_prepare, under the model lock).
// pending (or null): set when the table was launched on the legacy stream, for
// which the caller then waits before it gives up the lock.
gi_status ensure_root_z(Ctx* c, Basis& b, const VibPlan& vp, bool* pending = nullptr);
// Classes a (basis, gamma, slot) has coefficients on; rows of Z that final
// symmetry gF reads of component comp of an initial slot's columns (every final
// J that the owner's bases allow).
uint32_t vib_support(const VibPlan& vp, const Basis& b, int gamma, int slot);
void vib_rows_needed(const Ctx* c, const VibPlan& vp, const Basis& bI, int gF, int slot,
                     uint32_t rset[3]);
// One column band of the half-line-strength GEMM (host description).
struct Band8 {
  uint32_t kset = 0, rset[3] = {0, 0, 0};  // classes contracted; rows needed per component
  size_t col0 = 0, ncol = 0;               // columns of the round (col0 a multiple of 40)
  size_t boff = 0;                         // bytes into the B workspace
  int nk = 0;
  const uint16_t* kl = nullptr;            // device list of A slices
  const int32_t* vl = nullptr;             // and of the functions at their positions
  std::vector<const ATile*> at;            // device row tiles, per panel
  std::vector<int> nA;
};
gi_status split8_gemm_dipole(Ctx* c, const std::vector<Band8>& bands, double* Z, int ldz);
gi_status split8_gemm_final(Ctx* c, const std::vector<FinalJob>& jobs, const FusedLines* lines);
gi_status split8_launch(Ctx* c, int phase, std::vector<Prob8>& probs, const FusedLines* lines,
                        bool tune);
uint64_t split8_identity(Ctx* c);
const int* split8_error_word(const Ctx* c);
void split8_error_seen(Ctx* c);  // the word was read and is set: clear it before the next use
void split8_deactivate(Ctx* c);
void split8_invalidate(Ctx* c);
void split8_release(Ctx* c);
gi_status split8_probe(Ctx* c, int M, int N, int K, const double* dA, const double* dB, int ld,
                       double* dC);
}  // namespace gi
