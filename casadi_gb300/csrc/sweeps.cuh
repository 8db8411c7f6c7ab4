// Launch interface between the C-ABI layer (abi.cu) and the tape-sweep kernels (sweeps.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "device_ops.cuh"

namespace cgb {

constexpr int kChunk = 256;      // instructions per staged chunk (2 KiB), sparsity and activity sweeps
constexpr int kPofsGran = 16;    // granularity of the per-chunk partial offsets
constexpr int kLeanPB = 63;      // partials per staged chunk block (plan-free adjoint)
// entries per software-pipelined group of the batch kernel's tangent and adjoint walks: small
// groups keep the kernel's code (value walk and both keyed walks) small; the tangent walk
// of the coloured MPC items wants two entries of partial loads in flight
constexpr int kBatchTanGroup = 2;
constexpr int kBatchAdjGroup = 1;
constexpr unsigned kMaxPartials = 1u << 21;  // recorded partials per instance the entries address

// Instruction kinds of the derivative sweeps (the windowed tangent sweep's entries carry them
// in bits 5-8 of their meta word; mixed tangent entries in bits 19-22 of x).
enum LeanKind : unsigned {
  LK_NOP = 0, LK_GEN, LK_ADD, LK_SUB, LK_NEG, LK_TWICE, LK_ASSIGN, LK_IFZ, LK_INPUT, LK_OUTPUT,
  LK_CONST, LK_MIXED
};
constexpr int kMaxIo = 64;       // inputs/outputs per tape handled by one launch

// ---------------------------------------------------------------------------------------------
// Keyed entry streams of the tangent and adjoint walks. An entry is {x, y, z, w}: x the slot
// the entry writes (tangent) or whose adjoint it reads (adjoint), y and z its operand slots,
// all as byte offsets into the warp's work vector (slot * 256); inputs and outputs put their
// I/O index and nonzero in the fields the walks name. w bits 0-5 are the entry's key, the
// walk's jump-table case: the arithmetic form, and for the adjoint which operand receives its
// first contribution. w bits 6-31 describe the recorded partials of the entry G positions
// later (G: entries per pipeline group of the walk that reads the stream), so a walk issues
// the loads of group g+1 while group g computes, with no decoding of g+1's entries first:
// bit 6 load P, bit 7 load Q, bit 8 Q is the partial after P's (otherwise at P's index),
// bits 9-31 P's partial index. A stream for group size G is a header group (no work; it carries
// the first group's partials), the body (an even number of groups, NOP-padded) and one
// trailing NOP group: the walks unroll two groups per iteration and read one group past the
// body. Key 0 is NOP in both walks.
// ---------------------------------------------------------------------------------------------
constexpr int kNumGroupSizes = 4;  // streams are laid out for G = 1, 2, 4, 8
__host__ __device__ constexpr int group_slot(int g) { return g >= 8 ? 3 : g >= 4 ? 2 : g >= 2 ? 1 : 0; }
__host__ __device__ constexpr unsigned ent_key(unsigned w) { return w & 63u; }
constexpr unsigned kPiP = 1u, kPiQ = 2u, kPiQNext = 4u;  // partial-info bits (w >> 6)
constexpr unsigned kPiShift = 6, kPiIndexShift = 9;
// bit 22 of the index: not a recorded partial but entry `index` of the tape's constant partials
// (TapeView::pconsts; the factor of a product with a constant, the reciprocal of a constant
// divisor), which takes no trip to the partials in HBM
constexpr unsigned kPiConst = 1u << 22, kPiIndexMask = kPiConst - 1;
static_assert(kMaxPartials <= kPiConst, "partial indices fit the key word");
static_assert(kPiConst << kPiIndexShift == 1u << 31, "kPiConst is the key word's top bit");

// Tangent forms: the tangent of one arithmetic entry from operand tangents a (y) and b (z) and
// the recorded partials p (d0) and q (d1).
enum TanForm : int {
  TF_PY,    // p*a                     (recorded d0)
  TF_QZ,    // q*b                     (recorded d1)
  TF_PYQZ,  // fma(p, a, q*b)
  TF_Y,     // a                       (d0 = 1: ADD, SUB, ASSIGN and GEN ops with a unit d0)
  TF_Z,     // b                       (ADD)
  TF_YQZ,   // a + q*b                 (d0 = 1, d1 recorded: FMOD, REMAINDER)
  TF_YZ,    // a + b                   (ADD)
  TF_NZ,    // -b                      (SUB)
  TF_YMZ,   // a - b                   (SUB)
  TF_NY,    // -a                      (NEG)
  TF_2Y,    // 2a                      (TWICE)
  TF_IFZ,   // q == 0 ? 0 : b          (IF_ELSE_ZERO)
  TF_SY     // a times a power of two  (a constant partial; z: what it adds to a's high word)
};
__host__ __device__ constexpr bool tf_uses_y(int f) {
  return f == TF_PY || f == TF_PYQZ || f == TF_Y || f == TF_YQZ || f == TF_YZ || f == TF_YMZ ||
         f == TF_NY || f == TF_2Y || f == TF_SY;
}
__host__ __device__ constexpr bool tf_uses_z(int f) {
  return f == TF_QZ || f == TF_PYQZ || f == TF_Z || f == TF_YQZ || f == TF_YZ || f == TF_NZ ||
         f == TF_YMZ || f == TF_IFZ;
}
__host__ __device__ constexpr bool tf_uses_p(int f) { return f == TF_PY || f == TF_PYQZ; }
__host__ __device__ constexpr bool tf_uses_q(int f) {
  return f == TF_QZ || f == TF_PYQZ || f == TF_YQZ || f == TF_IFZ;
}
// Arithmetic tangent keys: (key, form). Operands are read from the work vector: taking the
// previous result from a register instead (operand forwarding) doubles the cases, and the
// larger jump tables cost more in instruction fetch than the shared-memory loads they save.
#define CGB_TK_ARITH(X)                                                                      \
  X(TK_PY, TF_PY) X(TK_QZ, TF_QZ) X(TK_Y, TF_Y) X(TK_Z, TF_Z) X(TK_NZ, TF_NZ)                 \
  X(TK_NY, TF_NY) X(TK_2Y, TF_2Y) X(TK_IFZ, TF_IFZ) X(TK_PYQZ, TF_PYQZ) X(TK_YQZ, TF_YQZ)    \
  X(TK_YZ, TF_YZ) X(TK_YMZ, TF_YMZ) X(TK_SY, TF_SY)
#define CGB_KEY_ENUM(K, ...) K,
// TK_OUT0/TK_OUT: an output's sensitivity (x output, y slot, z nonzero) is 0 or the slot's
// tangent; TK_IN: an input's seed (x slot, y input, z nonzero); TK_MIXED + pm: a union-stream
// entry whose flags differ between the directions (x bits 19-22 kind, 24+2k flags of
// direction k), pm its recorded-partial mask.
enum TanKey : unsigned {
  TK_NOP = 0, TK_OUT0, TK_OUT, TK_IN, TK_MIXED, TK_MIXED_LAST = TK_MIXED + 3,
  CGB_TK_ARITH(CGB_KEY_ENUM) TK_COUNT
};
static_assert(TK_COUNT <= 32, "tangent keys fit 5 bits");

// Adjoint contributions of one entry to an operand slot w, from the entry's adjoint s and the
// operand's partial m: R recorded partial, U unit (ADD, SUB's first operand, ASSIGN and GEN ops
// with a unit d0), M minus one (NEG, SUB's second operand), T two (TWICE), I IF_ELSE_ZERO
// (s unless m is zero); F the slot's first contribution (assigned), A a later one (added).
enum AdjForm : int { CF_N, CF_RF, CF_RA, CF_UF, CF_UA, CF_MF, CF_MA, CF_TF, CF_TA, CF_IF, CF_IA };
__host__ __device__ constexpr bool cf_reads(int f) {
  return f == CF_RA || f == CF_UA || f == CF_MA || f == CF_TA || f == CF_IA;
}
// Arithmetic adjoint keys: (key, contribution to y, contribution to z).
#define CGB_AK_ARITH(X)                                                                      \
  X(AK_RF_N, CF_RF, CF_N) X(AK_RF_RF, CF_RF, CF_RF) X(AK_RF_RA, CF_RF, CF_RA)                \
  X(AK_RA_N, CF_RA, CF_N) X(AK_RA_RF, CF_RA, CF_RF) X(AK_RA_RA, CF_RA, CF_RA)                \
  X(AK_UF_N, CF_UF, CF_N) X(AK_UF_RF, CF_UF, CF_RF) X(AK_UF_RA, CF_UF, CF_RA)                \
  X(AK_UF_UF, CF_UF, CF_UF) X(AK_UF_UA, CF_UF, CF_UA) X(AK_UF_MF, CF_UF, CF_MF)              \
  X(AK_UF_MA, CF_UF, CF_MA)                                                                  \
  X(AK_UA_N, CF_UA, CF_N) X(AK_UA_RF, CF_UA, CF_RF) X(AK_UA_RA, CF_UA, CF_RA)                \
  X(AK_UA_UF, CF_UA, CF_UF) X(AK_UA_UA, CF_UA, CF_UA) X(AK_UA_MF, CF_UA, CF_MF)              \
  X(AK_UA_MA, CF_UA, CF_MA)                                                                  \
  X(AK_MF_N, CF_MF, CF_N) X(AK_MA_N, CF_MA, CF_N) X(AK_TF_N, CF_TF, CF_N)                    \
  X(AK_TA_N, CF_TA, CF_N)                                                                    \
  X(AK_N_RF, CF_N, CF_RF) X(AK_N_RA, CF_N, CF_RA) X(AK_N_IF, CF_N, CF_IF)                    \
  X(AK_N_IA, CF_N, CF_IA)
// AK_OUT_SET/AK_OUT_ADD: an output's seed (x output, y slot, z nonzero) assigned to or added
// into the slot's adjoint; AK_IN: an input's sensitivity (x slot, y input, z nonzero).
enum AdjKey : unsigned {
  AK_NOP = 0, AK_OUT_SET, AK_OUT_ADD, AK_IN, CGB_AK_ARITH(CGB_KEY_ENUM) AK_COUNT
};
static_assert(AK_COUNT <= 32, "adjoint keys fit 5 bits");
// Cooperative tangent and adjoint: the team meets after the entry (bit 5 of the key).
constexpr unsigned kTeamKeyMeet = 32u;
constexpr int kTeamGroup = 2;  // entries per pipeline group: 64 registers a thread (4 take 97)
constexpr int kTeamDirSizes = 3;  // teams of 4, 8 and 16 warps
#undef CGB_KEY_ENUM

// Value entries (k_value, k_batch, k_coop): 16 bytes per instruction.
//   x  byte offset of the result slot in the work vector (OUTPUT: output index)
//   y, z  byte offsets of the operand slots (CONST: the constant's low and high word; INPUT:
//      input index and nonzero; OUTPUT: slot offset and nonzero)
//   w  bits 0-5 the key: the opcode, or VK_SIN_REUSE / VK_COS_REUSE for a SIN or COS that takes
//      the previous pair; bits 6-7 which of its recorded partials are stored (their places in the
//      order stay: the partials of constant operands are never read); in the streams of a cooperative
//      sweep's warps also its first recorded partial (bits 8-30) and whether the team meets
//      after it (bit 31)
constexpr int kEntBlock = 16;  // entries staged at a time
constexpr int kEntRingBytes = 2 * kEntBlock * 16;
constexpr unsigned kTeamPidxShift = 8, kTeamPidxMask = (1u << 23) - 1, kTeamMeet = 1u << 31;
constexpr int kTeamSizes = 4;  // teams of 4, 8, 16 and 32 warps
enum ValueKey : unsigned { VK_SIN_REUSE = 54, VK_COS_REUSE = 55 };
// const_ops: the operands that are constants (1 b, 2 c): their partials are not stored.
inline uint4 value_entry_of(u64 ins, const double* consts, unsigned const_ops) {
  const unsigned op = dec_op(ins), keep = (partial_mask(op) & ~const_ops) << 6;
  uint4 e = make_uint4(dec_a(ins) * 256u, dec_b(ins) * 256u, dec_c(ins) * 256u,
                       op | keep);
  if (op == D_CONST) {
    u64 b;
    memcpy(&b, consts + dec_b(ins), 8);
    e.y = static_cast<unsigned>(b);
    e.z = static_cast<unsigned>(b >> 32);
  } else if (op == D_INPUT) {
    e.y = dec_b(ins);
    e.z = dec_c(ins);
  } else if (op == D_OUTPUT) {
    e.x = dec_a(ins);
    e.z = dec_c(ins);
  } else if ((op == D_SIN || op == D_COS) && (ins & kSincosReuse)) {
    e.w = (op == D_SIN ? VK_SIN_REUSE : VK_COS_REUSE) | keep;
  }
  return e;
}

// Reverse sparsity entries (k_sp_team<true>), with the fields of the value entries: an operand's
// first contribution in sweep order is assigned, so no slot is cleared; constants receive none.
//   SP_OUT_*  x output index, y slot, z nonzero (CLEAR: the output is a constant)
//   SP_IN     x slot, y input index, z nonzero
//   SP_ARITH + mb + 4*mc  x result slot, y, z operand slots; m: 0 none, 1 assigned, 2 ORed
enum SpKey : unsigned { SP_NOP = 0, SP_OUT_SET, SP_OUT_OR, SP_OUT_CLEAR, SP_IN, SP_ARITH };

// One input/output block: element (direction d, nonzero k, instance i) lives at
// ptr[d*dir_stride + k*nz_stride + i*inst_stride].
struct IoDesc {
  void* ptr;
  long long nz_stride;
  long long inst_stride;
  long long dir_stride;
};

// What every sweep needs to know about the tape.
struct TapeView {
  const u64* code;          // kChunk-padded instruction stream (NOP padding)
  const int* pofs;          // pofs[k]: partials recorded before instruction k*kPofsGran
  const double* consts;     // constant pool
  const double* pconsts;    // constant partials (kPiConst)
  const int2* absent_in;    // (input, nonzero) pairs the tape never reads
  const uint4* ventries;    // value entries of the scheduled order
  int n_vblocks;            // their blocks of kEntBlock (NOP padding)
  int n_chunks;
  int n_absent_in;
  int sz_w;
  int n_partials;           // partials recorded per instance
  int* err;                 // device error word
  // work-vector lengths of the level schedules (0 until first needed)
  int lv_sz_w;
  int rlv_sz_w;
};

struct SweepArgs {
  TapeView t;
  long long n;              // instances in this launch
  long long i_begin;        // offset of the first instance inside the IoDesc blocks
  int n_in, n_out;
  int ndir;                 // directions (forward/adjoint sweeps)
  int dir0;                 // first direction of this launch (identity seeds)
  int identity_seed;        // forward: seed of direction d is the d-th unit vector
  int block;                // threads per CTA
  double* partials;         // scratch, tile-major: partials[(tile*P + p)*32 + lane]
  const int* pofs;          // = t.pofs
  int chunk;                // instructions per staged chunk in the derivative sweeps
  int n_code;               // padded instruction count (multiple of kChunk)
  IoDesc in[kMaxIo];        // values in (eval / AD / sparsity)
  IoDesc out[kMaxIo];       // values out
  IoDesc seed[kMaxIo];      // forward: input seeds / adjoint: output seeds
  IoDesc sens[kMaxIo];      // forward: output sensitivities / adjoint: input sensitivities
  const int2* zero_in;              // adjoint: (input, nonzero) pairs with a zero sensitivity
  int n_zero;
  // keyed entry streams (host-compiled, one layout per group size; the launchers pick the
  // variant's into dstream/dchunks)
  const uint4* dstream;             // entries of all streams
  const int2* dchunks;              // per direction (tangent) or one (adjoint): first entry,
                                    // body entries
  const uint4* dstreams[kNumGroupSizes];
  const int2* dchunkss[kNumGroupSizes];
  // global work vector (null: shared memory): CTA b uses wglob + b*wglob_stride
  unsigned char* wglob;
  long long wglob_stride;
  // tangent sweep work queue: items past the grid are claimed from *queue (zeroed before
  // each launch; null: static stride), direction groups of a tile in the order gorder
  // (longest entry stream first; null: natural order)
  unsigned long long* queue;
  const int* gorder;
  // windowed tangent sweep (launch_tangent_win): per (direction group, window) the window's
  // first partial row, partial rows, entry block start and length (uint4 units) in win_blocks;
  // win_dirs directions per CTA (one consumer warp each), win_stages ring stages of win_rows
  // partial rows + win_ents block uint4s each
  const uint4* win_blocks;
  const int4* win_meta;
  int win_n;
  int win_dirs;
  int win_stages;
  int win_rows;
  int win_ents;
};

// One item of a persistent batch: a tape over its own instance range.
struct BatchItem {
  TapeView t;
  int ndir;                 // 0: value sweep only; >0: value + derivative directions
  int forward;              // directions are tangent (1, identity-seeded) or adjoint (0)
  long long n;              // instances
  const IoDesc* io;         // 4*kMaxIo descriptors: inputs, outputs, seeds, sensitivities
  const uint4* adj_stream;  // adjoint entry stream (ndir > 0, !forward)
  int adj_ngr;              // its groups of kBatchAdjGroup entries
  const int2* zero_in;      // inputs with a structurally zero adjoint
  int n_zero;
  // cooperative units (k_batch_team): the streams of a kBatchTeam team's warps (split items
  // recorded before the directions: of the record team's)
  const uint4* team;
  const int2* team_at;      // per warp: first entry, blocks
  const uint4* dir_team;    // keyed adjoint entries, or tangent entries of each direction
  const int2* dir_team_at;  // per warp (tangent: [direction][warp]): first entry, body entries
  const uint4* tan_stream;  // tangent entry streams (forward)
  const int2* tan_chunks;   // per direction: (first entry, entry count)
  // split items (two or more directions): one record unit per tile writes the tile's partials
  // here, (tile*P + p)*32 + lane, then sets ready[tile]; one unit per (tile, direction) waits
  // for the flag and walks its direction
  double* tile_partials;
  unsigned* ready;
};

struct BatchArgs {
  const BatchItem* items;
  const int4* units;        // (item, tile, direction or -1, 0): record/whole units longest
                            // first, then the direction units of split items
  int n_units;
  unsigned* counter;        // next unit (zeroed before each launch)
  unsigned* err;            // kErr* bits (zeroed before each launch)
  double* scratch;          // partials of whole units, scratch_stride doubles per CTA
  long long scratch_stride;
  unsigned char* wglob;     // global work vectors (GW instance): CTA b at wglob + b*wglob_stride
  long long wglob_stride;
};

constexpr int kGwBlock = 128;   // threads per CTA of the global-work-vector value sweeps
constexpr int kWarpShapes = 3;   // CTAs of 1, 2 and 4 independent warps
constexpr int kDirWarps = 1 << (kWarpShapes - 1);
struct WarpShape {
  int ctas;    // resident CTAs per SM
  int block;   // threads per CTA
};
struct WarpOcc {
  int ctas[kWarpShapes] = {};  // resident CTAs per SM by shape
};
WarpOcc occupancy_value(bool record, int sz_w, bool global);
// Shape of a value/record launch of `warps` tiles
WarpShape shape_value(const WarpOcc& o, long long warps, int sms);
int occupancy_gw_sp();           // ... of the sparsity sweeps
int occupancy_gw_dir(bool adjoint);  // ... of the derivative sweeps (one warp per CTA)
cudaError_t launch_gather(long long n, long long ld, int count, const long long* src_row,
                          const double* src, double* dst, cudaStream_t s);
constexpr int kBatchTeamSize = 1, kBatchTeam = 4 << kBatchTeamSize;  // warps of a cooperative unit
// One launch over b.units, b.n_units: record (or value) walks, the one direction of items that are
// not split after them (both at most as many units as the scratch has places), or single directions
// of split items
enum BatchTeamKind { BT_VALUE, BT_WHOLE, BT_DIRECTION };
// threads: 32 * kBatchTeam; record walks of split items may have other teams (a multiple of 32)
cudaError_t launch_batch_team(const BatchArgs& b, BatchTeamKind kind, int threads, size_t smem,
                              cudaStream_t s);
// The persistent batch: work vectors in shared memory, for few units per SM or (dense) more, or in
// global memory (b.wglob)
enum BatchForm { BF_SHARED, BF_DENSE, BF_GLOBAL };
cudaError_t launch_batch(const BatchArgs& b, int grid, size_t smem, bool split, BatchForm form,
                         cudaStream_t s);
int occupancy_batch(size_t smem, bool split, BatchForm form);

// Error bits written to TapeView::err.
constexpr int kErrWaitTimeout = 1;   // a bounded wait on a staged chunk ran out
constexpr int kErrBadOpcode = 2;     // an instruction with an unknown opcode was met

// Shared memory a launch needs (bytes).
size_t smem_primal(int sz_w, int block);  // sparsity and activity sweeps: ring + work vectors
size_t smem_value(int sz_w);              // value and record sweeps: entry ring + one tile's work vector
size_t smem_dir(int sz_w, int dir_warps, int chunk);   // plan-free adjoint (8-byte stream)
size_t smem_lean(int sz_w, int dir_warps, int chunk);  // lean tangent / adjoint
int max_smem_optin();

cudaError_t launch_eval(const SweepArgs& a, int grid, cudaStream_t s);
cudaError_t launch_record(const SweepArgs& a, int grid, cudaStream_t s);
// Derivative sweeps: one-warp CTAs that stride over the (tile, direction group) items, or claim them
// from a.queue, one CTA per place on the GPU.
// Variants of the warp-independent derivative sweeps: entries per software-pipeline group,
// a register cap that lets more one-warp CTAs reside per SM, 32-instance tiles per warp (IPT)
// and, for the tangent sweep, directions per warp (K, walking the union stream of K
// directions). All variants do the same arithmetic in the same order; only speed differs, so
// the host may pick any. A variant's work vector takes smem_lean(sz_w, IPT*K, 0) bytes.
// G8/G4 variants keep more partial loads in flight per warp: for launches with few warps per SM
enum TanVariant : int {
  TV_G2_R80 = 0, TV_G2_R64, TV_G1_R64, TV_G2_K2, TV_G2_K4, TV_G4_R128, TV_G8_R256, TV_COUNT
};
enum AdjVariant : int {
  AV_G2_R80 = 0, AV_G1_R64, AV_G2_R64, AV_G2_I2_R128, AV_G4_R128, AV_G8_R256, AV_COUNT
};
void tan_variant_shape(int variant, int* ipt, int* k);
int adj_variant_ipt(int variant);
// entries per pipeline group (G) of a variant: the keyed-stream layout it reads
int tan_variant_group(int variant);
int adj_variant_group(int variant);
cudaError_t launch_tangent(const SweepArgs& a, int grid, int variant, cudaStream_t s);
// Windowed tangent sweep: one CTA per SM of a warp that stages, window by window, a tile's
// recorded partials and the window's entry block into a shared-memory ring with bulk copies,
// and win_dirs warps that each walk one direction's entries of the window from shared memory
// (the same arithmetic as k_tangent, so the same bits). Work items (tile, direction group)
// in a static stride over a persistent grid.
constexpr int kWinMaxDirs = 31;
constexpr int kWinBarBytes = 128;  // full/empty mbarriers of up to 8 stages
__host__ __device__ inline int win_header_words(int dirs) { return (dirs + 3 + 3) & ~3; }
size_t smem_tangent_win(int sz_w, int dirs, int stages, int rows, int ents);
cudaError_t launch_tangent_win(const SweepArgs& a, int grid, cudaStream_t s);
cudaError_t launch_adjoint(const SweepArgs& a, int grid, int variant, cudaStream_t s);
// The adjoint sweep without an activity plan (k_adjoint_tape<DW>).
cudaError_t launch_adjoint_dense(const SweepArgs& a, int grid, cudaStream_t s);
cudaError_t launch_sp_forward(const SweepArgs& a, int grid, cudaStream_t s);
cudaError_t launch_sp_reverse(const SweepArgs& a, int grid, cudaStream_t s);
cudaError_t launch_activity(const SweepArgs& a, int grid, cudaStream_t s);
// The persistent batch's bounded wait on flag (nonzero: ready); a timeout ORs kErrWaitTimeout
// into *err (one warp).
cudaError_t launch_wait_probe(const unsigned* flag, unsigned* err, cudaStream_t s);
// Cooperative value (record = false) or record sweep: a.block threads (a multiple of 32, at
// most kCoopMaxThreads) share one 32-instance tile and run its level schedule; the work vector
// in shared memory (lv_sz_w x 32 doubles), or in a.wglob blocks when set.
constexpr int kCoopMaxThreads = 1024;
// a.dstream, a.dchunks: the streams of a.block / 32 warps
cudaError_t launch_coop(const SweepArgs& a, bool record, int grid, cudaStream_t s);
size_t smem_team(int lv_sz_w, int threads, bool global);
// Cooperative sparsity sweeps (forward: the value sweep's levels; reverse: the reverse
// schedule's levels, last first); shared memory smem_team of the schedule's work vector.
cudaError_t launch_sp_team(const SweepArgs& a, bool reverse, int grid, cudaStream_t s);
int occupancy_sp_team(int threads, size_t smem);
// Cooperative tangent sweep over recorded partials: one CTA per (tile, direction) item; a.dchunks
// holds the keyed streams of the a.block / 32 warps of each direction, a.gorder the directions in
// work order (null: natural). smem: smem_coop of their level schedule.
cudaError_t launch_tangent_team(const SweepArgs& a, int grid, size_t smem, cudaStream_t s);
// Cooperative adjoint sweep over recorded partials: one CTA per (tile, direction) item;
// a.dstream/a.dchunks are the keyed streams of the a.block / 32 warps, a.zero_in the inputs whose
// sensitivity is a structural zero. Shared memory: smem_coop of the reverse schedule.
cudaError_t launch_adjoint_team(const SweepArgs& a, int grid, cudaStream_t s);
int occupancy_adjoint_team(int threads, size_t smem);
size_t smem_coop(int lv_sz_w);
int occupancy_coop(int threads, size_t smem, bool global);

// Resident CTAs per SM for a given kernel family and shared-memory footprint.
int occupancy_sp(int block, size_t smem);
int occupancy_dir(int variant, bool adjoint, size_t smem);  // warp-independent sweeps
int occupancy_dense(int dir_warps, size_t smem);   // plan-free adjoint

}  // namespace cgb
