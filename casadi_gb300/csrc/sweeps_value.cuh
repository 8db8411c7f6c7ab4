// The value walk: value and record sweeps over host-compiled 16-byte entries.
//
// Part of the sweeps.cu translation unit (included where it stands): it uses that file's
// helpers and is not compiled on its own.
#pragma once

// ---------------------------------------------------------------------------------------------
// One entry per instruction (sweeps.cuh, "Value entries"): the slots as byte offsets into the
// work vector w[slot][lane], a constant's bits in place of its operands, and the key of a
// jump-table case that holds the operation's own loads, arithmetic and stores. A warp owns a
// 32-instance tile and walks the entries from a ring in shared memory that it stages itself, a block
// of 16 in flight while the last one is walked (stage_block).
// ---------------------------------------------------------------------------------------------
// The last sin/cos pair of a sweep (VK_SIN_REUSE, VK_COS_REUSE take it again).
struct PairState {
  double s = 0.0, c = 0.0;
};

// One entry. ig: the lane's instance, the range's last one for lanes past its end (which compute
// like any other, so their values take no special path, and store nothing). pt: where the instruction's first recorded partial of this lane goes (RECORD);
// advanced past the partials recorded (rows of 32 lanes). SMALL: the operations of a few integer
// instructions (comparisons, FMIN, FMAX, selections, SIGN, FLOOR, ...) have cases of their own instead
// of a call. k_batch's walks, which the calls made slower than CUDA's functions inline had been (value
// and adjoint of 262144 instances in us, inline functions, calls, cases: a graph of LT, LE and
// IF_ELSE_ZERO 3018, 3793, 2850; of SIGN, COPYSIGN and FLOOR 2763, 3187, 2664; the 20-step rollout 6830,
// 4980, 4958); in the sweeps of one tape the cases make the rollout 1 to 4 % slower (1591 -> 1631 us).
template <bool RECORD, bool SMALL, class Units>
__device__ __forceinline__ void value_entry(const Units& u, const uint4& e, unsigned char* wb, double*& pt,
                                            const IoDesc* in, const IoDesc* out, bool active,
                                            long long ig, PairState& pair) {
#define CGB_X wreg(wb, e.y)
#define CGB_Y wreg(wb, e.z)
#define CGB_REC(bit, d)                     \
  if (RECORD) {                             \
    if (e.w & (bit)) {                      \
      const double dv = (d);                \
      if (active) *pt = dv;                 \
    }                                       \
    pt += 32;                               \
  }
#define CGB_SMALL(OP)                                         \
  case SMALL ? OP : 64u + OP: {                               \
    const double x = CGB_X, y = is_binary(OP) ? CGB_Y : 0.0;  \
    if constexpr (RECORD) {                                   \
      double d0 = 0.0, d1 = 0.0;                              \
      f = dev_fun_der(OP, x, y, d0, d1);                      \
      if (partial_mask(OP) & 1u) CGB_REC(64u, d0)             \
      if (partial_mask(OP) & 2u) CGB_REC(128u, d1)            \
    } else {                                                  \
      f = dev_fun(OP, x, y);                                  \
    }                                                         \
  } break;
  double f;
  switch (e.w & 63u) {
    case D_NOP: return;
    case D_CONST: f = __hiloint2double(static_cast<int>(e.z), static_cast<int>(e.y)); break;
    case D_INPUT: {
      const IoDesc& d = in[e.y];
      f = 0.0;
      if (d.ptr) f = __ldg(static_cast<const double*>(d.ptr) + io_off(d, 0, e.z, ig));
    } break;
    case D_OUTPUT: {
      const IoDesc& d = out[e.x];
      if (active && d.ptr) static_cast<double*>(d.ptr)[io_off(d, 0, e.z, ig)] = CGB_X;
      return;
    }
    case D_ASSIGN: f = CGB_X; break;
    case D_ADD: f = u_add(u, CGB_X, CGB_Y); break;
    case D_SUB: f = u_sub(u, CGB_X, CGB_Y); break;
    case D_MUL: {
      const double x = CGB_X, y = CGB_Y;
      CGB_REC(64u, y)
      CGB_REC(128u, x)
      f = u_mul(u, x, y);
    } break;
    case D_DIV: {
      const double x = CGB_X, y = CGB_Y;
      const FxDivisor d = fx_divisor(y);
      f = d_div(x, y, d);
      CGB_REC(64u, d_div(1.0, y, d))
      CGB_REC(128u, d_div(d_neg(f), y, d))
    } break;
    case D_NEG: f = d_neg(CGB_X); break;
    case D_SQ: {
      const double x = CGB_X;
      CGB_REC(64u, d_twice(x))
      f = u_mul(u, x, x);
    } break;
    case D_TWICE: f = d_twice(CGB_X); break;
    case D_SIN:
    case D_COS:
    case VK_SIN_REUSE:
    case VK_COS_REUSE: {
      const unsigned k = e.w & 63u;
      if (k == D_SIN || k == D_COS) d_sincos(CGB_X, &pair.s, &pair.c);
      const bool sine = k == D_SIN || k == VK_SIN_REUSE;
      f = sine ? pair.s : pair.c;
      CGB_REC(64u, sine ? pair.c : d_neg(pair.s))
    } break;
    case D_EXP: f = d_exp(CGB_X); CGB_REC(64u, f) break;
    case D_LOG: {
      const double x = CGB_X;
      f = d_log(x);
      CGB_REC(64u, d_rcp(x))
    } break;
    case D_SQRT: f = d_sqrt(CGB_X); CGB_REC(64u, d_rcp(d_twice(f))) break;
    case D_INV: f = d_rcp(CGB_X); CGB_REC(64u, d_neg(u_mul(u, f, f))) break;
    case D_TANH: f = d_tanh(CGB_X); CGB_REC(64u, u_sub(u, 1.0, u_mul(u, f, f))) break;
    case D_FABS: {
      const double x = CGB_X;
      f = d_fabs(x);
      CGB_REC(64u, d_sign(x))
    } break;
    CGB_SMALL(D_LT)
    CGB_SMALL(D_LE)
    CGB_SMALL(D_EQ)
    CGB_SMALL(D_NE)
    CGB_SMALL(D_NOT)
    CGB_SMALL(D_AND)
    CGB_SMALL(D_OR)
    CGB_SMALL(D_FLOOR)
    CGB_SMALL(D_CEIL)
    CGB_SMALL(D_SIGN)
    CGB_SMALL(D_COPYSIGN)
    CGB_SMALL(D_IF_ELSE_ZERO)
    CGB_SMALL(D_FMIN)
    CGB_SMALL(D_FMAX)
    default: {
      // the other operations, out of line: one copy serves every kernel
      const double x = CGB_X, y = CGB_Y;
      if constexpr (RECORD) {
        const FunDer r = rare_fun_der(e.w & 63u, x, y);
        f = r.f;
        const unsigned m = partial_mask(e.w & 63u);
        if (m & 1u) CGB_REC(64u, r.d0)
        if (m & 2u) CGB_REC(128u, r.d1)
      } else {
        f = rare_fun(e.w & 63u, x, y);
      }
    }
  }
  wreg(wb, e.x) = f;
#undef CGB_SMALL
#undef CGB_REC
#undef CGB_X
#undef CGB_Y
}

// Staging of an entry stream: the warp copies blocks of kEntBlock entries into a two-slot ring
// in shared memory with cp.async (one 16-byte copy per lane), the next block in flight while the
// current one is walked. Read straight from global memory, one entry ahead, a warp waited about
// 230 cycles per entry for them (every 32-byte sector an L2 access).
__device__ __forceinline__ void stage_block(uint4* ring, const uint4* st, int block) {
  const int lane = threadIdx.x & 31;
  if (lane < kEntBlock)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                     smem_u32(ring + (block & 1) * kEntBlock + lane)),
                 "l"(st + block * kEntBlock + lane)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// f(entry) over the nblocks blocks of st, in order; ring: 2*kEntBlock entries of the warp's own.
template <class F>
__device__ __forceinline__ void staged_walk(const uint4* st, int nblocks, uint4* ring, F&& f) {
  __syncwarp();
  stage_block(ring, st, 0);
#pragma unroll 1
  for (int b = 0; b < nblocks; ++b) {
    __syncwarp();  // every lane is done with the slot the next block takes
    if (b + 1 < nblocks) {
      stage_block(ring, st, b + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();  // the other lanes' copies of this block
    const uint4* blk = ring + (b & 1) * kEntBlock;
    uint4 nxt = blk[0];
#pragma unroll 1
    for (int k = 0; k < kEntBlock; ++k) {
      const uint4 e = nxt;
      nxt = blk[(k + 1) & (kEntBlock - 1)];
      f(e);
    }
  }
}

// The nblocks entry blocks of one tile by one warp.
template <bool RECORD, bool SMALL = false>
__device__ __forceinline__ void value_walk(const PlainUnits& u, const uint4* st, int nblocks, uint4* ring, double* pt,
                                           unsigned char* wb, const IoDesc* in,
                                           const IoDesc* out, bool active, long long ig) {
  PairState pair;
  staged_walk(st, nblocks, ring, [&](const uint4& e) {
    value_entry<RECORD, SMALL>(u, e, wb, pt, in, out, active, ig, pair);
  });
}

// Value (RECORD false) and record sweeps: the warps of a CTA are independent, tiles strided over
// them; a CTA has several warps so that the shared memory it reserves for itself is paid once (28
// instead of 26 resident warps on the 28-slot rollout: 131072 instances are 4096 tiles, which 28
// warps on 152 SMs hold at once and 26 do not). GW: the work vector lives in global memory
// (per-warp blocks of a.wglob) instead of shared memory.
//
// Bound by the FP64 pipe's additions and products and, in the record sweep, by the partials'
// HBM writes. The 20-step cart-pole rollout (3057 instructions, 3400 partials) at 262144
// instances: record 5.02 -> 1.98 ms (5.3 GB of partials, 2.7 TB/s) against the sweep that decoded
// 8-byte words with CUDA's functions inline: 177 thousand instead of 422 thousand executed
// instructions per tile, a third of the FP64 ones.
template <bool RECORD, bool GW>
__global__ void __launch_bounds__(32 * kDirWarps, 28 / kDirWarps) k_value(const __grid_constant__ SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const PlainUnits u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const long long wid = static_cast<long long>(blockIdx.x) * nw + warp;
  const long long nwarps = static_cast<long long>(gridDim.x) * nw;
  const size_t wsmem = kEntRingBytes + (GW ? 0 : static_cast<size_t>(a.t.sz_w) * 256);
  uint4* ring = reinterpret_cast<uint4*>(smem + warp * wsmem);
  unsigned char* wb =
      (GW ? a.wglob + wid * a.wglob_stride : smem + warp * wsmem + kEntRingBytes) + lane * 8;
  const long long ntiles = (a.n + 31) / 32;
  for (long long tile = wid; tile < ntiles; tile += nwarps) {
    const long long il = tile * 32 + lane;
    double* pt = RECORD ? a.partials + static_cast<size_t>(tile) * a.t.n_partials * 32 + lane
                        : nullptr;
    value_walk<RECORD>(u, a.t.ventries, a.t.n_vblocks, ring, pt, wb, a.in, a.out, il < a.n,
                       a.i_begin + (il < a.n ? il : a.n - 1));
  }
}
