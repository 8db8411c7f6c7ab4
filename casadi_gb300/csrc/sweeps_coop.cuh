// Cooperative (level-scheduled) sweeps.
//
// Part of the sweeps.cu translation unit (included where it stands): it uses that file's
// staging, decoding and I/O helpers and is not compiled on its own.
#pragma once

// ---------------------------------------------------------------------------------------------
// Cooperative value / record sweep for launches with few instances.
//
// One 32-instance tile per CTA (lane = instance) and several warps per CTA. The host's level
// schedule groups the tape into levels of independent instructions and lays each level out over
// the warps of the team, balanced by the operations' latencies, as one entry stream per warp
// (team_streams): the warps meet at a barrier only where one needs a slot another one wrote, so
// chains of dependent instructions run on one warp without meeting. Each instruction is the same
// operation on the same operand values as in the sequential sweep (identical bits), and writes
// its partials at its index of the sequential order. Against a barrier after every level and
// entries decoded from global memory: record of the 10000-node random graph at 16384 instances
// 3.72 -> 1.27 ms, of the MPC constraint and gradient tapes at 4096 scenarios 6.1 -> 2.1 ms.
// ---------------------------------------------------------------------------------------------
template <bool RECORD, bool GW>
__global__ void __launch_bounds__(kCoopMaxThreads) k_coop(const __grid_constant__ SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const PlainUnits u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint4* ring = reinterpret_cast<uint4*>(smem) + warp * (2 * kEntBlock);
  unsigned char* wb = (GW ? a.wglob + blockIdx.x * a.wglob_stride : smem + nw * kEntRingBytes) +
                      lane * 8;
  const long long ntiles = (a.n + 31) / 32;
  const int2 se = __ldg(a.dchunks + warp);  // (first entry, blocks) of this warp's stream
  const uint4* st = a.dstream + se.x;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long il = tile * 32 + lane;
    const bool active = il < a.n;
    const long long ig = a.i_begin + (active ? il : a.n - 1);
    double* pt = RECORD ? a.partials + static_cast<size_t>(tile) * a.t.n_partials * 32 + lane
                        : nullptr;
    PairState pair;
    staged_walk(st, se.y, ring, [&](const uint4& e) {
      double* p = RECORD ? pt + static_cast<size_t>((e.w >> kTeamPidxShift) & kTeamPidxMask) * 32
                         : nullptr;
      value_entry<RECORD, false>(u, e, wb, p, a.in, a.out, active, ig, pair);
      if (e.w & kTeamMeet) __syncthreads();
    });
    __syncthreads();  // the next tile's entries write the slots this one reads
  }
}

// Cooperative bvec_t sparsity sweeps (SXFunction::sp_forward / sp_reverse) by the same teams: the
// value sweep's streams with OR instead of arithmetic, and for the reverse sweep streams of their own
// over the reverse level schedule (sweeps.cuh, "Reverse sparsity entries"). OR does not depend on
// order: the same bits as the sequential sweeps. The 10000-node random graph at 16384 instances:
// sp_forward 440 -> 364 us, sp_reverse 508 -> 369 us against a barrier per level.
template <bool REV>
__global__ void __launch_bounds__(kCoopMaxThreads) k_sp_team(const __grid_constant__ SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint4* ring = reinterpret_cast<uint4*>(smem) + warp * (2 * kEntBlock);
  unsigned char* wb = smem + nw * kEntRingBytes + lane * 8;
  const long long ntiles = (a.n + 31) / 32;
  const int2 se = __ldg(a.dchunks + warp);  // (first entry, blocks) of this warp's stream
  const uint4* st = a.dstream + se.x;
#define CGB_U(off) (*reinterpret_cast<u64*>(wb + (off)))
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long il = tile * 32 + lane;
    const bool active = il < a.n;
    const long long ig = a.i_begin + il;
    staged_walk(st, se.y, ring, [&](const uint4& e) {
      const unsigned key = e.w & 63u;
      if constexpr (!REV) {
        if (key - D_CONST > D_OUTPUT - D_CONST && key != D_NOP) {  // most entries: no jump table
          CGB_U(e.x) = CGB_U(e.y) | CGB_U(e.z);
        } else switch (key) {
          case D_CONST:
            CGB_U(e.x) = 0;
            break;
          case D_INPUT: {
            const IoDesc& d = a.in[e.y];
            u64 v = 0;
            if (active && d.ptr) v = __ldg(static_cast<const u64*>(d.ptr) + io_off(d, 0, e.z, ig));
            CGB_U(e.x) = v;
          } break;
          case D_OUTPUT: {
            const IoDesc& d = a.out[e.x];
            if (active && d.ptr) static_cast<u64*>(d.ptr)[io_off(d, 0, e.z, ig)] = CGB_U(e.y);
          } break;
          default:
            break;
        }
      } else {
        if (key >= SP_ARITH) {
          // operand b, then c: nothing, set or OR
          const unsigned m = key - SP_ARITH, mb = m & 3u, mc = m >> 2;
          const u64 s = CGB_U(e.x);
          if (mb) CGB_U(e.y) = mb == 1u ? s : CGB_U(e.y) | s;
          if (mc) CGB_U(e.z) = mc == 1u ? s : CGB_U(e.z) | s;
        } else switch (key) {
          case SP_OUT_SET:
          case SP_OUT_OR:
          case SP_OUT_CLEAR: {
            const IoDesc& d = a.out[e.x];
            u64 v = 0;
            if (active && d.ptr) {
              u64* p = static_cast<u64*>(d.ptr) + io_off(d, 0, e.z, ig);
              v = *p;
              *p = 0;
            }
            if (key == SP_OUT_SET) CGB_U(e.y) = v;
            if (key == SP_OUT_OR) CGB_U(e.y) |= v;
          } break;
          case SP_IN: {
            const IoDesc& d = a.in[e.y];
            if (active && d.ptr) static_cast<u64*>(d.ptr)[io_off(d, 0, e.z, ig)] |= CGB_U(e.x);
          } break;
          default:
            break;
        }
      }
      if (e.w & kTeamMeet) __syncthreads();
    });
    __syncthreads();  // the next tile's entries write the slots this one reads
  }
#undef CGB_U
}
