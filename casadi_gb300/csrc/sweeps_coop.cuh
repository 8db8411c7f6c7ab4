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
      value_entry<RECORD>(u, e, wb, p, a.in, a.out, active, ig, pair);
      if (e.w & kTeamMeet) __syncthreads();
    });
    __syncthreads();  // the next tile's entries write the slots this one reads
  }
}

// Cooperative bvec_t sparsity sweeps (SXFunction::sp_forward / sp_reverse): the value
// sweep's level walk with OR instead of arithmetic; the reverse sweep walks the reverse level
// schedule last level first (no two users of a value in one level, so no two instructions of
// a level OR into one slot). OR does not depend on order: the same bits as the sequential
// sweeps.
template <bool REV>
__global__ void __launch_bounds__(kCoopMaxThreads) k_coop_sp(const __grid_constant__ SweepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  u64* w = reinterpret_cast<u64*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const long long ntiles = (a.n + 31) / 32;
  const int nl = REV ? a.t.n_rlevels : a.t.n_levels;
  const u64* code = REV ? a.t.rcode : a.t.lcode;
  const int* lb = REV ? a.t.rbegin : a.t.lbegin;
  const int lv = REV ? a.t.rlv_sz_w : a.t.lv_sz_w;
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const long long il = tile * 32 + lane;
    const bool active = il < a.n;
    const long long ig = a.i_begin + il;
    if (REV) {
      for (int k = warp; k < lv; k += nw) w[k * 32 + lane] = 0;
      __syncthreads();
    }
    for (int step = 0; step < nl; ++step) {
      const int l = REV ? nl - 1 - step : step;
      const int beg = __ldg(lb + l), end = __ldg(lb + l + 1);
      for (int i = beg + warp; i < end; i += nw) {
        const u64 ins = __ldg(code + i);
        const unsigned op = dec_op(ins), A = dec_a(ins), B = dec_b(ins), C = dec_c(ins);
        switch (op) {
          case D_CONST:
            w[A * 32 + lane] = 0;
            break;
          case D_INPUT: {
            const IoDesc& d = a.in[B];
            if (REV) {
              if (active && d.ptr) static_cast<u64*>(d.ptr)[io_off(d, 0, C, ig)] |= w[A * 32 + lane];
              w[A * 32 + lane] = 0;
            } else {
              u64 v = 0;
              if (active && d.ptr) v = __ldg(static_cast<const u64*>(d.ptr) + io_off(d, 0, C, ig));
              w[A * 32 + lane] = v;
            }
          } break;
          case D_OUTPUT: {
            const IoDesc& d = a.out[A];
            if (REV) {
              if (active && d.ptr) {
                u64* p = static_cast<u64*>(d.ptr) + io_off(d, 0, C, ig);
                w[B * 32 + lane] |= *p;
                *p = 0;
              }
            } else if (active && d.ptr) {
              static_cast<u64*>(d.ptr)[io_off(d, 0, C, ig)] = w[B * 32 + lane];
            }
          } break;
          default:
            if (REV) {
              const u64 seed = w[A * 32 + lane];
              w[A * 32 + lane] = 0;
              w[B * 32 + lane] |= seed;
              w[C * 32 + lane] |= seed;
            } else {
              w[A * 32 + lane] = w[B * 32 + lane] | w[C * 32 + lane];
            }
        }
      }
      __syncthreads();
    }
  }
}
