// The persistent multi-tape batch kernel.
//
// Part of the sweeps.cu translation unit (included where it stands): it uses that file's
// staging, decoding and I/O helpers and is not compiled on its own.
#pragma once

// ---------------------------------------------------------------------------------------------
// Persistent multi-tape batch: one launch drains a host-built list of work units
// (item, 32-instance tile), longest first, through an atomic counter. An item is one tape over
// its own instance range: a value sweep, a value + adjoint sweep, or a value + tangent sweep
// with identity (or colour-compressed) seeds. Each one-warp CTA grabs a unit, runs the
// warp-level value (or record) walk for its tile and then the adjoint or tangent walk of every
// direction, then grabs the next unit. Tapes of any length and
// instance count share the GPU in one launch instead of one underfilled launch per tape.
// ---------------------------------------------------------------------------------------------
// Bounded wait (lane 0, then shared with the warp) for a split item's tile flag. Every record
// unit precedes every direction unit in the list, so the unit that sets the flag was taken by
// a CTA that is already running and waits on nothing: the wait ends unless that CTA faults.
__device__ __forceinline__ bool wait_tile(const unsigned* flag, unsigned* err) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) {
    const long long t0 = clock64();
    for (unsigned k = 0;; ++k) {
      if (*reinterpret_cast<const volatile unsigned*>(flag)) break;
      if ((k & 63u) == 63u && clock64() - t0 > kWaitCycles) {
        ok = false;
        atomicOr(err, kErrWaitTimeout);
        break;
      }
      __nanosleep(128);
    }
  }
  ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
  __threadfence();  // the partials written before the flag are visible from here on
  return ok;
}

// One warp waiting, with the batch's bounded wait, on a flag that nothing sets: the wait runs
// out after kWaitCycles, records kErrWaitTimeout in *err and the kernel returns.
__global__ void k_wait_probe(const unsigned* flag, unsigned* err) { wait_tile(flag, err); }

cudaError_t launch_wait_probe(const unsigned* flag, unsigned* err, cudaStream_t s) {
  k_wait_probe<<<1, 32, 0, s>>>(flag, err);
  return cudaGetLastError();
}

// kSplit: the batch has split items (per-tile record units and per-direction units); batches
// without any run the instance that holds only the whole-unit path. GW: the work vector lives
// in global memory (per-CTA blocks) instead of shared memory, so residency is not capped by
// the longest tape's work vector.
// MB 28: 72 registers, 28 CTAs to an SM, for batches of more units than the 20 per SM that are resident
// with the 86 to 90 registers of MB 16 (5 warps to a sub-partition's 16384): those would take a second
// wave (100000 instances of the 20-step rollout, 20.6 units per SM: values 1174 and adjoint 2832 us
// against 742 and 1842; of a graph of sums and products 660 and 1562 against 399 and 981). Smaller
// batches run MB 16, 1 to 4 % faster for the moves the cap costs.
template <bool kSplit, bool GW, int MB>
__global__ void __launch_bounds__(32, MB) k_batch(const __grid_constant__ BatchArgs b) {
  extern __shared__ __align__(128) unsigned char smem[];
  const PlainUnits fu;
  const int lane = threadIdx.x;
  uint4* ring = reinterpret_cast<uint4*>(smem);
  unsigned char* wb =
      (GW ? b.wglob + blockIdx.x * b.wglob_stride : smem + kEntRingBytes) + lane * 8;
  double* const pcta = b.scratch + static_cast<size_t>(blockIdx.x) * b.scratch_stride + lane;
  for (;;) {
    unsigned u = 0;
    if (lane == 0) u = atomicAdd(b.counter, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= static_cast<unsigned>(b.n_units)) break;
    const int4 unit = __ldg(b.units + u);
    const BatchItem& it = b.items[unit.x];
    const long long il = static_cast<long long>(unit.y) * 32 + lane;
    const bool active = il < it.n;
    const long long iv = active ? il : it.n - 1;
    const IoDesc* io = it.io;
    // partials: the item's per-tile buffer (split items) or this CTA's scratch (whole units)
    double* pt = (kSplit && it.tile_partials)
                     ? it.tile_partials + static_cast<size_t>(unit.y) * it.t.n_partials * 32 + lane
                     : pcta;
    int d0 = 0, d1 = it.ndir;
    if (!kSplit || unit.z < 0) {
      // record (or value) unit
      if (it.ndir == 0) {
        value_walk<false, true>(fu, it.t.ventries, it.t.n_vblocks, ring, nullptr, wb, io, io + kMaxIo, active,
                          iv);
        continue;
      }
      value_walk<true, true>(fu, it.t.ventries, it.t.n_vblocks, ring, pt, wb, io, io + kMaxIo, active, iv);
      if (kSplit && it.tile_partials) {
        // split item: publish the tile's partials; its directions are separate units
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(it.ready + unit.y, 1u);
        continue;
      }
      // whole unit: the warp's own partial stores must be visible to its loads below
      __syncwarp();
    } else {
      // one direction of a split item, after its tile's record unit
      if (!wait_tile(it.ready + unit.y, b.err)) continue;
      d0 = unit.z;
      d1 = unit.z + 1;
    }
    const bool act1[1] = {active}, tok1[1] = {true};
    const long long ig1[1] = {il};
    for (int dir = d0; dir < d1; ++dir) {
      if (it.forward) {
        const int2 se = __ldg(it.tan_chunks + dir);
        tangent_walk<false, kBatchTanGroup, 1, 1>(fu, it.tan_stream + se.x, se.y / kBatchTanGroup,
                                                  pt, it.t.pconsts, 0, tok1, wb, io + 2 * kMaxIo,
                                                  io + 3 * kMaxIo, true, act1, dir, it.ndir, ig1);
        continue;
      }
      // (the work vector needs no clearing: the adjoint walk assigns every slot before reading)
      if (active) {
        for (int k = 0; k < it.n_zero; ++k) {
          const int2 jk = __ldg(it.zero_in + k);
          const IoDesc& d = io[3 * kMaxIo + jk.x];
          if (d.ptr) static_cast<double*>(d.ptr)[io_off(d, dir, jk.y, il)] = 0.0;
        }
      }
      adjoint_walk<false, kBatchAdjGroup, 1>(fu, it.adj_stream, it.adj_ngr, pt, it.t.pconsts, 0, tok1, wb,
                                             io + 2 * kMaxIo, io + 3 * kMaxIo, act1, dir, ig1);
    }
  }
}

// The batch by teams of kBatchTeam warps, for batches whose longest work vector leaves few warps per
// SM resident (a team shares one work vector between its warps). The units run in rounds of as many
// as the scratch has places for: one launch of cooperative value or record walks, a CTA per unit,
// then one of cooperative adjoint walks over the partials just written; the directions of split
// items follow, a CTA each. Teams of 8, four to an SM, at 64 registers a thread: the mixed queue
// (262144 instances) 21.1 -> 16.0 ms against teams of 4 at 90 registers, the MPC directions (14
// and 10 of 34156 and 76851 instructions, 4096 scenarios) 8.97 -> 6.79 ms; teams of 16, two to an SM,
// 16.3 and 9.04 ms, five teams of 8 at 48 registers 18.6 and 9.63 ms. Separate launches, because a persistent CTA that alternates between the
// walks drifts apart from its neighbours, and then every SM fetches both walks' instructions and
// streams at different places: 65536 instances of the 5365-node random graph took 9.2 ms in one
// persistent launch of teams (187940 instances 33.7 ms), 5.4 ms (14.3 ms) in rounds.
__device__ __forceinline__ double* batch_partials(const BatchArgs& b, const BatchItem& it,
                                                  const int4& unit, int lane) {
  return (it.tile_partials
              ? it.tile_partials + static_cast<size_t>(unit.y) * it.t.n_partials * 32
              : b.scratch + static_cast<size_t>(blockIdx.x) * b.scratch_stride) + lane;
}

// (blockDim.x: 32 * kBatchTeam, or the warps of the split items' record teams)
__global__ void __launch_bounds__(kCoopMaxThreads)
    k_batch_team(const __grid_constant__ BatchArgs b) {
  const PlainUnits u;
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int4 unit = __ldg(b.units + blockIdx.x);
  const BatchItem& it = b.items[unit.x];
  const long long il = static_cast<long long>(unit.y) * 32 + lane;
  const bool active = il < it.n;
  const long long iv = active ? il : it.n - 1;
  const IoDesc* io = it.io;
  uint4* ring = reinterpret_cast<uint4*>(smem) + warp * (2 * kEntBlock);
  unsigned char* wb = smem + (blockDim.x >> 5) * kEntRingBytes + lane * 8;
  const int2 vs = __ldg(it.team_at + warp);
  PairState pair;
  if (it.ndir == 0) {
    staged_walk(it.team + vs.x, vs.y, ring, [&](const uint4& e) {
      double* none = nullptr;
      value_entry<false, false>(u, e, wb, none, io, io + kMaxIo, active, iv, pair);
      if (e.w & kTeamMeet) __syncthreads();
    });
    return;
  }
  double* const pt = batch_partials(b, it, unit, lane);
  staged_walk(it.team + vs.x, vs.y, ring, [&](const uint4& e) {
    double* p = pt + static_cast<size_t>((e.w >> kTeamPidxShift) & kTeamPidxMask) * 32;
    value_entry<true, false>(u, e, wb, p, io, io + kMaxIo, active, iv, pair);
    if (e.w & kTeamMeet) __syncthreads();
  });
}

// SPLIT false: the one direction, tangent or adjoint, of a unit k_batch_team has just recorded (same
// places); true: direction unit.z of a split item.
template <bool SPLIT>
__global__ void __launch_bounds__(32 * kBatchTeam, 4)
    k_batch_team_dir(const __grid_constant__ BatchArgs b) {
  const FmaUnits u = fma_units();
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int4 unit = __ldg(b.units + blockIdx.x);
  const BatchItem& it = b.items[unit.x];
  if (!SPLIT && (it.ndir == 0 || it.tile_partials)) return;
  const long long il = static_cast<long long>(unit.y) * 32 + lane;
  const int dir = SPLIT ? unit.z : 0;  // an item that is not split has at most one direction
  const IoDesc* io = it.io;
  const double* pt = batch_partials(b, it, unit, lane);
  unsigned char* wb = smem + lane * 8;
  const bool active[1] = {il < it.n}, tok[1] = {true};
  const long long ig[1] = {il};
  if (it.forward) {
    const int2 se = __ldg(it.dir_team_at + dir * kBatchTeam + warp);
    tangent_walk<true, kTeamGroup, 1, 1, true>(u, it.dir_team + se.x, se.y / kTeamGroup, pt,
                                               it.t.pconsts, 0, tok, wb, io + 2 * kMaxIo,
                                               io + 3 * kMaxIo, true, active, dir, it.ndir, ig);
    return;
  }
  if (active[0]) {
    for (int k = warp; k < it.n_zero; k += kBatchTeam) {
      const int2 jk = __ldg(it.zero_in + k);
      const IoDesc& d = io[3 * kMaxIo + jk.x];
      if (d.ptr) static_cast<double*>(d.ptr)[io_off(d, dir, jk.y, il)] = 0.0;
    }
  }
  const int2 se = __ldg(it.dir_team_at + warp);
  adjoint_walk<true, kTeamGroup, 1, true>(u, it.dir_team + se.x, se.y / kTeamGroup, pt,
                                          it.t.pconsts, 0, tok, wb, io + 2 * kMaxIo,
                                          io + 3 * kMaxIo, active, dir, ig);
}
