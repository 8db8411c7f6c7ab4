// C ABI: persistent multi-tape batches (host side of k_batch).
//
// Part of the abi.cu translation unit (included at its end): it uses that file's internal
// registry, plans and launch helpers and is not compiled on its own.
#pragma once

// ---------------------------------------------------------------------------------------------
// Persistent multi-tape batches.
// ---------------------------------------------------------------------------------------------
namespace {

struct BatchHost {
  struct Item {
    int tape;
    long long n;
    int ndir;
    bool forward = false;
    std::vector<int> dirmap;  // forward items: direction of each flat input nonzero (-1: none)
    std::vector<IoDesc> io;   // 4*kMaxIo
  };
  std::vector<Item> items;
  bool dirty = true;
  // device side, rebuilt when dirty
  BatchItem* d_items = nullptr;
  IoDesc* d_io = nullptr;
  int4* d_units = nullptr;
  unsigned* d_counter = nullptr;  // [0] next unit, [1] error bits
  unsigned* d_flags = nullptr;    // tile flags of split items
  size_t n_flags = 0;
  std::vector<double*> d_tile_partials;  // per split item
  // split items whose record sweep runs as a cooperative level sweep before the persistent
  // launch (few tiles: the per-tile record units would leave the GPU idle), their flags set
  // once it is done
  struct PreRecord {
    int item;
    size_t flag0;
    long long tiles;
  };
  std::vector<PreRecord> pre;
  int n_pre_units = 0;  // their (item, tile) units, past the others in d_units
  int pre_threads = 0;
  size_t smem_pre = 0;
  int n_units = 0;
  int szw = 1, pmax = 0, grid = 1;
  size_t smem = 0;
  BatchForm form = BF_SHARED;  // of the shared-memory launch
  // work-vector residence: 0 shared memory, 1 global memory (grid_gw CTAs), 2 shared by a team of
  // warps, -1 not tuned yet
  int residence = -1;
  int forced = 0;  // 0 tune, 1 global memory, 2 shared memory
  int grid_gw = 1;
  bool by_teams = false, whole_dirs = false;  // whole_dirs: items of one direction
  size_t smem_value_team = 0, smem_dir_team = 0;
  int n_dir_units = 0;     // the last units: directions of split items
  unsigned char* d_gw = nullptr;
  int device = 0;
  cudaStream_t stream = nullptr;  // owned: graph capture needs a non-legacy stream
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaGraphExec_t exec = nullptr;
  void* exec_scratch = nullptr;
  ~BatchHost() {
    if (exec) cudaGraphExecDestroy(exec);
    cudaFree(d_items);
    cudaFree(d_io);
    cudaFree(d_units);
    cudaFree(d_counter);
    cudaFree(d_flags);
    cudaFree(d_gw);
    for (double* p : d_tile_partials) cudaFree(p);
    if (ev_in) cudaEventDestroy(ev_in);
    if (ev_out) cudaEventDestroy(ev_out);
    if (stream) cudaStreamDestroy(stream);
  }
};

std::vector<std::unique_ptr<BatchHost>> g_batches;

BatchHost* get_batch(int id) {
  std::lock_guard<std::mutex> lk(g_mtx);
  if (id < 0 || id >= static_cast<int>(g_batches.size()) || !g_batches[id]) return nullptr;
  return g_batches[id].get();
}

// The items' tapes are still registered: a prepared batch (and its captured graph) points into
// their device buffers, so a run without one of them is refused.
int batch_tapes(const BatchHost& b) {
  for (size_t k = 0; k < b.items.size(); ++k)
    if (!get_tape(b.items[k].tape))
      return fail(CASADI_GB300_ERR_ID, "batch item %zu: tape %d is gone", k, b.items[k].tape);
  return 0;
}

// The residence before tuning: a forced one (shared memory where the entry ring fits beside the longest
// work vector, which the last two slots before the limit leave no room for), teams, or to be tuned.
int batch_residence(const BatchHost& b) {
  if (b.forced == 1) return 1;
  if (b.forced == 2) return b.smem <= static_cast<size_t>(max_smem_optin()) ? 0 : 1;
  return b.by_teams ? 2 : -1;
}

// Build items, the longest-first unit list and the launch shape.
int batch_prepare(BatchHost& b) {
  if (!b.dirty) return 0;
  if (int rc = batch_tapes(b)) return rc;
  if (b.exec) {
    cudaGraphExecDestroy(b.exec);
    b.exec = nullptr;
  }
  cudaFree(b.d_items);
  cudaFree(b.d_io);
  cudaFree(b.d_units);
  cudaFree(b.d_flags);
  for (double* p : b.d_tile_partials) cudaFree(p);
  b.d_tile_partials.clear();
  b.d_items = nullptr;
  b.d_io = nullptr;
  b.d_units = nullptr;
  b.d_flags = nullptr;
  std::vector<BatchItem> items;
  std::vector<IoDesc> io;
  // (cost, unit): record and whole units first (longest first), then direction units
  std::vector<std::pair<double, int4>> units, dir_units;
  std::vector<std::pair<size_t, size_t>> flag_off;  // (item, first flag) of split items
  size_t n_flags = 0;
  b.szw = 1;
  bool split = false;  // items of two or more directions
  for (const auto& it : b.items) {
    b.szw = std::max(b.szw, get_tape(it.tape)->sz_w);
    split = split || it.ndir >= 2;
  }
  b.smem = smem_value(b.szw);
  auto occ_of = [&](BatchForm form) {
    return b.smem <= static_cast<size_t>(max_smem_optin())
               ? std::max(1, occupancy_batch(b.smem, split, form)) : 1;
  };
  // Teams where one-warp units would leave an SM fewer than 20 warps: below that the walks are
  // bound by each warp's own latency, above it the sequential walks need no meetings. Random graphs
  // of 4000 nodes, value and adjoint of 65536 instances, one-warp units against teams: 24 slots
  // (20 warps per SM) 3.74 and 4.84 ms, 45 slots (17 warps) 4.27 and 3.14, 66 slots (12) 6.67 and
  // 3.08, 142 slots (6) 7.80 and 2.73 ms. They need every item's streams: a batch that runs without
  // them builds none (values and adjoint of the 20-step rollout: 0.40 ms to prepare, not 4.3).
  bool team_ok = occ_of(BF_SHARED) < 20;
  int team_slots = 1, dir_slots = 1;
  bool whole_dirs = false;  // items of one direction, which are not split
  b.pre.clear();
  b.pmax = 0;
  for (size_t k = 0; k < b.items.size(); ++k) {
    const auto& it = b.items[k];
    Tape* t = get_tape(it.tape);
    BatchItem bi;
    std::memset(&bi, 0, sizeof(bi));
    bi.t = t->view();
    bi.ndir = it.ndir;
    bi.n = it.n;
    bi.forward = it.forward ? 1 : 0;
    if (it.ndir > 0 && it.forward) {
      if (static_cast<unsigned>(t->n_partials) >= kMaxPartials)
        return fail(CASADI_GB300_ERR_UNSUPPORTED, "batch item %zu records too many partials", k);
      int err = 0;
      TanPlan* tp = tan_plan(*t, it.ndir, 1, 0, true, std::vector<char>(t->n_in, 0),
                                   it.dirmap, std::vector<char>(t->n_out, 1), &err);
      if (!tp) return err;
      bi.tan_stream = tp->d_stream[group_slot(kBatchTanGroup)];
      bi.tan_chunks = tp->d_chunks[group_slot(kBatchTanGroup)];
      if (team_ok && ensure_tangent_levels(*t) && tan_team(*t, *tp, kBatchTeamSize)) {
        bi.dir_team = tp->d_team[kBatchTeamSize];
        bi.dir_team_at = tp->d_team_at[kBatchTeamSize];
        dir_slots = std::max(dir_slots, t->h_tlv->sz_w);
      }
    } else if (it.ndir > 0) {
      if (static_cast<unsigned>(t->n_partials) >= kMaxPartials)
        return fail(CASADI_GB300_ERR_UNSUPPORTED, "batch item %zu records too many partials", k);
      std::vector<char> seeded(t->n_out);
      for (int j = 0; j < t->n_out; ++j) seeded[j] = it.io[2 * kMaxIo + j].ptr != nullptr;
      int err = 0;
      AdjPlan* ap = adj_plan(*t, 1, 0, seeded, &err);
      if (!ap) return err;
      if (team_ok && ensure_levels(*t, true) && adj_team(*t, *ap)) {
        bi.dir_team = ap->d_team[kBatchTeamSize];
        bi.dir_team_at = ap->d_team_at[kBatchTeamSize];
        dir_slots = std::max(dir_slots, t->rlv_sz_w);
      }
      const int2 se = ap->h_chunks[group_slot(kBatchAdjGroup)];
      bi.adj_stream = ap->d_stream[group_slot(kBatchAdjGroup)] + se.x;
      bi.adj_ngr = se.y / kBatchAdjGroup;
      bi.zero_in = ap->d_zero;
      bi.n_zero = ap->n_zero;
    }
    if (team_ok && ensure_levels(*t)) {
      bi.t = t->view();
      bi.team = t->d_team[kBatchTeamSize];
      bi.team_at = t->d_team_at[kBatchTeamSize];
      team_slots = std::max(team_slots, t->lv_sz_w);
    }
    team_ok = team_ok && bi.team && (it.ndir == 0 || bi.dir_team);
    const long long tiles = (it.n + 31) / 32;
    if (it.ndir >= 2) {
      // split: one record unit per tile into the item's own partial buffer, then one unit
      // per (tile, direction), so the directions of a tile run on different SMs
      double* tp = nullptr;
      const size_t bytes = static_cast<size_t>(tiles) * t->n_partials * 32 * sizeof(double);
      cudaError_t e = cudaMalloc(&tp, std::max<size_t>(bytes, 8));
      if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc(batch tile partials)");
      b.d_tile_partials.push_back(tp);
      bi.tile_partials = tp;
      flag_off.push_back({k, n_flags});
      std::vector<int2> se(it.forward ? it.ndir : 1);
      if (it.forward &&
          (e = cudaMemcpy(se.data(), bi.tan_chunks, sizeof(int2) * it.ndir,
                          cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(e, "read tangent plan");
      // few tiles: the record sweep runs cooperatively (several warps per tile) before the
      // persistent launch instead of as one-warp record units
      const bool pre = tiles <= 4ll * sm_count() && ensure_levels(*t) &&
                       smem_team(t->lv_sz_w, 128, false) <= static_cast<size_t>(max_smem_optin());
      if (pre) {
        b.pre.push_back({static_cast<int>(k), n_flags, tiles});
        bi.t = t->view();
      }
      for (long long tile = 0; tile < tiles; ++tile) {
        if (!pre)
          units.push_back({static_cast<double>(t->n_instr),
                           make_int4(static_cast<int>(k), static_cast<int>(tile), -1, 0)});
        for (int d = 0; d < it.ndir; ++d) {
          const double len = it.forward ? se[d].y : bi.adj_ngr * kBatchAdjGroup;
          dir_units.push_back({len, make_int4(static_cast<int>(k), static_cast<int>(tile), d, 0)});
        }
      }
      n_flags += static_cast<size_t>(tiles);
    } else {
      // whole units: value sweep plus the (at most one) direction in one warp
      const double cost = static_cast<double>(t->n_instr) * (1 + it.ndir);
      for (long long tile = 0; tile < tiles; ++tile)
        units.push_back({cost, make_int4(static_cast<int>(k), static_cast<int>(tile), -1, 0)});
      if (it.ndir > 0) b.pmax = std::max(b.pmax, t->n_partials);
      whole_dirs = whole_dirs || it.ndir > 0;
    }
    items.push_back(bi);
    io.insert(io.end(), it.io.begin(), it.io.end());
  }
  auto longest_first = [](const std::pair<double, int4>& x, const std::pair<double, int4>& y) {
    return x.first > y.first;
  };
  std::stable_sort(units.begin(), units.end(), longest_first);
  std::stable_sort(dir_units.begin(), dir_units.end(), longest_first);
  std::vector<int4> ulist;
  ulist.reserve(units.size() + dir_units.size());
  for (const auto& u : units) ulist.push_back(u.second);
  for (const auto& u : dir_units) ulist.push_back(u.second);
  b.n_dir_units = static_cast<int>(dir_units.size());
  b.n_units = static_cast<int>(ulist.size());
  // The split items' records: one launch of all their tiles, longest tape first, by teams that
  // together fill the GPU.
  long long pre_tiles = 0;
  int pre_slots = 1;
  std::vector<std::pair<double, int4>> pre_units;
  for (const auto& pr : b.pre) {
    const Tape* t = get_tape(b.items[pr.item].tape);
    pre_tiles += pr.tiles;
    pre_slots = std::max(pre_slots, t->lv_sz_w);
    for (long long tile = 0; tile < pr.tiles; ++tile)
      pre_units.push_back({static_cast<double>(t->n_instr), make_int4(pr.item, static_cast<int>(tile), -1, 0)});
  }
  std::stable_sort(pre_units.begin(), pre_units.end(), longest_first);
  for (const auto& u : pre_units) ulist.push_back(u.second);
  b.n_pre_units = static_cast<int>(pre_units.size());
  b.pre_threads = coop_threads_for(pre_tiles);
  while (b.pre_threads > 128 && smem_team(pre_slots, b.pre_threads, false) >
                                    static_cast<size_t>(max_smem_optin()))
    b.pre_threads /= 2;  // the team's entry rings beside the longest work vector
  b.smem_pre = smem_team(pre_slots, b.pre_threads, false);
  for (const auto& pr : b.pre) {
    const Tape* t = get_tape(b.items[pr.item].tape);
    int size = 0;
    while (size + 1 < kTeamSizes && (128 << size) < b.pre_threads) ++size;
    items[pr.item].team = t->d_team[size];
    items[pr.item].team_at = t->d_team_at[size];
  }
  cudaError_t e;
  if (n_flags && (e = cudaMalloc(&b.d_flags, n_flags * sizeof(unsigned))) != cudaSuccess)
    return cuda_fail(e, "cudaMalloc(batch flags)");
  b.n_flags = n_flags;
  for (const auto& fo : flag_off) items[fo.first].ready = b.d_flags + fo.second;
  if ((e = upload(&b.d_io, io)) != cudaSuccess) return cuda_fail(e, "upload batch I/O");
  for (size_t k = 0; k < items.size(); ++k) items[k].io = b.d_io + k * 4 * kMaxIo;
  if ((e = upload(&b.d_items, items)) != cudaSuccess || (e = upload(&b.d_units, ulist)) != cudaSuccess)
    return cuda_fail(e, "upload batch");
  if (!b.d_counter && (e = cudaMalloc(&b.d_counter, 2 * sizeof(unsigned))) != cudaSuccess)
    return cuda_fail(e, "cudaMalloc(counter)");
  // more units at a time than one-warp CTAs of the uncapped form are resident (the directions of split
  // items start as their records end: two directions of 40000 instances of the rollout, 8 record and 16
  // direction units per SM, take 1.71 ms uncapped and 1.84 capped)
  const int at_once = std::max(b.n_dir_units, b.n_units - b.n_dir_units);
  b.form = at_once > sm_count() * occ_of(BF_SHARED) && occ_of(BF_DENSE) > occ_of(BF_SHARED)
               ? BF_DENSE : BF_SHARED;
  b.grid = std::max(1, std::min(sm_count() * occ_of(b.form), std::max(1, b.n_units)));
  // global-memory work vectors: residency capped by registers (and at 8 CTAs per SM, which
  // bounds the per-CTA partial scratch the caller provides)
  const int occ_gw = std::max(1, std::min(8, occupancy_batch(kEntRingBytes, b.n_flags > 0, BF_GLOBAL)));
  b.grid_gw = std::max(1, std::min(sm_count() * occ_gw, std::max(1, b.n_units)));
  cudaFree(b.d_gw);
  b.d_gw = nullptr;
  const size_t gw_bytes = static_cast<size_t>(b.grid_gw) * b.szw * 256;
  if ((e = cudaMalloc(&b.d_gw, std::max<size_t>(gw_bytes, 256))) != cudaSuccess)
    return cuda_fail(e, "cudaMalloc(batch work vectors)");
  b.smem_value_team = smem_team(team_slots, 32 * kBatchTeam, false);
  b.smem_dir_team = smem_coop(dir_slots);
  b.by_teams = team_ok &&
               std::max(b.smem_value_team, b.smem_dir_team) <= static_cast<size_t>(max_smem_optin());
  b.whole_dirs = whole_dirs;
  b.residence = batch_residence(b);
  b.dirty = false;
  return 0;
}

int batch_enqueue(BatchHost& b, void* scratch, cudaStream_t s, int residence) {
  const bool gw = residence == 1;
  cudaError_t e = cudaMemsetAsync(b.d_counter, 0, 2 * sizeof(unsigned), s);
  if (e == cudaSuccess && b.n_flags)
    e = cudaMemsetAsync(b.d_flags, 0, b.n_flags * sizeof(unsigned), s);
  if (e != cudaSuccess) return cuda_fail(e, "reset batch counter");
  BatchArgs a;
  a.items = b.d_items;
  a.units = b.d_units;
  a.n_units = b.n_units;
  a.counter = b.d_counter;
  a.err = b.d_counter + 1;
  a.scratch = static_cast<double*>(scratch);
  a.scratch_stride = static_cast<long long>(b.pmax) * 32;
  a.wglob = gw ? b.d_gw : nullptr;
  a.wglob_stride = static_cast<long long>(b.szw) * 256;
  if (b.n_pre_units) {
    a.units = b.d_units + b.n_units;
    a.n_units = b.n_pre_units;
    if ((e = launch_batch_team(a, BT_VALUE, b.pre_threads, b.smem_pre, s)) != cudaSuccess)
      return cuda_fail(e, "batch record");
    // every tile of the items is recorded: their direction units need not wait
    for (const auto& pr : b.pre)
      if ((e = cudaMemsetAsync(b.d_flags + pr.flag0, 0xff, pr.tiles * sizeof(unsigned), s)) !=
          cudaSuccess)
        return cuda_fail(e, "batch flags");
    a.units = b.d_units;
    a.n_units = b.n_units;
  }
  if (residence == 2) {
    const int places = std::max(b.grid, b.grid_gw);  // of the scratch
    const int whole = b.n_units - b.n_dir_units;
    for (int u0 = 0; u0 < whole; u0 += places) {
      BatchArgs r = a;
      r.units = b.d_units + u0;
      r.n_units = std::min(places, whole - u0);
      e = launch_batch_team(r, BT_VALUE, 32 * kBatchTeam, b.smem_value_team, s);
      if (e == cudaSuccess && b.whole_dirs)
        e = launch_batch_team(r, BT_WHOLE, 32 * kBatchTeam, b.smem_dir_team, s);
      if (e != cudaSuccess) return cuda_fail(e, "batch launch");
    }
    if (b.n_dir_units) {
      a.units = b.d_units + whole;
      a.n_units = b.n_dir_units;
      if ((e = launch_batch_team(a, BT_DIRECTION, 32 * kBatchTeam, b.smem_dir_team, s)) != cudaSuccess)
        return cuda_fail(e, "batch directions launch");
    }
    return 0;
  }
  e = launch_batch(a, gw ? b.grid_gw : b.grid, b.smem, b.n_flags > 0, gw ? BF_GLOBAL : b.form, s);
  if (e != cudaSuccess) return cuda_fail(e, "batch launch");
  return 0;
}

}  // namespace

extern "C" {

int casadi_gb300_batch_create(void) {
  auto b = std::make_unique<BatchHost>();
  cudaError_t e = cudaGetDevice(&b->device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if ((e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaEventCreateWithFlags(&b->ev_in, cudaEventDisableTiming)) != cudaSuccess ||
      (e = cudaEventCreateWithFlags(&b->ev_out, cudaEventDisableTiming)) != cudaSuccess)
    return cuda_fail(e, "batch stream");
  std::lock_guard<std::mutex> lk(g_mtx);
  g_batches.push_back(std::move(b));
  return static_cast<int>(g_batches.size()) - 1;
}

int casadi_gb300_batch_free(int batch) {
  std::lock_guard<std::mutex> lk(g_mtx);
  if (batch < 0 || batch >= static_cast<int>(g_batches.size()) || !g_batches[batch])
    return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  g_batches[batch].reset();
  return 0;
}

int casadi_gb300_batch_add(int batch, int id, int64_t n, int64_t ld, int nadj,
                           const double* const* arg, double* const* res,
                           const double* const* aseed, double* const* asens) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  Tape* t = get_tape(id);
  if (!t) return fail(CASADI_GB300_ERR_ID, "no tape with id %d", id);
  if (int rc = check_device(*t)) return rc;
  if (int rc = check_n(n, ld)) return rc;
  if (nadj < 0 || nadj > 65535) return fail(CASADI_GB300_ERR_ARG, "bad direction count %d", nadj);
  if (n > (1ll << 36)) return fail(CASADI_GB300_ERR_ARG, "too many instances");
  BatchHost::Item it;
  it.tape = id;
  it.n = n;
  it.ndir = nadj;
  it.io.assign(4 * kMaxIo, IoDesc{nullptr, 0, 0, 0});
  fill_io(it.io.data(), t->n_in, vptrs(arg), t->nnz_in, ld, false);
  fill_io(it.io.data() + kMaxIo, t->n_out, vptrs(res), t->nnz_out, ld, false);
  if (nadj > 0) {
    fill_io(it.io.data() + 2 * kMaxIo, t->n_out, vptrs(aseed), t->nnz_out, ld, true);
    fill_io(it.io.data() + 3 * kMaxIo, t->n_in, vptrs(asens), t->nnz_in, ld, true);
  }
  b->items.push_back(std::move(it));
  b->dirty = true;
  return static_cast<int>(b->items.size()) - 1;
}

int casadi_gb300_batch_add_jacobian_colored(int batch, int id, int64_t n, int64_t ld,
                                            int n_colors, const int* color,
                                            const double* const* arg, double* const* res,
                                            double* const* comp) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  Tape* t = get_tape(id);
  if (!t) return fail(CASADI_GB300_ERR_ID, "no tape with id %d", id);
  if (int rc = check_device(*t)) return rc;
  if (int rc = check_n(n, ld)) return rc;
  if (n > (1ll << 36)) return fail(CASADI_GB300_ERR_ARG, "too many instances");
  int nz = 0;
  for (int v : t->nnz_in) nz += v;
  if (!color || n_colors < 1 || n_colors > nz)
    return fail(CASADI_GB300_ERR_ARG, "bad colouring (%d colours for %d input nonzeros)",
                n_colors, nz);
  BatchHost::Item it;
  it.tape = id;
  it.n = n;
  it.ndir = n_colors;
  it.forward = true;
  it.dirmap.assign(color, color + nz);
  for (int v : it.dirmap)
    if (v < -1 || v >= n_colors) return fail(CASADI_GB300_ERR_ARG, "colour %d out of range", v);
  it.io.assign(4 * kMaxIo, IoDesc{nullptr, 0, 0, 0});
  fill_io(it.io.data(), t->n_in, vptrs(arg), t->nnz_in, ld, false);
  fill_io(it.io.data() + kMaxIo, t->n_out, vptrs(res), t->nnz_out, ld, false);
  fill_io(it.io.data() + 3 * kMaxIo, t->n_out, vptrs(comp), t->nnz_out, ld, true);
  b->items.push_back(std::move(it));
  b->dirty = true;
  return static_cast<int>(b->items.size()) - 1;
}

int casadi_gb300_batch_set_residence(int batch, int mode) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  if (mode < 0 || mode > 2) return fail(CASADI_GB300_ERR_ARG, "residence must be 0, 1 or 2");
  b->forced = mode;
  b->residence = batch_residence(*b);
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  return 0;
}

int casadi_gb300_batch_status(int batch) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  if (!b->d_counter) return 0;
  unsigned w[2] = {0, 0};
  cudaError_t e = cudaStreamSynchronize(b->stream);
  if (e == cudaSuccess) e = cudaMemcpy(w, b->d_counter, sizeof(w), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "batch status");
  if (w[1] & kErrWaitTimeout)
    return fail(CASADI_GB300_ERR_CUDA, "batch: a direction unit timed out waiting for its tile");
  return 0;
}

int casadi_gb300_batch_scratch_size(int batch, size_t* bytes) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  if (!bytes) return fail(CASADI_GB300_ERR_ARG, "bad arguments");
  if (int rc = batch_prepare(*b)) return rc;
  *bytes = static_cast<size_t>(std::max(b->grid, b->grid_gw)) * b->pmax * 32 * 8;
  return 0;
}

int casadi_gb300_batch_run(int batch, void* scratch, size_t scratch_bytes, int use_graph,
                           void* stream) {
  BatchHost* b = get_batch(batch);
  if (!b) return fail(CASADI_GB300_ERR_ID, "no batch %d", batch);
  int cur = -1;
  cudaGetDevice(&cur);
  if (cur != b->device) return fail(CASADI_GB300_ERR_ARG, "batch lives on device %d", b->device);
  if (int rc = batch_tapes(*b)) return rc;
  if (int rc = batch_prepare(*b)) return rc;
  const size_t need = static_cast<size_t>(std::max(b->grid, b->grid_gw)) * b->pmax * 32 * 8;
  if (need > 0 && (!scratch || scratch_bytes < need))
    return fail(CASADI_GB300_ERR_SCRATCH, "batch needs %zu bytes of scratch, got %zu", need,
                scratch_bytes);
  cudaStream_t caller = static_cast<cudaStream_t>(stream);
  // order after the caller's stream, run on the owned stream, order the caller after it
  cudaError_t e = cudaEventRecord(b->ev_in, caller);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(b->stream, b->ev_in, 0);
  if (e != cudaSuccess) return cuda_fail(e, "batch ordering");
  if (b->residence < 0) {
    // tune the work-vector residence once per batch layout: both runs produce the results
    if (g_autotune && !capturing(caller)) {
      float ms[2] = {0, 0};
      for (int gw = 0; gw < 2; ++gw) {
        if (gw == 0 && b->smem > static_cast<size_t>(max_smem_optin())) {
          ms[0] = 3.0e38f;  // the shared-memory instance cannot hold this batch
          continue;
        }
        int rc = 0;
        if (int trc = time_runs(b->stream, [&] {
              rc = batch_enqueue(*b, scratch, b->stream, gw);
              return cudaSuccess;
            }, &ms[gw], false))
          return trc;
        if (rc) return rc;
      }
      b->residence = ms[1] < ms[0] ? 1 : 0;
    } else {
      b->residence = b->smem <= static_cast<size_t>(max_smem_optin()) ? 0 : 1;
    }
  }
  if (use_graph) {
    if (b->exec && b->exec_scratch != scratch) {
      cudaGraphExecDestroy(b->exec);
      b->exec = nullptr;
    }
    if (!b->exec) {
      cudaGraph_t g = nullptr;
      e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return cuda_fail(e, "begin capture");
      int rc = batch_enqueue(*b, scratch, b->stream, b->residence);
      e = cudaStreamEndCapture(b->stream, &g);
      if (rc) {
        if (g) cudaGraphDestroy(g);
        return rc;
      }
      if (e != cudaSuccess) return cuda_fail(e, "end capture");
      e = cudaGraphInstantiate(&b->exec, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return cuda_fail(e, "instantiate batch graph");
      b->exec_scratch = scratch;
    }
    e = timed(F_BATCH, b->stream, [&] { return cudaGraphLaunch(b->exec, b->stream); });
    if (e != cudaSuccess) return cuda_fail(e, "graph launch");
  } else {
    int rc = 0;
    e = timed(F_BATCH, b->stream, [&] {
      rc = batch_enqueue(*b, scratch, b->stream, b->residence);
      return cudaSuccess;
    });
    if (rc) return rc;
  }
  e = cudaEventRecord(b->ev_out, b->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(caller, b->ev_out, 0);
  if (e != cudaSuccess) return cuda_fail(e, "batch ordering");
  return 0;
}

}  // extern "C"
