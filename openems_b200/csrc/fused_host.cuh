// fused_host.cuh -- host side of the fused passes (yee_fused.cuh): which
// engines take them, tile shapes, the second set of field and psi buffers,
// the tables of sources and probe taps.  Included by engine.cu.
#pragma once

namespace oems {

// Kernels of a pass: the boxes clear of the CPML slabs, the boxes that meet them.
template <typename T, int kIdBytes, bool kCpml>
static FusedKernel pick_fused_t(int steps) {
  return steps == 2 ? k_fused<2, kIdBytes, kCpml, T> : k_fused<1, kIdBytes, kCpml, T>;
}
template <typename T>
static FusedKernel pick_fused_s(int steps, int id_bytes, bool cpml) {
  if (id_bytes == 1) return cpml ? pick_fused_t<T, 1, true>(steps) : pick_fused_t<T, 1, false>(steps);
  return cpml ? pick_fused_t<T, 2, true>(steps) : pick_fused_t<T, 2, false>(steps);
}
static FusedKernel pick_fused(const oems_engine* en, int steps, bool cpml) {
  const int ib = en->fus.id_bytes;
  if (en->storage == 1) return pick_fused_s<__half>(steps, ib, cpml);
  if (en->storage == 2) return pick_fused_s<__nv_bfloat16>(steps, ib, cpml);
  return pick_fused_s<float>(steps, ib, cpml);
}

// Extensions whose hooks sit inside a timestep run one step a pass, with
// sources and probes in k_post_step after the hooks.
static bool fused_hooks(const oems_engine* en) { return en->mur.on || !en->disp.empty() || !en->rlc.q.empty(); }
// Steps a pass may take: field dumps and near-field boxes read the fields
// after every step; a chunk that meets both z slabs (they are at most three
// cells apart) has more psi than a thread carries from step to step.
static int fused_max_steps(const oems_engine* en) {
  int qa = 0, qb = 0;
  if (en->cpml.on) zfree_chunks(en, &qa, &qb);
  return fused_hooks(en) || !en->fdumps.empty() || !en->boxes.empty() || qa > qb ? 1 : 2;
}

// Whether there is room; a refusal is not an error of the batch, the engine
// goes on without what the buffer was for.
template <typename... A>
static bool got_room(A... allocated) {
  const bool ok = ((allocated == cudaSuccess) && ...);
  if (!ok) cudaGetLastError();
  return ok;
}

// Gives back what fused passes hold beside the engine's own buffers.
static void fused_release(oems_engine* en) {
  FusedHost& F = en->fus;
  F.own_ids.release();
  F.own_table.release();
  F.alt.release();
  F.psi.release();
}

// Ids and table of the distinct coefficient sets of a full-array engine, by
// two kernels over the arrays.  More than 65,536 sets or two sets with one hash:
// the engine keeps its full arrays and the register kernels for good; no room
// for the tables: for now.
static oems_status fused_ids(oems_engine* en, bool* ok) {
  FusedHost& F = en->fus;
  *ok = false;
  if (en->id_bytes) {
    F.ids = en->ids;
    F.table = en->table;
    F.id_bytes = en->id_bytes;
    F.ntable = en->ntable;
    *ok = true;
    return OEMS_OK;
  }
  DevBuf<unsigned long long> key;
  DevBuf<long long> rep;
  DevBuf<int> list, count, id_of;
  if (!got_room(key.ensure(kCoefSlots), rep.ensure(kCoefSlots), list.ensure(kCoefMax), count.ensure(2),
                id_of.ensure(kCoefSlots)))
    return OEMS_OK;
  OEMS_CUDA(cudaMemsetAsync(key.p, 0, kCoefSlots * sizeof(*key.p), en->stream));
  OEMS_CUDA(cudaMemsetAsync(rep.p, 0x7f, kCoefSlots * sizeof(*rep.p), en->stream));
  OEMS_CUDA(cudaMemsetAsync(count.p, 0, 2 * sizeof(int), en->stream));
  CoefArgs a{};
  a.c = en->coeffs;
  a.comp = en->ncells_padded;
  a.nz = en->nz;
  a.nzp = en->g.nzp;
  a.rows = (long long)en->nx * en->ny;
  a.key = key.p;
  a.rep = rep.p;
  a.list = list.p;
  a.count = count.p;
  a.id_of = id_of.p;
  const int grid = (int)std::min<long long>((a.rows * a.nz + 255) / 256, 148 * 8);
  k_coef_sets<<<grid, 256, 0, en->stream>>>(a);
  OEMS_CUDA(cudaGetLastError());
  int n[2];
  OEMS_CUDA(cudaMemcpyAsync(n, count.p, sizeof(n), cudaMemcpyDeviceToHost, en->stream));
  OEMS_CUDA(cudaStreamSynchronize(en->stream));
  if (n[1] || n[0] > kCoefMax) {
    F.state = -1;
    return OEMS_OK;
  }
  DevBuf<long long> first;
  if (!got_room(first.ensure(n[0]))) return OEMS_OK;
  k_coef_first<<<blocks_for(n[0], 256), 256, 0, en->stream>>>(list.p, rep.p, n[0], first.p);
  OEMS_CUDA(cudaGetLastError());
  std::vector<std::pair<long long, int>> sets(n[0]);
  std::vector<int> slots(n[0]);
  std::vector<long long> cells(n[0]);
  OEMS_CUDA(cudaMemcpyAsync(slots.data(), list.p, n[0] * sizeof(int), cudaMemcpyDeviceToHost, en->stream));
  OEMS_CUDA(cudaMemcpyAsync(cells.data(), first.p, n[0] * sizeof(long long), cudaMemcpyDeviceToHost, en->stream));
  OEMS_CUDA(cudaStreamSynchronize(en->stream));
  // ids in cell order, as oems_compress_coefficients numbers them
  for (int k = 0; k < n[0]; ++k) sets[k] = {cells[k], slots[k]};
  std::sort(sets.begin(), sets.end());
  for (int k = 0; k < n[0]; ++k) {
    cells[k] = sets[k].first;
    slots[k] = sets[k].second;
  }
  F.id_bytes = n[0] <= 256 ? 1 : 2;
  F.ntable = n[0];
  if (!got_room(F.own_ids.ensure((size_t)en->ncells_padded * F.id_bytes), F.own_table.ensure((size_t)n[0] * 12)))
    return OEMS_OK;
  OEMS_CUDA(cudaMemsetAsync(F.own_ids.p, 0, (size_t)en->ncells_padded * F.id_bytes, en->stream));
  OEMS_CUDA(cudaMemcpyAsync(list.p, slots.data(), n[0] * sizeof(int), cudaMemcpyHostToDevice, en->stream));
  OEMS_CUDA(cudaMemcpyAsync(first.p, cells.data(), n[0] * sizeof(long long), cudaMemcpyHostToDevice, en->stream));
  k_coef_number<<<blocks_for(n[0], 256), 256, 0, en->stream>>>(list.p, n[0], id_of.p);
  OEMS_CUDA(cudaGetLastError());
  a.ids = F.own_ids.p;
  a.id_bytes = F.id_bytes;
  k_coef_ids<<<grid, 256, 0, en->stream>>>(a);
  OEMS_CUDA(cudaGetLastError());
  k_coef_table<<<blocks_for(n[0] * 12, 256), 256, 0, en->stream>>>(en->coeffs, en->ncells_padded, first.p, n[0],
                                                                  F.own_table.p);
  OEMS_CUDA(cudaGetLastError());
  OEMS_CUDA(cudaMemcpyAsync(n, count.p, sizeof(n), cudaMemcpyDeviceToHost, en->stream));
  OEMS_CUDA(cudaStreamSynchronize(en->stream));
  if (n[1]) {
    F.state = -1;
    return OEMS_OK;
  }
  F.ids = F.own_ids.p;
  F.table = F.own_table.p;
  *ok = true;
  return OEMS_OK;
}

// Whether the engine's kind allows fused passes.  Kernels asked for by name,
// TF/SF planes and the UPML (which change fields between the H and E halves)
// keep the separate updates.
static bool fused_kind(const oems_engine* en) {
  const uint32_t forced = OEMS_ENGINE_STAGED_KERNELS | OEMS_ENGINE_REGISTER_KERNELS | OEMS_ENGINE_SPLIT_KERNELS |
                          OEMS_ENGINE_ZSPLIT_KERNELS | OEMS_ENGINE_PIPE_KERNELS;
  return !((en->flags & forced) || en->tfsf.on || en->upml.on || en->fus.state < 0 ||
           (long long)en->ny * en->g.nzq > INT32_MAX / 2);
}

// Device memory that an engine's buffers may still take: the driver's free
// bytes and the freed blocks that the pool holds.
static oems_status fused_free_bytes(const oems_engine* en, size_t* out) {
  size_t total = 0;
  OEMS_CUDA(cudaMemGetInfo(out, &total));
  cudaMemPool_t pool = nullptr;
  uint64_t held = 0, used = 0;
  if (device_pool(en->device, false, &pool) == cudaSuccess && pool) {
    OEMS_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held));
    OEMS_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
    *out += held > used ? (size_t)(held - used) : 0;
  }
  return OEMS_OK;
}

// What the engine's second buffers are still to take; a quarter of the free
// memory at most, or it keeps the separate kernels (until there is more).
static size_t fused_need(const oems_engine* en) {
  return en->fus.state > 0 ? 0 : en->field_bytes() + (en->id_bytes ? 0 : (size_t)en->ncells_padded);
}

// Whether this engine's batches run as fused passes; prepares ids and the
// second buffers on first use.
static oems_status fused_ready(oems_engine* en, bool* yes) {
  FusedHost& F = en->fus;
  *yes = false;
  if (!fused_kind(en)) return OEMS_OK;
  if (F.state == 0) {
    size_t free_b = 0;
    OEMS_TRY(fused_free_bytes(en, &free_b));
    if (fused_need(en) > free_b / 4) return OEMS_OK;
    bool ok = false;
    OEMS_TRY(fused_ids(en, &ok));
    if (!ok || !got_room(F.alt.ensure(en->field_bytes()))) {
      fused_release(en);
      return OEMS_OK;
    }
    // pads and rows no pass writes stay 0, as in the first buffers
    OEMS_CUDA(cudaMemsetAsync(F.alt.p, 0, en->field_bytes(), en->stream));
    F.state = 1;
  }
  if (en->cpml.on && F.psi.n != en->cpml.psi.n) {
    if (!got_room(F.psi.ensure(en->cpml.psi.n))) {
      F.state = 0;
      fused_release(en);
      return OEMS_OK;
    }
    OEMS_CUDA(cudaMemsetAsync(F.psi.p, 0, F.psi.n * sizeof(float), en->stream));
  }
  *yes = true;
  return OEMS_OK;
}

// The buffers a pass wrote become the current ones.
static void fused_swap(oems_engine* en) {
  FusedHost& F = en->fus;
  char* f = reinterpret_cast<char*>(en->fields);
  en->fields = reinterpret_cast<float*>(F.alt.p);
  F.alt.p = f;
  if (en->cpml.on) {
    const ptrdiff_t d = reinterpret_cast<char*>(F.psi.p) - reinterpret_cast<char*>(en->cpml.psi.p);
    CpmlArgs& A = en->cpml.args;
    for (int s = 0; s < 12; ++s) {
      float*& h = A.psi_h[s / 2][s % 2];
      float*& e = A.psi_e[s / 2][s % 2];
      if (h) h = reinterpret_cast<float*>(reinterpret_cast<char*>(h) + d);
      if (e) e = reinterpret_cast<float*>(reinterpret_cast<char*>(e) + d);
    }
    std::swap(F.psi.p, en->cpml.psi.p);
  }
  F.parity ^= 1;
}

// CPML profiles as a CTA lays them out in shared memory (offset per face).
static int fused_prof_floats(const oems_engine* en, int* off = nullptr) {
  int n = 0;
  for (int f = 0; f < 6; ++f) {
    const CpmlArgs& cp = en->cpml.args;
    if (f >= 4) n = (n + 3) & ~3;  // z rows are read four at a time
    if (off) off[f] = n;
    if (en->cpml.on && cp.L[f] > 0) n += 6 * (f < 4 ? cp.L[f] : cp.zw[f - 4]);
  }
  return n;
}

// Most (cell column, slab) pairs a tile of box B holds: its rows in the y
// slabs, its chunks in the z slabs, and, where the box reaches an x slab,
// every column (the places fused_item gives them).
static int fused_pairs(const oems_engine* en, const FusedBox& B) {
  const CpmlArgs& cp = en->cpml.args;
  const int nzq = (en->nz + 3) / 4;
  int rows = 0, cols = 0;
  for (int t = 0; t < B.nty; ++t) {
    const int j0 = B.ja + t * B.sy, je = std::min(j0 + B.ty, en->ny);
    const int lo = std::max(std::min(cp.L[2], je) - j0, 0);
    const int hi = std::max(je - std::max(cp.L[3] ? cp.start[3] : en->ny, j0), 0);
    rows = std::max(rows, lo + hi);
  }
  for (int t = 0; t < B.ntz; ++t) {
    const int q0 = B.qa + t * B.sz, qe = std::min(q0 + B.wz, nzq);
    const int lo = std::max(std::min((cp.L[4] + 3) / 4, qe) - q0, 0);
    const int hi = std::max(qe - std::max(cp.L[5] ? cp.zbase[1] / 4 : nzq, q0 + lo), 0);
    cols = std::max(cols, lo + hi);
  }
  return rows * B.wz + cols * B.ty + (B.axes & 1 ? B.wz * B.ty : 0);
}

// Tiles of nt threads over box B: the shape with the fewest tiles, and of
// those the one that loads the fewest cells, among those whose psi fits
// `room` pairs.  False: no shape fits.
static bool fused_tile(const oems_engine* en, int steps, int nt, int room, FusedBox& B) {
  const int nzq = (en->nz + 3) / 4;
  B.ja = std::max(B.j0 - steps, 0);
  B.qa = std::max(B.q0 - 1, 0);
  const int rows = std::min(B.j1 + steps, en->ny) - B.ja, cols = std::min(B.q1 + 1, nzq) - B.qa;
  long long best = -1;
  FusedBox got = B;
  for (int wz = 1; wz <= std::min(cols, nt); ++wz) {
    if (wz < cols && wz < 3) continue;
    FusedBox t = B;
    t.wz = wz;
    t.sz = wz == cols ? cols : wz - 2;
    t.ntz = wz == cols ? 1 : (cols - wz + t.sz - 1) / t.sz + 1;
    bool fits = false;
    for (int ty = std::min(nt / wz, rows); ty >= 1 && !fits; ty -= std::max(1, ty / 16)) {
      if (ty < rows && ty < 2 * steps + 1) break;
      t.ty = ty;
      t.sy = ty == rows ? rows : ty - 2 * steps;
      t.nty = ty == rows ? 1 : (rows - ty + t.sy - 1) / t.sy + 1;
      fits = !t.axes || fused_pairs(en, t) <= room;
    }
    if (!fits) continue;
    // rows of a warp's accesses shorter than 128 bytes waste sectors
    const long long tiles = (long long)t.ntz * t.nty;
    const long long cost = tiles * (1 << 20) + tiles * wz * t.ty * (wz < 8 && wz < cols ? 2 : 1);
    if (best >= 0 && cost >= best) continue;
    best = cost;
    got = t;
  }
  B = got;
  return best >= 0;
}

// The grid as boxes: one, or (CPML, split) the box whose tiles and their
// overlap stay clear of every slab, and up to six around it that between them
// hold the slabs: x faces (whole planes), y faces (rows of the planes
// between), z faces (chunks of the rows between).
static int fused_boxes(const oems_engine* en, int steps, bool split, FusedBox* box) {
  const int nzq = (en->nz + 3) / 4;
  const CpmlArgs& cp = en->cpml.args;
  int n = 0;
  auto add = [&](int i0, int i1, int j0, int j1, int q0, int q1, int axes) {
    if (i1 <= i0 || j1 <= j0 || q1 <= q0) return;
    FusedBox B{};
    B.i0 = i0;
    B.i1 = i1;
    B.j0 = j0;
    B.j1 = j1;
    B.q0 = q0;
    B.q1 = q1;
    B.axes = axes;
    box[n++] = B;
  };
  if (!en->cpml.on || !split) {
    add(0, en->nx, 0, en->ny, 0, nzq, en->cpml.on ? 7 : 0);
    return n;
  }
  int qa = 0, qb = nzq;
  zfree_chunks(en, &qa, &qb);
  const int ia = cp.L[0] ? cp.L[0] + steps : 0, ib = cp.L[1] ? cp.start[1] - steps : en->nx;
  const int ja = cp.L[2] ? cp.L[2] + steps : 0, jb = cp.L[3] ? cp.start[3] - steps : en->ny;
  if (cp.L[4]) qa += 1;
  if (cp.L[5]) qb -= 1;
  if (ia >= ib || ja >= jb || qa >= qb) return 0;
  add(0, ia, 0, en->ny, 0, nzq, 7);
  add(ib, en->nx, 0, en->ny, 0, nzq, 7);
  add(ia, ib, 0, ja, 0, nzq, 6);
  add(ia, ib, jb, en->ny, 0, nzq, 6);
  add(ia, ib, ja, jb, 0, qa, 4);
  add(ia, ib, ja, jb, qb, nzq, 4);
  add(ia, ib, ja, jb, qa, qb, 0);
  return n;
}

// Time of a pass by a model, in cycles: an item takes (planes + the
// pipeline's lead-in) iterations; an iteration the larger of its latency
// (barriers, shuffles, shared memory) and the SM's issue slots for the
// resident threads, more of both in the slabs; CTAs go to the SMs as they
// come free.  The constants are what B200 showed; the tuner times the model's
// best.
static double fused_item_cost(const FusedPlan& p, int b, int planes, const int (&occ)[2]) {
  const int c = b < p.ncpml ? 1 : 0;
  const double w = p.box[b].axes == 7 ? 2.2 : p.box[b].axes == 6 ? 1.8 : p.box[b].axes == 4 ? 1.7 : 1.0;
  const double slots = (p.steps == 2 ? 5.5 : 2.8) * w * occ[c] * p.nt[c], latency = (p.steps == 2 ? 1800.0 : 1000.0) * w;
  return (planes + (p.steps == 2 ? 4.5 : 2.5)) * std::max(latency, slots) / occ[c];
}

// Most items an SM of plans that cut x into runs: past that, shorter runs only
// add lead-in planes.  (A plan of one run is always a candidate: its items
// follow the size of the (y, z) plane, whatever the number of SMs.)
constexpr int kFusedItems = 16;

static double fused_cost(const FusedPlan& p, int sms, const int (&occ)[2], std::vector<double>& heap) {
  heap.assign(sms, 0.0);
  for (int b = 0; b < p.nbox; ++b) {
    const FusedBox& B = p.box[b];
    for (int i = B.i0; i < B.i1; i += B.xlen) {
      const double t = fused_item_cost(p, b, std::min(B.xlen, B.i1 - i), occ);
      int left = B.ntz * B.nty;
      if (left > kFusedItems * sms) {  // a very wide plane: whole rounds of the SMs at once
        for (double& h : heap) h += (left / sms) * t;
        left %= sms;
      }
      for (int k = 0; k < left; ++k) {
        std::pop_heap(heap.begin(), heap.end(), std::greater<double>());
        heap.back() += t;
        std::push_heap(heap.begin(), heap.end(), std::greater<double>());
      }
    }
  }
  return *std::max_element(heap.begin(), heap.end());
}

// Grids below this many cells are tuned over more shapes (30 instead of 12): a
// pass takes tens of microseconds, and latency the model does not see decides.
// 121 x 98 x 75 with CPML 25.7 -> 24.0 us a step, 48 x 160 x 70 20.4 -> 19.6, the
// other twelve shapes below a million cells tried within 1%; the first batch
// takes 3 to 14 ms more.  Above, 18 more shapes gave 1 to 3% (170^3 78.8 -> 76.5,
// 256^3 188.9 -> 186.7, none at 200^3) for 20 to 30 ms.  (One-step passes, with
// fewer planes of lead-in, measure level with two-step ones there when launched
// back to back, and a fifth slower inside a graph.)
constexpr long long kFusedSmall = 3000000;

// Sets of the table a CTA's shared memory has room for: plans, and the tuning
// they take, are shared by the grids of one size whose numbers of sets round up
// to the same (a new scene of boxes is rarely of the same number).
static int fused_table_room(const oems_engine* en) {
  if (en->fus.id_bytes != 1) return 0;
  int n = 32;
  while (n < en->fus.ntable) n *= 2;
  return n;
}

// Shapes for passes of `steps`, best first by the model.
static std::vector<FusedPlan> fused_shapes(const oems_engine* en, int steps, int sms, size_t smem_cta,
                                           size_t smem_sm) {
  const int prof = fused_prof_floats(en);
  const int tab = fused_table_room(en) * 12;
  std::vector<FusedPlan> all;
  std::vector<double> heap;
  struct Cta {
    int plain, cpml;
  };
  std::vector<Cta> ctas;
  if (!en->cpml.on) {
    for (int nt : {512, 448, 384, 256, 192, 128, 64}) ctas.push_back({nt, 0});
  } else {
    for (int nt : {512, 384, 256, 192, 128, 64}) ctas.push_back({0, nt});
    for (int nt : {512, 448, 256})
      for (int nc : {512, 448, 384, 256}) ctas.push_back({nt, nc});
  }
  for (const Cta& c : ctas) {
    FusedPlan p;
    p.steps = steps;
    p.nt[0] = c.plain;
    p.nt[1] = c.cpml;
    p.nbox = fused_boxes(en, steps, c.plain && c.cpml, p.box);
    if (!p.nbox) continue;
    for (int b = 0; b < p.nbox; ++b) p.ncpml += p.box[b].axes ? 1 : 0;
    int occ[2] = {1, 1};
    bool ok = true;
    for (int k = 0; ok && k < 2; ++k) {
      if (!p.nt[k]) continue;
      const size_t base = fused_smem(steps, k == 1, p.nt[k], (int)en->elem, en->fus.id_bytes, tab, k ? prof : 0, 0);
      const size_t pair = fused_smem(steps, true, 0, 4, 0, 0, 0, 1) - fused_smem(steps, true, 0, 4, 0, 0, 0, 0);
      ok = base <= smem_cta;
      const int room = ok ? (int)((smem_cta - base) / pair) : 0;
      for (int b = k ? 0 : p.ncpml; ok && b < (k ? p.ncpml : p.nbox); ++b) {
        ok = fused_tile(en, steps, p.nt[k], room, p.box[b]);
        if (ok && k) p.pairs = std::max(p.pairs, fused_pairs(en, p.box[b]));
      }
      p.smem[k] = base + (k ? p.pairs * pair : 0);
      occ[k] = std::max(1, std::min({kFusedMaxThreads / p.nt[k], (int)(smem_sm / (p.smem[k] + 1024)), 32}));
    }
    if (!ok) continue;
    const FusedBox& last = p.box[p.nbox - 1];
    const int planes = last.i1 - last.i0;
    std::vector<FusedPlan> kept;  // the best x-runs of this CTA size
    for (int n = 1, prev = 0; n <= planes; n += 1 + n / 8) {
      const int len = (planes + n - 1) / n;
      if (len == prev) continue;
      prev = len;
      const double target = fused_item_cost(p, p.nbox - 1, len, occ) * occ[p.ncpml == p.nbox ? 1 : 0];
      p.items[0] = p.items[1] = 0;
      for (int b = 0; b < p.nbox; ++b) {
        // x-runs of the slabs' boxes about as long in time as the others'
        FusedBox& B = p.box[b];
        const int k = b < p.ncpml ? 1 : 0, all_b = B.i1 - B.i0;
        int x = len;
        if (p.nbox > 1 && k) {
          const double per = (fused_item_cost(p, b, 100, occ) - fused_item_cost(p, b, 0, occ)) * occ[1] / 100;
          x = std::max((int)(target / per) - steps - 3, 4);
        }
        x = std::min(x, all_b);
        const int runs = (all_b + x - 1) / x;
        B.xlen = (all_b + runs - 1) / runs;
        B.item0 = p.items[k];
        p.items[k] += B.ntz * B.nty * ((all_b + B.xlen - 1) / B.xlen);
      }
      if (n > 1 && p.items[0] + p.items[1] > kFusedItems * sms) break;
      p.cost = fused_cost(p, sms, occ, heap);
      kept.push_back(p);
    }
    const size_t most = std::min<size_t>(kept.size(), en->ncells_padded < kFusedSmall ? 5 : 2);
    std::partial_sort(kept.begin(), kept.begin() + most, kept.end(),
                      [](const FusedPlan& x, const FusedPlan& y) { return x.cost < y.cost; });
    all.insert(all.end(), kept.begin(), kept.begin() + most);
  }
  std::sort(all.begin(), all.end(), [](const FusedPlan& x, const FusedPlan& y) { return x.cost < y.cost; });
  return all;
}

static FusedArgs fused_args(oems_engine* en, int local, bool posts) {
  FusedHost& F = en->fus;
  FusedArgs a{};
  a.nx = en->nx;
  a.ny = en->ny;
  a.nz = en->nz;
  a.nzp = en->g.nzp;
  a.nzq = en->g.nzq;
  a.plane = en->g.plane;
  a.comp = en->ncells_padded;
  a.in = en->fields;
  a.out = F.alt.p;
  a.ids = F.ids;
  a.table = F.table;
  a.ntable = F.ntable;
  a.cp = en->cpml.args;
  a.psi_out = en->cpml.on ? F.psi.p - en->cpml.psi.p : 0;
  fused_prof_floats(en, a.poff);
  a.d_base = en->d_base.p;
  a.local = local;
  a.h_inv = 1.0f / en->h_scale;
  if (posts && en->nexc > 0) {
    a.nsrc = en->nexc;
    a.src_lo = F.src_lo;
    a.src_hi = F.src_hi;
    a.src_off = F.src_i.p;
    a.src_key = a.src_off + en->nx + 1;
    a.src_meta = a.src_key + en->nexc;
    a.src_first = F.src_q.p;
    a.src_count = a.src_first + en->nexc;
    a.samples = en->d_exc_samples.p;
  }
  if (posts && F.ntap > 0) {
    a.ntap = F.ntap;
    a.tap_lo = F.tap_lo;
    a.tap_hi = F.tap_hi;
    a.tap_off = F.tap_i.p;
    a.tap_key = a.tap_off + en->nx + 1;
    a.tap_meta = a.tap_key + F.ntap;
    a.tap_slot = a.tap_meta + F.ntap;
    a.taps = F.taps.p;
  }
  return a;
}

// A pass that is a single launch may start while the kernel before it in the
// stream is draining: until its griddepcontrol.wait it only reads its
// arguments, the table and the profiles.
static void launch_pass(FusedKernel k, const FusedArgs& a, int grid, int nt, size_t smem, cudaStream_t s, bool early) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)nt);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&c, k, a);  // an error is seen by the caller's cudaGetLastError
}

// One pass of p.steps steps, starting at step `local` of the span: the boxes
// with slabs on a second stream beside the others (they read and write the
// same buffers, but no cell is written by both).
// early: the launch may start while the kernel before it drains.
static cudaError_t launch_fused(oems_engine* en, const FusedPlan& p, int local, bool posts, bool early = true) {
  FusedArgs a = fused_args(en, local, posts);
  const bool fork = p.items[0] && p.items[1] && side_stream(en);
  cudaStream_t side = fork ? en->side : en->stream;
  if (fork) {
    cudaEventRecord(en->fork_ev, en->stream);
    cudaStreamWaitEvent(side, en->fork_ev, 0);
  }
  if (p.items[1]) {
    a.nbox = p.ncpml;
    std::copy(p.box, p.box + p.ncpml, a.box);
    a.pairs = p.pairs;
    launch_pass(pick_fused(en, p.steps, true), a, p.items[1], p.nt[1], p.smem[1], side, early && !fork);
  }
  if (p.items[0]) {
    a.nbox = p.nbox - p.ncpml;
    std::copy(p.box + p.ncpml, p.box + p.nbox, a.box);
    launch_pass(pick_fused(en, p.steps, false), a, p.items[0], p.nt[0], p.smem[0], en->stream, early && !p.items[1]);
  }
  if (fork) {
    cudaEventRecord(en->join_ev, side);
    cudaStreamWaitEvent(en->stream, en->join_ev, 0);
  }
  return cudaGetLastError();
}

// Plans already tuned in this process, with the candidates that were timed.
struct FusedTuned {
  std::vector<FusedPlan> plans;
  std::vector<oems_tune_entry> report;
};
static std::map<FusedKey, FusedTuned>& fused_cache() {
  static std::map<FusedKey, FusedTuned> m;
  return m;
}

// Tile shapes of the passes the engine may take (fused_max_steps): the model's
// best, or (with the autotuner) the fastest of its first few on the engine's
// own state, which a pass only reads.  *ok: false where a CTA's shared memory takes no
// tile at all (CPML profiles of thousands of layers): the engine then keeps
// the separate kernels.
static oems_status fused_tune(oems_engine* en, bool* ok) {
  FusedHost& F = en->fus;
  *ok = false;
  int sms = 0, smem_cta = 0, smem_sm = 0;
  OEMS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, en->device));
  OEMS_CUDA(cudaDeviceGetAttribute(&smem_cta, cudaDevAttrMaxSharedMemoryPerBlockOptin, en->device));
  OEMS_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, en->device));
  const int longest = fused_max_steps(en);
  for (int steps = 1; steps <= longest; ++steps)
    for (bool cpml : {false, true})
      OEMS_CUDA(cudaFuncSetAttribute((const void*)pick_fused(en, steps, cpml),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem_cta));
  if (en->cpml.on) side_stream(en);  // (not for the first time inside a capture)
  const bool time_it = !(en->flags & OEMS_ENGINE_NO_AUTOTUNE);
  std::array<int, 6> layers{};
  if (en->cpml.on) std::copy(en->cpml.args.L, en->cpml.args.L + 6, layers.begin());
  const FusedKey key{en->device, en->nx, en->ny, en->nz, F.id_bytes, fused_table_room(en),
                     (en->cpml.on ? 1 : 0) | en->storage << 1 | (time_it ? 8 : 0) | longest << 4, layers};
  std::vector<FusedPlan> plans;
  en->tune_report.clear();
  {
    std::lock_guard<std::mutex> lock(tune_mutex());
    auto hit = fused_cache().find(key);
    if (hit != fused_cache().end()) {
      plans = hit->second.plans;
      en->tune_report = hit->second.report;
    }
  }
  const bool cached = !plans.empty();
  for (int steps = 1; steps <= longest; ++steps) {
    std::vector<FusedPlan> c;
    if (cached)
      c.push_back(plans[steps - 1]);
    else
      c = fused_shapes(en, steps, sms, smem_cta, smem_sm);
    if (c.empty()) {
      F.state = -1;
      fused_release(en);
      return OEMS_OK;
    }
    // shorter passes only finish odd spans; but batches of a step are all theirs,
    // and below kFusedSmall the first three of the model are not the best: 64^3
    // with CPML 21.7 us, 15.1 of 30; 100^3 18.9, 13.6; 60 x 100 x 75 11.6, 8.3 (above:
    // the same at 128^3 to 200^3)
    const bool small = en->ncells_padded < kFusedSmall;
    const size_t most = cached || !time_it ? 1 : small ? 30 : steps != longest ? 3 : 12;
    if (c.size() > most) c.resize(most);
    FusedPlan best = c[0];
    if (c.size() > 1 || (steps == longest && time_it && !cached)) {
      float best_ms = 1e30f;
      for (FusedPlan& p : c) {
        // (a one-step pass has a hook, a recorder or another batch before it, not a pass like it)
        const bool early = steps > 1;
        OEMS_CUDA(launch_fused(en, p, 0, false, early));
        const int kReps = (int)std::max<long long>(3, std::min<long long>(8, 24000000 / en->ncells_padded));
        OEMS_CUDA(cudaEventRecord(en->ev0, en->stream));
        for (int r = 0; r < kReps; ++r) OEMS_CUDA(launch_fused(en, p, 0, false, early));
        OEMS_CUDA(cudaEventRecord(en->ev1, en->stream));
        OEMS_CUDA(cudaEventSynchronize(en->ev1));
        float ms = 0.f;
        OEMS_CUDA(cudaEventElapsedTime(&ms, en->ev0, en->ev1));
        oems_tune_entry te{};
        te.kind = 5;
        te.threads = p.nt[0] + 1000 * p.nt[1];
        te.ichunk = p.box[p.nbox - 1].xlen;
        te.extra = p.nbox * 1000 + p.box[p.nbox - 1].wz * 10 + steps;
        te.reps = kReps * steps;
        te.ms = ms;
        en->tune_report.push_back(te);
        if (ms < best_ms) {
          best_ms = ms;
          best = p;
        }
      }
    }
    F.plan[steps - 1] = best;
  }
  if (!cached) {
    std::lock_guard<std::mutex> lock(tune_mutex());
    fused_cache()[key] = FusedTuned{{F.plan[0], F.plan[1]}, en->tune_report};
  }
  F.tuned = longest;
  *ok = true;
  en->graph_epoch++;
  return OEMS_OK;
}

// Milliseconds a step of the fastest candidate of a tuning report: passes of
// `steps` (fused: true), or the separate kernels.
static float best_of_report(const std::vector<oems_tune_entry>& report, bool fused, int steps) {
  float best = 1e30f;
  for (const oems_tune_entry& t : report)
    if ((t.kind == 5) == fused && (!fused || t.extra % 10 == steps)) best = std::min(best, t.ms / (float)t.reps);
  return best;
}

// Whether the tuned passes are to be taken, by the times of the two.  Two-step
// passes were the faster ones on every grid measured (1.02 to 3 times, 24^3 to
// 256^3, both coefficient forms) but a single plane's, which has nothing to
// march through (1 x 1500 x 1500: 30.5 us a step, separate 21.4).  One-step
// passes lose to kernels that find their arrays in the L2: 24^3 to 64^3 with
// CPML and dispersive cells 22 to 25 us a step, separate 17.5 to 21; 121 x 196 x
// 123, compressed, 81 against 70 there and 49.5 against 43.5 with Mur faces; but
// 95 against 172 at 200^3 with Mur faces.  So where one of these holds the
// separate kernels are tuned too, and taken if they are faster.  kHookUs: what
// the hooks around a pass cost more than around the pair (their launches do not
// hide behind its second kernel): 1.5 to 5 us measured, with one to four hooks.
// The pair is not timed where its bytes alone, past the L2, take longer.
constexpr float kHookUs = 3.0f;
constexpr double kL2Bytes = 126e6, kPeakBytes = 6.5e9;  // per ms: the measured copy rate
static oems_status fused_or_separate(oems_engine* en, bool* yes) {
  FusedHost& F = en->fus;
  const int longest = fused_max_steps(en);
  if ((en->flags & OEMS_ENGINE_NO_AUTOTUNE) || (longest > 1 && en->nx > 1)) return OEMS_OK;
  const std::vector<oems_tune_entry> passes = en->tune_report;
  const float pass = best_of_report(passes, true, longest) + (fused_hooks(en) ? kHookUs * 1e-3f : 0.0f);
  const double cells = (double)en->nx * en->ny * en->nz, coefs = en->id_bytes ? en->id_bytes : 24;
  const double held = cells * (6 * en->elem + (en->id_bytes ? en->id_bytes : 48));
  if (held > 2 * kL2Bytes && pass < 2 * cells * (9 * en->elem + coefs) / kPeakBytes) return OEMS_OK;
  if (!en->tuned) {
    // (without room for the copy of the state that tuning them saves, the passes it is)
    void* save = nullptr;
    if (!got_room(pool_alloc(&save, en->field_bytes() + (en->cpml.on ? en->cpml.psi.n * sizeof(float) : 0), en->stream)))
      return OEMS_OK;
    OEMS_CUDA(cudaFreeAsync(save, en->stream));
    OEMS_TRY(autotune(en));
  }
  *yes = !(best_of_report(en->tune_report, false, 0) < pass);
  en->tune_report.insert(en->tune_report.begin(), passes.begin(), passes.end());
  if (!*yes) {
    F.state = -1;
    fused_release(en);
  }
  return OEMS_OK;
}

// Shapes for an engine that shares the device with others: the model's best
// on `sms` SMs.  *ok as for fused_tune.
static oems_status fused_pack_tune(oems_engine* en, int sms, bool* ok) {
  FusedHost& F = en->fus;
  const int most = fused_max_steps(en);
  *ok = F.pack_sms == sms && F.tuned_pack == most;
  if (*ok) return OEMS_OK;
  if (en->cpml.on) side_stream(en);  // (not for the first time inside a capture)
  int smem_cta = 0, smem_sm = 0;
  OEMS_CUDA(cudaDeviceGetAttribute(&smem_cta, cudaDevAttrMaxSharedMemoryPerBlockOptin, en->device));
  OEMS_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, en->device));
  for (int steps = 1; steps <= most; ++steps) {
    for (bool cpml : {false, true})
      OEMS_CUDA(cudaFuncSetAttribute((const void*)pick_fused(en, steps, cpml),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, smem_cta));
    const std::vector<FusedPlan> c = fused_shapes(en, steps, sms, smem_cta, smem_sm);
    if (c.empty()) {
      F.state = -1;
      fused_release(en);
      return OEMS_OK;
    }
    F.pack_plan[steps - 1] = c[0];
  }
  *ok = true;
  F.pack_sms = sms;
  F.tuned_pack = most;
  en->graph_epoch++;
  return OEMS_OK;
}

// Longest spans of a batch, and the tap buffers for them.
static oems_status fused_taps_ready(oems_engine* en, uint64_t span, bool* room);
static uint64_t fused_span_cap(const oems_engine* en);
static oems_status fused_spans(oems_engine* en, const oems_batch* b, uint64_t* cap) {
  if (en->nprobe() == 0) return OEMS_OK;
  *cap = std::min(*cap, fused_span_cap(en));
  uint64_t longest = std::min(b->num_steps, *cap);
  if (b->sample_interval > 0) longest = std::min<uint64_t>(longest, b->sample_interval);
  // (the first check comes after step check_interval, not after step 0)
  if (b->has_energy_decay_db && b->check_interval > 0) longest = std::min<uint64_t>(longest, b->check_interval + 1);
  // shorter spans where there is no room for the longest one's taps
  for (;; longest /= 2) {
    bool room = false;
    OEMS_TRY(fused_taps_ready(en, longest, &room));
    if (room) break;
    if (longest <= 1) return fail(OEMS_ERR_CUDA, "no device memory for the probes' values of one step");
    *cap = longest / 2;
  }
  return OEMS_OK;
}

// Sources of the batch sorted by (plane, row, chunk); equal cells keep the
// list's order, which is the order they are applied in.  Tables equal to the
// last batch's are there already: batches of a step or two, one after the
// other, took up to 10 us longer for sending them.
static oems_status fused_upload_sources(oems_engine* en, const oems_batch* b, const std::vector<long long>& first,
                                        const std::vector<long long>& count) {
  FusedHost& F = en->fus;
  const int n = en->nexc;
  if (n == 0) return OEMS_OK;
  std::vector<int> order(n), plane(n), key(n);
  for (int x = 0; x < n; ++x) {
    const uint64_t* p = b->excitations[x].position;
    order[x] = x;
    plane[x] = (int)p[0];
    key[x] = (int)p[1] * en->g.nzq + (int)(p[2] / 4);
  }
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return std::tie(plane[x], key[x]) < std::tie(plane[y], key[y]); });
  std::vector<int> I((size_t)en->nx + 1 + 2 * n, 0);
  std::vector<long long> Q(2 * (size_t)n);
  for (int x = 0; x < n; ++x) I[plane[x] + 1]++;
  for (int i = 0; i < en->nx; ++i) I[i + 1] += I[i];
  for (int s = 0; s < n; ++s) {
    const int x = order[s];
    const oems_scheduled_excitation& e = b->excitations[x];
    I[en->nx + 1 + s] = key[x];
    I[en->nx + 1 + n + s] = (int)(e.position[2] & 3) | (int)e.direction << 2 | (e.soft_source ? 1 : 0) << 4;
    Q[s] = first[x];
    Q[n + s] = count[x];
  }
  const int lo = plane[order[0]], hi = plane[order[n - 1]] + 1;
  if (F.src_i.n < I.size() || F.src_q.n < Q.size() || lo != F.src_lo || hi != F.src_hi) en->graph_epoch++;
  F.src_lo = lo;
  F.src_hi = hi;
  if (F.src_i.p && F.src_q.p && I == F.sent_i && Q == F.sent_q) return OEMS_OK;
  F.sent_i.clear();
  OEMS_CUDA(F.src_i.ensure(I.size()));
  OEMS_CUDA(F.src_q.ensure(Q.size()));
  OEMS_CUDA(cudaMemcpyAsync(F.src_i.p, I.data(), I.size() * sizeof(int), cudaMemcpyHostToDevice, en->stream));
  OEMS_CUDA(cudaMemcpyAsync(F.src_q.p, Q.data(), Q.size() * sizeof(long long), cudaMemcpyHostToDevice, en->stream));
  OEMS_CUDA(cudaStreamSynchronize(en->stream));
  F.sent_i.swap(I);
  F.sent_q.swap(Q);
  return OEMS_OK;
}

// Most steps of a span: its taps take at most 256 MB.
static uint64_t fused_span_cap(const oems_engine* en) {
  return std::max<uint64_t>(1, ((uint64_t)64 << 20) / std::max<uint64_t>(1, en->term_idx.size()));
}

// Tap tables (after probes were added) and the buffer of a batch's longest span.
static oems_status fused_taps_ready(oems_engine* en, uint64_t span, bool* room) {
  FusedHost& F = en->fus;
  const int n = (int)en->term_idx.size();
  *room = true;
  if (n == 0) return OEMS_OK;
  if (F.ntap != n) {
    const int nzp = en->g.nzp, nzq = en->g.nzq;
    std::vector<int> order(n), plane(n), key(n);
    for (int x = 0; x < n; ++x) {
      const long long q = en->term_idx[x], row = q / nzp;
      const int k = (int)(q - row * nzp);
      order[x] = x;
      plane[x] = (int)(row / en->ny);
      key[x] = (int)(row % en->ny) * nzq + k / 4;
    }
    std::sort(order.begin(), order.end(),
              [&](int x, int y) { return std::tie(plane[x], key[x], x) < std::tie(plane[y], key[y], y); });
    std::vector<int> I((size_t)en->nx + 1 + 3 * (size_t)n, 0);
    for (int x = 0; x < n; ++x) I[plane[x] + 1]++;
    for (int i = 0; i < en->nx; ++i) I[i + 1] += I[i];
    int* K = I.data() + en->nx + 1;
    for (int s = 0; s < n; ++s) {
      const int x = order[s];
      K[s] = key[x];
      K[n + s] = (int)(en->term_idx[x] % nzp & 3) | en->term_comp[x] << 2;
      K[2 * n + s] = x;
    }
    F.tap_lo = plane[order[0]];
    F.tap_hi = plane[order[n - 1]] + 1;
    OEMS_CUDA(F.tap_i.ensure(I.size()));
    OEMS_CUDA(cudaMemcpyAsync(F.tap_i.p, I.data(), I.size() * sizeof(int), cudaMemcpyHostToDevice, en->stream));
    OEMS_CUDA(cudaStreamSynchronize(en->stream));
    F.ntap = n;
    en->graph_epoch++;
  }
  const size_t need = (size_t)std::max<uint64_t>(span, 1) * n;
  if (F.taps.n < need) {
    *room = got_room(F.taps.ensure(need));
    en->graph_epoch++;
  }
  return OEMS_OK;
}

static cudaError_t launch_probe_sums(oems_engine* en, int steps) {
  ProbeSumArgs a{};
  a.nprobe = en->nprobe();
  a.ntap = (int)en->term_idx.size();
  a.steps = steps;
  a.probe_off = en->d_probe_off.p;
  a.probe_mode = en->d_probe_mode.p;
  a.term_w = en->d_term_w.p;
  a.taps = en->fus.taps.p;
  a.traces = en->d_traces.p;
  a.d_base = en->d_base.p;
  k_probe_sums<<<blocks_for((long long)steps * a.nprobe, 64), 64, 0, en->stream>>>(a);
  return cudaGetLastError();
}

// Steps [0, steps) of a span.
static oems_status launch_steps_fused(oems_engine* en, int steps) {
  FusedHost& F = en->fus;
  const bool hooks = fused_hooks(en);
  const int most = fused_max_steps(en);
  cudaEvent_t* ev = en->profiling ? en->prof_ev.data() : nullptr;
  for (int s = 0; s < steps;) {
    const int k = std::min(most, steps - s);
    if (hooks) OEMS_CUDA(launch_pre_e(en));
    if (ev) OEMS_CUDA(cudaEventRecord(ev[0], en->stream));
    OEMS_CUDA(launch_fused(en, F.current(k), s, !hooks));
    if (ev) OEMS_CUDA(cudaEventRecord(ev[1], en->stream));
    fused_swap(en);
    if (hooks) {
      OEMS_CUDA(launch_post_e(en));
      if (need_post(en)) OEMS_CUDA(launch_post(en, s));
    } else {
      OEMS_CUDA(launch_fd(en, s));
    }
    if (ev) {
      OEMS_CUDA(cudaEventSynchronize(ev[1]));
      float ms = 0.f;
      OEMS_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      en->prof_h_s += ms * 1e-3;
      en->prof_h_n += 1;
    }
    s += k;
  }
  if (!hooks && en->nprobe() > 0) OEMS_CUDA(launch_probe_sums(en, steps));
  return OEMS_OK;
}

// Launches of a pass and what follows it.
static int fused_pass_launches(const oems_engine* en) {
  const FusedPlan& p = en->fus.current(fused_max_steps(en));
  const int per = (p.items[0] ? 1 : 0) + (p.items[1] ? 1 : 0);
  if (fused_hooks(en)) return per + ext_kernels(en) + post_kernels(en);
  return per + (int)(en->fdumps.size() + en->boxes.size());
}

static uint64_t fused_launches(const oems_engine* en, int steps) {
  const int most = fused_max_steps(en);
  const uint64_t passes = (uint64_t)(steps + most - 1) / most;
  return passes * fused_pass_launches(en) + (!fused_hooks(en) && en->nprobe() > 0 ? 1 : 0);
}

// Steps of the pieces a span is run in: as even as it divides, of at most 256
// launches (2.6 ms to make a graph of, under 1% of a piece between two of them),
// and of four steps' multiples, which come back to the same buffers.
constexpr int kGraphLaunches = 256;
static int fused_piece(const oems_engine* en, int steps) {
  const int most = std::max(4, kGraphLaunches / std::max(1, fused_pass_launches(en)) * fused_max_steps(en) / 4 * 4);
  if (steps <= most) return steps;
  const int pieces = (steps + most - 1) / most;
  return ((steps + pieces - 1) / pieces + 3) / 4 * 4;
}

}  // namespace oems
