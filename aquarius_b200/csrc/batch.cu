// Host side of scene batches (aq_batch_* in include/aquarius_b200.h): many
// independent single-phase scenes of uneven grid sizes stepped together, one
// launch per stage over all scenes, the whole step captured in one CUDA graph.
//
// Layout in HBM: every per-particle, per-cell, per-node and per-brick array of
// the single-scene fluid becomes one concatenation over the scenes (scene s at
// offsets p_off / c_off / f_off / br_off / rp_off).  The particle counting
// sort runs once over the concatenated cell keys (key = c_off + cell): the
// exclusive scan then places scene s's particles at [p_off, p_off + n), so
// the sorted order inside a scene is exactly the single-scene order.
//
// Scenes are created by the single-scene path (aq_fluid_create: seeding,
// initial sort and transfer), copied into the concatenated arrays and
// released, so a scene's initial state is the single-scene one bit for bit.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "fluid_impl.cuh"

using namespace aqb;

#define AQB_CUDA(call)                                                                           \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess)                                                                       \
      return fail(e_ == cudaErrorMemoryAllocation ? AQ_ERR_OUT_OF_MEMORY : AQ_ERR_CUDA,          \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                           \
  } while (0)

#define AQB_TRY(expr)             \
  do {                            \
    aq_status s_ = (expr);        \
    if (s_ != AQ_OK) return s_;   \
  } while (0)

namespace {

__global__ void kb_add_const(int* __restrict__ dst, const int* __restrict__ src, int n, int add) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[i] + add;
}

__global__ void kb_copy_f(const float* __restrict__ a, float* __restrict__ b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

}  // namespace

struct aq_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  aq_config solver{};  // the shared solver settings
  int ns = 0;
  std::vector<SceneDesc> scenes;
  std::vector<aq_config> cfgs;
  std::vector<double> time;
  std::vector<int> phase;
  // prefix sums of virtual blocks per family, ns + 1 each
  std::vector<int> pre_p, pre_n, pre_b, pre_s, pre_f, pre_r;
  SceneDesc* scenes_d = nullptr;
  int* pre_d = nullptr;
  BatchIndex bi{};
  int N = 0, C = 0, F = 0, NB = 0, NRP = 0;
  int sms = 148;
  int multiple = 64;  // cap on CTAs per SM of a batched launch (occupancy decides below it)
  int xs = 1;         // x planes per packed-row Jacobi item
  bool pipe = false;  // pipelined plane loads (xs > 1)
  int2* row_list = nullptr;  // active (scene, item) pairs of the current systems
  int* n_row_list = nullptr;
  int row_list_cap = 0;

  // Cluster solve (when every scene fits one): scenes by cluster width, largest
  // first; each width is a launch on a stream of its own inside the step.  A
  // fluid that has outgrown its cluster stays live and is solved behind them
  // in a cluster of 16 CTAs, or else by the row sweeps (cl_spill, cl_spill16:
  // some scene can come to that).
  static constexpr int kWidths = 5;  // 1, 2, 4, 8, 16 CTAs
  bool cl_planned = false;  // every scene fits a cluster
  bool clusters = false;    // and is solved in it
  bool cl_spill = false, cl_spill16 = false;
  int cl_first[kWidths + 1] = {0};
  int* cl_order = nullptr;
  int2* cl_scratch = nullptr;
  int *cl_map = nullptr, *cl_list = nullptr;
  double* cl_part = nullptr;
  int* cl_spilled = nullptr;  // some scene did not fit its cluster; one of 16 CTAs
  cudaStream_t cl_stream[kWidths] = {nullptr};
  cudaEvent_t cl_event[kWidths + 1] = {nullptr};

  Particles cur{}, tmp{};
  int *key = nullptr, *slot = nullptr, *perm_u = nullptr, *sort_index = nullptr;
  int *count = nullptr, *off = nullptr, *tile_sums = nullptr;
  float *u0 = nullptr, *v0 = nullptr, *w0 = nullptr;
  float *un1 = nullptr, *vn1 = nullptr, *wn1 = nullptr;
  float *un2 = nullptr, *vn2 = nullptr, *wn2 = nullptr;
  uint8_t *h1 = nullptr, *h2 = nullptr;
  int8_t* type = nullptr;
  float *density = nullptr, *div = nullptr, *rhs = nullptr, *pa = nullptr, *pb = nullptr;
  int* pcount = nullptr;
  uint8_t* bact = nullptr;
  double *part_b2 = nullptr, *rpart = nullptr;
  int* part_nf = nullptr;
  SolveState* ss = nullptr;
  int* live = nullptr;

  cudaGraphExec_t exec = nullptr;
  // the step in two graphs, split behind the sort (as aq_fluid's)
  cudaGraphExec_t exec_sort = nullptr, exec_rest = nullptr;
  cudaStream_t copy = nullptr;
  cudaEvent_t sorted = nullptr, copied = nullptr;
  int graph_launches = 0, body_launches = 0;  // of a step of row sweeps
  int step_launches = 0;                      // of a step as it runs, outside conditional nodes
  std::vector<void*> allocs;

  ~aq_batch() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    invalidate_graph();
    if (copy) cudaStreamSynchronize(copy);
    if (copy) cudaStreamDestroy(copy);
    if (sorted) cudaEventDestroy(sorted);
    if (copied) cudaEventDestroy(copied);
    for (cudaEvent_t e : cl_event)
      if (e) cudaEventDestroy(e);
    for (cudaStream_t q : cl_stream)
      if (q) cudaStreamDestroy(q);
    for (void* p : allocs) cudaFree(p);
    if (own_stream && stream) cudaStreamDestroy(stream);
  }

  template <typename T>
  aq_status alloc(T** p, size_t n) {
    void* q = nullptr;
    const size_t bytes = std::max<size_t>(n * sizeof(T), 16);
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess)
      return fail(e == cudaErrorMemoryAllocation ? AQ_ERR_OUT_OF_MEMORY : AQ_ERR_CUDA,
                  std::string("cudaMalloc: ") + cudaGetErrorString(e));
    allocs.push_back(q);
    *p = (T*)q;
    e = cudaMemsetAsync(q, 0, bytes, stream);
    if (e != cudaSuccess) return fail(AQ_ERR_CUDA, cudaGetErrorString(e));
    return AQ_OK;
  }

  int grid() const { return std::max(1, sms * multiple); }
  int grid512() const { return std::max(1, sms * std::max(1, multiple / 2)); }
  aq_status set_sweep_plan(int planes, bool pipelined);
  aq_status enq_row_list() {
    if (cudaError_t e = launch_batch_row_list(stream, bi, pre_r[ns], xs, bact, row_list, n_row_list))
      return fail(AQ_ERR_CUDA, std::string("row list: ") + cudaGetErrorString(e));
    return AQ_OK;
  }

  aq_status allocate();
  aq_status plan_clusters();
  aq_status enq_clusters(unsigned long long spill);
  aq_status enq_wide_clusters(unsigned long long rows);
  aq_status add_scene(int s, aq_fluid* f);
  aq_status enq_sort();       // the step's particle stage
  aq_status enq_pre_solve();  // the rest up to the solve
  aq_status enq_sweeps(int sweeps);
  aq_status enq_solve_fixed();  // by row sweeps, of the live scenes
  aq_status enq_solve_body(unsigned long long handle);
  aq_status enq_post_solve();
  aq_status capture_step(bool sort, bool rest, cudaGraphExec_t* out);
  aq_status build_graph();
  void invalidate_graph() {
    for (cudaGraphExec_t* e : {&exec, &exec_sort, &exec_rest}) {
      if (*e) cudaGraphExecDestroy(*e);
      *e = nullptr;
    }
  }
};

aq_status aq_batch::allocate() {
  const size_t n = (size_t)N, c = (size_t)C, fz = (size_t)F;
  AQB_TRY(alloc(&cur.px, n)); AQB_TRY(alloc(&cur.py, n)); AQB_TRY(alloc(&cur.pz, n));
  AQB_TRY(alloc(&cur.vx, n)); AQB_TRY(alloc(&cur.vy, n)); AQB_TRY(alloc(&cur.vz, n));
  AQB_TRY(alloc(&tmp.px, n)); AQB_TRY(alloc(&tmp.py, n)); AQB_TRY(alloc(&tmp.pz, n));
  AQB_TRY(alloc(&tmp.vx, n)); AQB_TRY(alloc(&tmp.vy, n)); AQB_TRY(alloc(&tmp.vz, n));
  AQB_TRY(alloc(&key, n)); AQB_TRY(alloc(&slot, n)); AQB_TRY(alloc(&perm_u, n)); AQB_TRY(alloc(&sort_index, n));
  AQB_TRY(alloc(&count, c + 1)); AQB_TRY(alloc(&off, c + 1));
  AQB_TRY(alloc(&tile_sums, cell_scan_tiles(C)));
  AQB_TRY(alloc(&u0, fz)); AQB_TRY(alloc(&v0, fz)); AQB_TRY(alloc(&w0, fz));
  AQB_TRY(alloc(&un1, fz)); AQB_TRY(alloc(&vn1, fz)); AQB_TRY(alloc(&wn1, fz));
  AQB_TRY(alloc(&un2, fz)); AQB_TRY(alloc(&vn2, fz)); AQB_TRY(alloc(&wn2, fz));
  AQB_TRY(alloc(&h1, fz)); AQB_TRY(alloc(&h2, fz));
  AQB_TRY(alloc(&type, c)); AQB_TRY(alloc(&density, c)); AQB_TRY(alloc(&div, c)); AQB_TRY(alloc(&rhs, c));
  AQB_TRY(alloc(&pa, c)); AQB_TRY(alloc(&pb, c)); AQB_TRY(alloc(&pcount, c));
  AQB_TRY(alloc(&bact, (size_t)NB)); AQB_TRY(alloc(&part_b2, (size_t)NB)); AQB_TRY(alloc(&part_nf, (size_t)NB));
  AQB_TRY(alloc(&rpart, (size_t)NRP));
  AQB_TRY(alloc(&ss, (size_t)ns)); AQB_TRY(alloc(&live, (size_t)ns));
  AQB_TRY(alloc(&scenes_d, (size_t)ns));
  AQB_TRY(alloc(&pre_d, 6 * (size_t)(ns + 1)));
  row_list_cap = 0;
  for (const SceneDesc& S : scenes) row_list_cap += batch_row_items(S.d, 1);  // one plane per item: the most items
  AQB_TRY(alloc(&row_list, (size_t)row_list_cap));
  AQB_TRY(alloc(&n_row_list, 1));
  AQB_CUDA(cudaMemcpyAsync(scenes_d, scenes.data(), sizeof(SceneDesc) * ns, cudaMemcpyHostToDevice, stream));
  std::vector<int> pre;
  for (const auto* v : {&pre_p, &pre_n, &pre_b, &pre_s, &pre_f}) pre.insert(pre.end(), v->begin(), v->end());
  pre.resize(6 * (size_t)(ns + 1), 0);
  AQB_CUDA(cudaMemcpyAsync(pre_d, pre.data(), sizeof(int) * pre.size(), cudaMemcpyHostToDevice, stream));
  AQB_CUDA(cudaStreamSynchronize(stream));
  bi.scenes = scenes_d;
  bi.n_scenes = ns;
  bi.particles = pre_d;
  bi.nodes = pre_d + (ns + 1);
  bi.bricks = pre_d + 2 * (ns + 1);
  bi.slayer = pre_d + 3 * (ns + 1);
  bi.flat = pre_d + 4 * (ns + 1);
  bi.rows = pre_d + 5 * (ns + 1);
  AQB_TRY(plan_clusters());
  return set_sweep_plan(xs, pipe);
}

// Sorts the scenes into clusters of 1 to 16 CTAs, if each fits one.
aq_status aq_batch::plan_clusters() {
  std::vector<std::vector<int>> by(kWidths);
  std::vector<int2> scratch((size_t)ns);
  long long units = 0, parts = 0;
  for (int s = 0; s < ns; ++s) {
    const SceneDesc& S = scenes[s];
    const int w = batch_cluster_width(S.d, S.n);
    if (w == 0) return AQ_OK;
    int k = 0;
    while ((1 << k) < w) ++k;
    by[k].push_back(s);
    cl_spill |= !cluster_solve_holds(S.d, w);
    cl_spill16 |= !cluster_solve_holds(S.d, 16);
    scratch[s] = make_int2((int)units, (int)parts);
    const long long u = cluster_solve_units(S.d);
    units += u;
    parts += u / 32 + 1;
  }
  for (int k = 0; k < kWidths; ++k)
    if ((!by[k].empty() || (cl_spill && k == kWidths - 1)) && !cluster_solve_runs(1 << k)) return AQ_OK;
  std::vector<int> order;
  for (int k = 0; k < kWidths; ++k) {
    std::stable_sort(by[k].begin(), by[k].end(), [&](int a, int b) { return scenes[a].n > scenes[b].n; });
    cl_first[k] = (int)order.size();
    order.insert(order.end(), by[k].begin(), by[k].end());
    if (!by[k].empty()) AQB_CUDA(cudaStreamCreateWithFlags(&cl_stream[k], cudaStreamNonBlocking));
  }
  cl_first[kWidths] = ns;
  for (cudaEvent_t& e : cl_event) AQB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  AQB_TRY(alloc(&cl_order, (size_t)ns));
  AQB_TRY(alloc(&cl_scratch, (size_t)ns));
  AQB_TRY(alloc(&cl_map, (size_t)units));
  AQB_TRY(alloc(&cl_list, (size_t)units));
  AQB_TRY(alloc(&cl_part, (size_t)parts));
  AQB_TRY(alloc(&cl_spilled, 2));
  AQB_CUDA(cudaMemcpyAsync(cl_order, order.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, stream));
  AQB_CUDA(cudaMemcpyAsync(cl_scratch, scratch.data(), sizeof(int2) * ns, cudaMemcpyHostToDevice, stream));
  AQB_CUDA(cudaStreamSynchronize(stream));
  cl_planned = clusters = true;
  return AQ_OK;
}

// The solves of all scenes; widest clusters first.
aq_status aq_batch::enq_clusters(unsigned long long spill) {
  const int fixed = solver.solve_mode == AQ_SOLVE_RESIDUAL ? 0 : solver.pressure_iterations;
  AQB_CUDA(cudaEventRecord(cl_event[kWidths], stream));
  for (int k = kWidths - 1; k >= 0; --k) {
    const int n = cl_first[k + 1] - cl_first[k];
    if (n == 0) continue;
    AQB_CUDA(cudaStreamWaitEvent(cl_stream[k], cl_event[kWidths], 0));
    AQB_CUDA(launch_batch_cluster_solve(cl_stream[k], bi, n, 1 << k, cl_order + cl_first[k], cl_scratch, live, pa, rhs,
                                        type, cl_map, cl_list, cl_part, ss, fixed, solver.check_interval,
                                        solver.max_iterations, (double)solver.rel_residual,
                                        spill ? cl_spilled : nullptr));
    AQB_CUDA(cudaEventRecord(cl_event[k], cl_stream[k]));
    AQB_CUDA(cudaStreamWaitEvent(stream, cl_event[k], 0));
  }
  if (spill) AQB_CUDA(launch_spill_condition(stream, cl_spilled, spill));
  return AQ_OK;
}

// The scenes still live, a cluster of 16 CTAs each; rows: the condition of the
// row sweeps (0: 16 CTAs hold every scene).
aq_status aq_batch::enq_wide_clusters(unsigned long long rows) {
  AQB_CUDA(launch_batch_cluster_solve(stream, bi, ns, 1 << (kWidths - 1), cl_order, cl_scratch, live, pa, rhs, type,
                                      cl_map, cl_list, cl_part, ss,
                                      solver.solve_mode == AQ_SOLVE_RESIDUAL ? 0 : solver.pressure_iterations,
                                      solver.check_interval, solver.max_iterations, (double)solver.rel_residual,
                                      rows ? cl_spilled + 1 : nullptr));
  if (rows) AQB_CUDA(launch_spill_condition(stream, cl_spilled + 1, rows));
  return AQ_OK;
}

// Packed-row Jacobi items depend on the x planes per item: rebuild their
// prefix sums (and the step graph).
aq_status aq_batch::set_sweep_plan(int planes, bool pipelined) {
  if (planes != 1 && planes != 2 && planes != 4 && planes != 8)
    return fail(AQ_ERR_INVALID_ARGUMENT, "x planes per sweep item must be 1, 2, 4 or 8");
  if (pipelined && planes == 1) return fail(AQ_ERR_INVALID_ARGUMENT, "pipelined sweeps need x planes > 1");
  xs = planes;
  pipe = pipelined;
  pre_r.assign(1, 0);
  for (const SceneDesc& S : scenes) pre_r.push_back(pre_r.back() + batch_row_items(S.d, xs));
  AQB_CUDA(cudaMemcpyAsync(pre_d + 5 * (ns + 1), pre_r.data(), sizeof(int) * (ns + 1), cudaMemcpyHostToDevice,
                           stream));
  AQB_TRY(enq_row_list());  // items depend on the plane count
  AQB_CUDA(cudaStreamSynchronize(stream));
  invalidate_graph();
  return AQ_OK;
}

// Copies the state a step carries over from a freshly initialised scene.
aq_status aq_batch::add_scene(int s, aq_fluid* f) {
  const SceneDesc& S = scenes[s];
  const size_t n = (size_t)S.n, c = (size_t)S.d.C, fz = (size_t)S.d.F;
  auto cp = [&](void* dst, const void* src, size_t bytes) -> aq_status {
    if (bytes) AQB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream));
    return AQ_OK;
  };
  const int p = S.p_off;
  AQB_TRY(cp(cur.px + p, f->cur.px, 4 * n)); AQB_TRY(cp(cur.py + p, f->cur.py, 4 * n));
  AQB_TRY(cp(cur.pz + p, f->cur.pz, 4 * n)); AQB_TRY(cp(cur.vx + p, f->cur.vx, 4 * n));
  AQB_TRY(cp(cur.vy + p, f->cur.vy, 4 * n)); AQB_TRY(cp(cur.vz + p, f->cur.vz, 4 * n));
  if (n) {
    kb_add_const<<<cdiv((int)n, 256), 256, 0, stream>>>(sort_index + p, f->sort_index, (int)n, p);
    AQB_CUDA(cudaGetLastError());
  }
  kb_add_const<<<cdiv((int)c + 1, 256), 256, 0, stream>>>(off + S.c_off, f->off, (int)c + 1, p);
  AQB_CUDA(cudaGetLastError());
  const int o = S.f_off;
  AQB_TRY(cp(u0 + o, f->u0, 4 * fz)); AQB_TRY(cp(v0 + o, f->v0, 4 * fz)); AQB_TRY(cp(w0 + o, f->w0, 4 * fz));
  AQB_TRY(cp(un1 + o, f->un1, 4 * fz)); AQB_TRY(cp(vn1 + o, f->vn1, 4 * fz)); AQB_TRY(cp(wn1 + o, f->wn1, 4 * fz));
  AQB_TRY(cp(un2 + o, f->un2, 4 * fz)); AQB_TRY(cp(vn2 + o, f->vn2, 4 * fz)); AQB_TRY(cp(wn2 + o, f->wn2, 4 * fz));
  AQB_TRY(cp(h1 + o, f->h1, fz)); AQB_TRY(cp(h2 + o, f->h2, fz));
  const int q = S.c_off;
  AQB_TRY(cp(type + q, f->type, c)); AQB_TRY(cp(density + q, f->density, 4 * c)); AQB_TRY(cp(div + q, f->div, 4 * c));
  AQB_TRY(cp(rhs + q, f->rhs, 4 * c)); AQB_TRY(cp(pa + q, f->pa, 4 * c)); AQB_TRY(cp(pb + q, f->pb, 4 * c));
  AQB_TRY(cp(pcount + q, f->pcount, 4 * c));
  AQB_TRY(cp(bact + S.br_off, f->bact, (size_t)f->nbricks));
  AQB_TRY(cp(ss + s, f->ss, sizeof(SolveState)));
  return AQ_OK;
}

// ------------------------------------------------------------------ stages
aq_status aq_batch::enq_sort() {
  const int tp = pre_p[ns];
  if (N > 0) {
    AQB_CUDA(launch_batch_particles_advance(stream, bi, tp, grid(), true, cur, tmp, u0, v0, w0, un2, vn2, wn2, key,
                                            slot, count));
    AQB_CUDA(launch_cell_scan(stream, C, count, off, tile_sums));
    AQB_CUDA(launch_scatter(stream, key, slot, off, perm_u, N));
    AQB_CUDA(launch_rank_gather(stream, false, key, off, perm_u, tmp, cur, sort_index, N));
  } else {
    AQB_CUDA(launch_cell_scan(stream, C, count, off, tile_sums));
  }
  return AQ_OK;
}

aq_status aq_batch::enq_pre_solve() {
  const int tn = pre_n[ns], tb = pre_b[ns], tsl = pre_s[ns];
  AQB_CUDA(launch_batch_p2g(stream, bi, tn, grid(), true, cur, off, u0, v0, w0, un1, vn1, wn1, type, density));
  AQB_CUDA(launch_batch_slayer(stream, bi, tsl, grid(), type, un2, vn2, wn2, un1, vn1, wn1, un2, vn2, wn2));
  AQB_CUDA(launch_batch_divergence(stream, bi, tb, grid512(), off, type, density, un1, vn1, wn1, pcount, div, rhs,
                                   pa, pb, solver.pressure_init == AQ_PRESSURE_ZERO, bact, part_b2, part_nf));
  AQB_CUDA(launch_batch_b2_finalize(stream, bi, part_b2, part_nf, ss, live));
  if (!clusters) AQB_TRY(enq_row_list());
  return AQ_OK;
}

// `sweeps` sweeps of every live scene from pa; the result of an even count
// ends in pa, of an odd count in pb.
aq_status aq_batch::enq_sweeps(int sweeps) {
  float* bufs[2] = {pa, pb};
  for (int k = 0; k < sweeps; ++k)
    AQB_CUDA(launch_batch_jacobi_rows(stream, bi, pre_r[ns], xs, pipe, grid(), live, bufs[k % 2], bufs[(k + 1) % 2],
                                      rhs, type, bact, row_list, n_row_list));
  return AQ_OK;
}

aq_status aq_batch::enq_solve_fixed() {
  const int K = solver.pressure_iterations;
  if (K <= 0) return AQ_OK;
  // an odd count sweeps from a copy in pb, so that it ends in pa, where the
  // scenes that are not live keep theirs
  if (K % 2) {
    kb_copy_f<<<cdiv(C, 256), 256, 0, stream>>>(pa, pb, C);
    AQB_CUDA(cudaGetLastError());
    std::swap(pa, pb);
  }
  const aq_status st = enq_sweeps(K);
  if (K % 2) std::swap(pa, pb);
  AQB_TRY(st);
  AQB_CUDA(launch_batch_resid_flat(stream, bi, pre_f[ns], grid(), live, pa, rhs, type, bact, rpart));
  AQB_CUDA(launch_batch_resid_finalize(stream, bi, rpart, ss, live, K, 0.0, 0));
  return AQ_OK;
}

aq_status aq_batch::enq_solve_body(unsigned long long handle) {
  const int m = solver.check_interval;  // even: the iterate ends in pa
  AQB_TRY(enq_sweeps(m));
  AQB_CUDA(launch_batch_resid_flat(stream, bi, pre_f[ns], grid(), live, pa, rhs, type, bact, rpart));
  AQB_CUDA(launch_batch_resid_finalize(stream, bi, rpart, ss, live, m, (double)solver.rel_residual,
                                       solver.max_iterations));
  AQB_CUDA(launch_batch_solve_condition(stream, live, ns, handle));
  return AQ_OK;
}

aq_status aq_batch::enq_post_solve() {
  const int tn = pre_n[ns];
  AQB_CUDA(launch_batch_project(stream, bi, tn, grid(), type, pa, density, un1, vn1, wn1, h1));
  // extrapolateVelocity: three ping-pong passes, 1 -> 2 -> 1 -> 2
  AQB_CUDA(launch_batch_extrapolate(stream, bi, tn, grid(), un1, vn1, wn1, h1, un2, vn2, wn2, h2));
  AQB_CUDA(launch_batch_extrapolate(stream, bi, tn, grid(), un2, vn2, wn2, h2, un1, vn1, wn1, h1));
  AQB_CUDA(launch_batch_extrapolate(stream, bi, tn, grid(), un1, vn1, wn1, h1, un2, vn2, wn2, h2));
  return AQ_OK;
}

aq_status aq_batch::build_graph() {
  invalidate_graph();
  return capture_step(true, true, &exec);
}

aq_status aq_batch::capture_step(bool sort, bool rest, cudaGraphExec_t* out) {
  cudaGraph_t g = nullptr;
  AQB_CUDA(cudaGraphCreate(&g, 0));
  // counted as the row sweeps run; the cluster solve does a step's blocks in
  // one launch per cluster width instead
  const int pre_launches = (N > 0 ? 6 : 3) + 5;  // sort; p2g, s-layer, divergence, b2, row list
  const int post_launches = 4;
  const bool residual = solver.solve_mode == AQ_SOLVE_RESIDUAL;
  const int K = residual ? 0 : std::max(0, solver.pressure_iterations);
  auto before_solve = [&]() -> aq_status {
    if (sort) AQB_TRY(enq_sort());
    return rest ? enq_pre_solve() : AQ_OK;
  };
  auto build = [&]() -> aq_status {
    if (!rest) return capture_into(stream, g, nullptr, 0, before_solve);
    body_launches = residual ? solver.check_interval + 3 : 0;
    graph_launches = pre_launches + post_launches + (K > 0 ? K + 2 + (K % 2) : 0);
    cudaGraphConditionalHandle spill = 0, rows = 0;
    cudaGraphNode_t node;
    cudaGraph_t body;
    const bool solve = residual || K > 0;
    step_launches = pre_launches + post_launches;
    if (clusters) {
      step_launches -= 1;  // no row list
      for (int k = 0; k < kWidths && solve; ++k) step_launches += cl_first[k + 1] > cl_first[k] ? 1 : 0;
      if (solve && cl_spill) step_launches += 1;  // their condition
    } else if (!residual) {
      step_launches = graph_launches;
    }
    if (solve && clusters && !cl_spill) {
      return capture_into(stream, g, nullptr, 0, [&]() -> aq_status {
        AQB_TRY(before_solve());
        AQB_TRY(enq_clusters(0));
        return enq_post_solve();
      });
    }
    if (!residual && !(solve && clusters)) {
      return capture_into(stream, g, nullptr, 0, [&]() -> aq_status {
        AQB_TRY(before_solve());
        AQB_TRY(enq_solve_fixed());
        return enq_post_solve();
      });
    }
    // conditional nodes, one behind the other: the scenes that spill go to
    // clusters of 16 CTAs, those that do not fit them to the row sweeps
    if (clusters) AQB_TRY(make_condition(g, 0, &spill));
    if (!clusters || cl_spill16) AQB_TRY(make_condition(g, clusters ? 0 : 1, &rows));
    AQB_TRY(capture_into(stream, g, nullptr, 0, [&]() -> aq_status {
      AQB_TRY(before_solve());
      return clusters ? enq_clusters(spill) : AQ_OK;
    }));
    if (clusters) {
      AQB_TRY(add_conditional(g, spill, false, &node, &body));
      AQB_TRY(capture_into(stream, body, nullptr, 0, [&]() { return enq_wide_clusters(rows); }));
    }
    if (rows) {
      AQB_TRY(add_conditional(g, rows, residual, &node, &body));
      AQB_TRY(capture_into(stream, body, nullptr, 0, [&]() -> aq_status {
        if (clusters) AQB_TRY(enq_row_list());
        return residual ? enq_solve_body(rows) : enq_solve_fixed();
      }));
    }
    return capture_into(stream, g, &node, 1, [&]() { return enq_post_solve(); });
  };
  const aq_status st = build();
  if (st != AQ_OK) { cudaGraphDestroy(g); return st; }
  cudaError_t e = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) { *out = nullptr; return fail(AQ_ERR_CUDA, std::string("instantiate: ") + cudaGetErrorString(e)); }
  return AQ_OK;
}

// ====================================================================== ABI
namespace {

bool same_solver(const aq_config& a, const aq_config& b) {
  return a.pressure_iterations == b.pressure_iterations && a.pressure_init == b.pressure_init &&
         a.solve_mode == b.solve_mode && a.rel_residual == b.rel_residual &&
         a.max_iterations == b.max_iterations && a.check_interval == b.check_interval && a.device == b.device &&
         a.stream == b.stream;
}

}  // namespace

extern "C" {

aq_status aq_batch_create(const aq_config* configs, int32_t n_scenes, aq_batch** out) {
  if (!out) return fail(AQ_ERR_INVALID_ARGUMENT, "out is NULL");
  *out = nullptr;
  if (!configs || n_scenes < 1) return fail(AQ_ERR_INVALID_ARGUMENT, "need at least one scene config");
  const aq_config& c0 = configs[0];
  long long C = 0, F = 0, NB = 0, NRP = 0;
  for (int s = 0; s < n_scenes; ++s) {
    const aq_config& c = configs[s];
    AQB_TRY(aq_config_validate(&c));
    if (c.size_z % 4 != 0) return fail(AQ_ERR_INVALID_CONFIG, "batched scenes need size_z % 4 == 0");
    if (!same_solver(c, c0))
      return fail(AQ_ERR_INVALID_CONFIG, "batched scenes must share the pressure solver settings, device and stream");
    for (int v = 1; v < c.volume_count; ++v)
      if (c.volumes[v].phase != c.volumes[0].phase)
        return fail(AQ_ERR_INVALID_CONFIG, "batched scenes must be single-phase");
    C += (long long)c.size_x * c.size_y * c.size_z;
    F += (long long)(c.size_x + 1) * (c.size_y + 1) * (c.size_z + 1);
    NB += (long long)cdiv(c.size_x, kBrick) * cdiv(c.size_y, kBrick) * cdiv(c.size_z, kBrick);
    NRP += (long long)((c.size_z / 4 + 31) / 32) * ((c.size_y + 7) / 8) * c.size_x;
  }
  if (c0.pressure_init == AQ_PRESSURE_LEARNED)
    return fail(AQ_ERR_INVALID_CONFIG, "batched scenes do not take the learned warm start");
  if (c0.solve_mode == AQ_SOLVE_RESIDUAL && c0.check_interval % 2 != 0)
    return fail(AQ_ERR_INVALID_CONFIG, "batched residual solves need an even check_interval");
  if (C + 1 >= (1LL << 31) || F >= (1LL << 31)) return fail(AQ_ERR_INVALID_CONFIG, "batch too large for 32-bit indices");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return fail(AQ_ERR_NO_DEVICE, "no CUDA device");
  }
  if (c0.device < 0 || c0.device >= ndev) return fail(AQ_ERR_INVALID_CONFIG, "device ordinal out of range");

  aq_batch* b = new aq_batch();
  b->device = c0.device;
  b->solver = c0;
  b->ns = n_scenes;
  auto bail = [&](aq_status st) {
    delete b;
    return st;
  };
  if (cudaSetDevice(b->device) != cudaSuccess) return bail(fail(AQ_ERR_CUDA, "cudaSetDevice"));
  if (c0.stream) {
    b->stream = (cudaStream_t)c0.stream;
  } else {
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess)
      return bail(fail(AQ_ERR_CUDA, "cudaStreamCreate"));
    b->own_stream = true;
  }
  cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device);
  b->C = (int)C;
  b->F = (int)F;
  b->NB = (int)NB;
  b->NRP = (int)NRP;

  // Each scene is created alone (seeding, initial sort and transfer), then
  // copied into the concatenated arrays; the scene fluids are released after.
  std::vector<aq_fluid*> fl((size_t)n_scenes, nullptr);
  auto release = [&]() {
    for (aq_fluid*& f : fl) {
      if (f) aq_fluid_destroy(f);
      f = nullptr;
    }
  };
  b->scenes.resize(n_scenes);
  b->cfgs.assign(configs, configs + n_scenes);
  b->time.assign(n_scenes, 0.0);
  b->phase.assign(n_scenes, 0);
  long long P = 0;
  int c_off = 0, f_off = 0, br_off = 0, rp_off = 0;
  b->pre_p.assign(1, 0); b->pre_n.assign(1, 0); b->pre_b.assign(1, 0); b->pre_s.assign(1, 0); b->pre_f.assign(1, 0);
  for (int s = 0; s < n_scenes; ++s) {
    aq_config c = configs[s];
    c.stream = b->stream;
    aq_status st = aq_fluid_create(&c, &fl[s]);
    if (st != AQ_OK) { release(); return bail(st); }
    const aq_fluid* f = fl[s];
    if (f->multiphase) {
      release();
      return bail(fail(AQ_ERR_INVALID_CONFIG, "batched scenes must be single-phase"));
    }
    SceneDesc& S = b->scenes[s];
    S.d = f->d;
    S.sp = f->sp;
    S.n = f->n;
    S.p_off = (int)P;
    S.c_off = c_off;
    S.f_off = f_off;
    S.br_off = br_off;
    S.rp_off = rp_off;
    b->phase[s] = f->phase;
    P += S.n;
    if (P >= (1LL << 31)) {
      release();
      return bail(fail(AQ_ERR_INVALID_CONFIG, "batch too large for 32-bit particle indices"));
    }
    const Dims& d = S.d;
    c_off += d.C;
    f_off += d.F;
    br_off += d.bx * d.by * d.bz;
    rp_off += resid_flat_parts(d);
    b->pre_p.push_back(b->pre_p.back() + cdiv(S.n, 256));
    b->pre_n.push_back(b->pre_n.back() + cdiv(d.sz, 32) * cdiv(d.sy, 8) * d.sx);
    b->pre_b.push_back(b->pre_b.back() + d.bx * d.by * d.bz);
    b->pre_s.push_back(b->pre_s.back() + cdiv(d.F - d.C, 256));
    b->pre_f.push_back(b->pre_f.back() + resid_flat_parts(d));
  }
  b->N = (int)P;
  aq_status st = b->allocate();
  for (int s = 0; s < n_scenes && st == AQ_OK; ++s) st = b->add_scene(s, fl[s]);
  if (st == AQ_OK) st = b->enq_row_list();  // the scenes' initial activity bricks
  if (st == AQ_OK && cudaStreamSynchronize(b->stream) != cudaSuccess)
    st = fail(AQ_ERR_CUDA, "batch initialisation failed");
  release();
  if (st != AQ_OK) return bail(st);

  *out = b;
  return AQ_OK;
}

aq_status aq_batch_step(aq_batch* b, int32_t n_steps) {
  if (!b || n_steps < 0) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  if (!b->exec) AQB_TRY(b->build_graph());
  for (int i = 0; i < n_steps; ++i) {
    AQB_CUDA(cudaGraphLaunch(b->exec, b->stream));
    for (int s = 0; s < b->ns; ++s) b->time[s] += (double)b->cfgs[s].timestep;
  }
  return AQ_OK;
}

aq_status aq_batch_step_host(aq_batch* b, int32_t n_steps, const float* pin, const float* vin, float* pout,
                             float* vout) {
  if (!b || n_steps < 0) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  const size_t N = (size_t)b->N;
  cudaStream_t s = b->stream;
  float* dp[3] = {b->cur.px, b->cur.py, b->cur.pz};
  float* dv[3] = {b->cur.vx, b->cur.vy, b->cur.vz};
  if (N) {
    for (int k = 0; k < 3; ++k) {
      if (pin) AQB_CUDA(cudaMemcpyAsync(dp[k], pin + k * N, 4 * N, cudaMemcpyHostToDevice, s));
      if (vin) AQB_CUDA(cudaMemcpyAsync(dv[k], vin + k * N, 4 * N, cudaMemcpyHostToDevice, s));
    }
  }
  // copies out go beside the rest of the last step, as aq_fluid_step_host's
  const size_t bytes = ((pout ? 12 : 0) + (vout ? 12 : 0)) * N;
  const bool split = n_steps > 0 && bytes >= kSplitBytes;
  cudaStream_t out = s;
  if (split) {
    if (!b->copy) {
      AQB_CUDA(cudaStreamCreateWithFlags(&b->copy, cudaStreamNonBlocking));
      AQB_CUDA(cudaEventCreateWithFlags(&b->sorted, cudaEventDisableTiming));
      AQB_CUDA(cudaEventCreateWithFlags(&b->copied, cudaEventDisableTiming));
    }
    if (n_steps > 1) AQB_TRY(aq_batch_step(b, n_steps - 1));
    if (!b->exec_sort) AQB_TRY(b->capture_step(true, false, &b->exec_sort));
    if (!b->exec_rest) AQB_TRY(b->capture_step(false, true, &b->exec_rest));
    AQB_CUDA(cudaGraphLaunch(b->exec_sort, s));
    AQB_CUDA(cudaEventRecord(b->sorted, s));
    AQB_CUDA(cudaGraphLaunch(b->exec_rest, s));
    for (int k = 0; k < b->ns; ++k) b->time[k] += (double)b->cfgs[k].timestep;
    AQB_CUDA(cudaStreamWaitEvent(b->copy, b->sorted, 0));
    out = b->copy;
  } else {
    AQB_TRY(aq_batch_step(b, n_steps));
  }
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 3 && N && e == cudaSuccess; ++k) {
    if (pout) e = cudaMemcpyAsync(pout + k * N, dp[k], 4 * N, cudaMemcpyDeviceToHost, out);
    if (vout && e == cudaSuccess) e = cudaMemcpyAsync(vout + k * N, dv[k], 4 * N, cudaMemcpyDeviceToHost, out);
  }
  if (split) {  // whatever follows on the batch's stream finds the copies done
    const cudaError_t r = cudaEventRecord(b->copied, b->copy);
    const cudaError_t w = cudaStreamWaitEvent(s, b->copied, 0);
    if (e == cudaSuccess) e = r != cudaSuccess ? r : w;
  }
  AQB_CUDA(e);
  AQB_CUDA(cudaStreamSynchronize(s));
  return AQ_OK;
}

aq_status aq_batch_stream(const aq_batch* b, void** stream) {
  if (!b || !stream) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  *stream = (void*)b->stream;
  return AQ_OK;
}

aq_status aq_batch_synchronize(aq_batch* b) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  cudaSetDevice(b->device);
  AQB_CUDA(cudaStreamSynchronize(b->stream));
  return AQ_OK;
}

int32_t aq_batch_scene_count(const aq_batch* b) { return b ? b->ns : 0; }

aq_status aq_batch_scene_info(const aq_batch* b, int32_t scene, int32_t size_xyz[3], int64_t* particle_count) {
  if (!b || scene < 0 || scene >= b->ns) return fail(AQ_ERR_INVALID_ARGUMENT, "bad scene index");
  const SceneDesc& S = b->scenes[scene];
  if (size_xyz) { size_xyz[0] = S.d.sx; size_xyz[1] = S.d.sy; size_xyz[2] = S.d.sz; }
  if (particle_count) *particle_count = S.n;
  return AQ_OK;
}

aq_status aq_batch_totals(const aq_batch* b, int64_t* cells, int64_t* nodes, int64_t* particles) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  if (cells) *cells = b->C;
  if (nodes) *nodes = b->F;
  if (particles) *particles = b->N;
  return AQ_OK;
}

aq_status aq_batch_download_scene(aq_batch* b, int32_t scene, aq_host_state* s) {
  if (!b || !s || scene < 0 || scene >= b->ns) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  const SceneDesc& S = b->scenes[scene];
  // A non-owning single-scene view of the scene's slices.
  aq_fluid v;
  v.cfg = b->cfgs[scene];
  v.device = b->device;
  v.stream = b->stream;
  v.d = S.d;
  v.sp = S.sp;
  v.n = S.n;
  v.multiphase = false;
  v.phase = b->phase[scene];
  v.time = b->time[scene];
  v.index_base = S.p_off;
  const int p = S.p_off, c = S.c_off, o = S.f_off;
  v.cur.px = b->cur.px + p; v.cur.py = b->cur.py + p; v.cur.pz = b->cur.pz + p;
  v.cur.vx = b->cur.vx + p; v.cur.vy = b->cur.vy + p; v.cur.vz = b->cur.vz + p;
  v.sort_index = b->sort_index + p;
  v.off = b->off + c;
  v.u0 = b->u0 + o; v.v0 = b->v0 + o; v.w0 = b->w0 + o;
  v.un1 = b->un1 + o; v.vn1 = b->vn1 + o; v.wn1 = b->wn1 + o;
  v.un2 = b->un2 + o; v.vn2 = b->vn2 + o; v.wn2 = b->wn2 + o;
  v.h1 = b->h1 + o; v.h2 = b->h2 + o;
  v.nv_cur = v.has_cur = 2;
  v.type = b->type + c; v.density = b->density + c; v.div = b->div + c; v.rhs = b->rhs + c;
  v.pa = b->pa + c; v.pb = b->pb + c; v.pcount = b->pcount + c;
  aq_status st = v.download(s);
  v.stream = nullptr;  // the view owns nothing
  v.device = -1;
  return st;
}

aq_status aq_batch_solve_stats(aq_batch* b, int32_t scene, aq_solve_stats* out) {
  if (!b || !out || scene < 0 || scene >= b->ns) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  SolveState s;
  AQB_CUDA(cudaStreamSynchronize(b->stream));
  AQB_CUDA(cudaMemcpy(&s, b->ss + scene, sizeof(SolveState), cudaMemcpyDeviceToHost));
  out->iterations = s.iterations;
  out->rel_residual = s.rel_residual;
  out->b_norm = s.b2 >= 0 ? sqrt(s.b2) : -1.0;
  out->fluid_cells = s.fluid_cells;
  out->converged = s.converged;
  out->blocks = s.bodies;
  out->total_sweeps = s.total_sweeps;
  out->total_blocks = s.total_bodies;
  out->warm_start = s.warm;
  out->warm_rel_residual = s.warm_rel;
  out->zero_rel_residual = s.zero_rel;
  return AQ_OK;
}

aq_status aq_batch_launch_counts(const aq_batch* b, int32_t* per_step, int32_t* per_block) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  if (!b->exec) AQB_TRY(const_cast<aq_batch*>(b)->build_graph());
  if (per_step) *per_step = b->graph_launches;
  if (per_block) *per_block = b->body_launches;
  return AQ_OK;
}

aq_status aq_batch_step_launches(const aq_batch* b, int32_t* launches) {
  if (!b || !launches) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  if (!b->exec) AQB_TRY(const_cast<aq_batch*>(b)->build_graph());
  *launches = b->step_launches;
  return AQ_OK;
}

aq_status aq_batch_set_cluster_solve(aq_batch* b, int32_t clusters) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  if (clusters && !b->cl_planned)
    return fail(AQ_ERR_INVALID_ARGUMENT, "a scene of the batch does not fit a thread-block cluster");
  cudaSetDevice(b->device);
  AQB_CUDA(cudaStreamSynchronize(b->stream));
  b->clusters = clusters != 0;
  b->invalidate_graph();
  return AQ_OK;
}

aq_status aq_batch_get_cluster_solve(const aq_batch* b, int32_t* clusters) {
  if (!b || !clusters) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  *clusters = b->clusters ? 1 : 0;
  return AQ_OK;
}

aq_status aq_batch_set_grid_multiple(aq_batch* b, int32_t multiple) {
  if (!b || multiple < 1 || multiple > 64) return fail(AQ_ERR_INVALID_ARGUMENT, "multiple must be in [1, 64]");
  b->multiple = multiple;
  b->invalidate_graph();
  return AQ_OK;
}

aq_status aq_batch_set_sweep_plan(aq_batch* b, int32_t x_planes, int32_t pipelined) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  cudaSetDevice(b->device);
  return b->set_sweep_plan(x_planes, pipelined != 0);
}

aq_status aq_batch_get_sweep_plan(const aq_batch* b, int32_t* x_planes, int32_t* pipelined) {
  if (!b) return fail(AQ_ERR_INVALID_ARGUMENT, "batch is NULL");
  if (x_planes) *x_planes = b->xs;
  if (pipelined) *pipelined = b->pipe ? 1 : 0;
  return AQ_OK;
}

aq_status aq_batch_autotune(aq_batch* b, int32_t sweeps_per_trial, int32_t* x_planes, int32_t* pipelined,
                            float* sweep_us) {
  if (!b || sweeps_per_trial < 2) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  int best = b->xs;
  bool best_pipe = b->pipe;
  float best_ms = -1.f;
  const int cand[][2] = {{1, 0}, {2, 0}, {4, 0}, {8, 0}, {2, 1}, {4, 1}, {8, 1}};
  for (const auto& c : cand) {
    AQB_TRY(b->set_sweep_plan(c[0], c[1] != 0));
    float ms = 0.f;
    AQB_TRY(aq_batch_benchmark_pressure(b, sweeps_per_trial, &ms, nullptr));
    if (best_ms < 0.f || ms < best_ms) {
      best_ms = ms;
      best = c[0];
      best_pipe = c[1] != 0;
    }
  }
  AQB_TRY(b->set_sweep_plan(best, best_pipe));
  if (x_planes) *x_planes = best;
  if (pipelined) *pipelined = best_pipe ? 1 : 0;
  if (sweep_us) *sweep_us = 1000.f * best_ms / (float)sweeps_per_trial;
  return AQ_OK;
}

aq_status aq_batch_benchmark_pressure(aq_batch* b, int32_t sweeps, float* ms, int64_t* cells_per_sweep) {
  if (!b || sweeps < 1) return fail(AQ_ERR_INVALID_ARGUMENT, "bad argument");
  cudaSetDevice(b->device);
  // every scene takes part
  std::vector<int> ones((size_t)b->ns, 1);
  AQB_CUDA(cudaMemcpyAsync(b->live, ones.data(), sizeof(int) * ones.size(), cudaMemcpyHostToDevice, b->stream));
  AQB_TRY(b->enq_row_list());  // the row sweeps are timed, whichever solve the steps use
  AQB_CUDA(cudaStreamSynchronize(b->stream));
  const int k = sweeps + (sweeps % 2);  // even: the iterate stays in pa
  AQB_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  aq_status st = b->enq_sweeps(k);
  cudaGraph_t g = nullptr;
  cudaError_t ce = cudaStreamEndCapture(b->stream, &g);
  if (st != AQ_OK) { if (g) cudaGraphDestroy(g); return st; }
  if (ce != cudaSuccess) return fail(AQ_ERR_CUDA, cudaGetErrorString(ce));
  cudaGraphExec_t ex = nullptr;
  ce = cudaGraphInstantiate(&ex, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) return fail(AQ_ERR_CUDA, cudaGetErrorString(ce));
  cudaEvent_t e0, e1;
  AQB_CUDA(cudaEventCreate(&e0));
  AQB_CUDA(cudaEventCreate(&e1));
  AQB_CUDA(cudaGraphLaunch(ex, b->stream));
  AQB_CUDA(cudaEventRecord(e0, b->stream));
  AQB_CUDA(cudaGraphLaunch(ex, b->stream));
  AQB_CUDA(cudaEventRecord(e1, b->stream));
  AQB_CUDA(cudaEventSynchronize(e1));
  cudaGraphExecDestroy(ex);
  float t = 0.f;
  AQB_CUDA(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ms) *ms = t * (float)sweeps / (float)k;
  if (cells_per_sweep) {
    std::vector<uint8_t> act((size_t)b->NB);
    AQB_CUDA(cudaMemcpy(act.data(), b->bact, act.size(), cudaMemcpyDeviceToHost));
    long long cells = 0;
    for (int s = 0; s < b->ns; ++s)
      cells += batch_row_cells_updated(b->scenes[s].d, b->xs, act.data() + b->scenes[s].br_off);
    *cells_per_sweep = cells;
  }
  return AQ_OK;
}

void aq_batch_destroy(aq_batch* b) { delete b; }

}  // extern "C"
