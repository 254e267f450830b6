// Batched A11 over many independent one-rank boxes (the batched and served
// forms).  A pt_batch is a pair of work-lists, one per precision, built once from
// a set of ops.  Boxes on layer tiles: every (problem, tile) in one launch and
// every run of nodes in a second.  Boxes on streaming tiles: every (problem,
// x-tile, row, z-chunk), one launch per non-empty (colour, tile width) class,
// the colours in a fixed order, and one for the Dirichlet rows.  A box is batched
// on the tiles of its own apply in that precision, so its result is bitwise the
// one it gets alone; boxes whose own applies use element matrices, and boxes with
// a z-chunk depth of the caller's, agree with it to rounding.
// Included from pt_b200.cu after struct pt_op.
#pragma once

#include <algorithm>
#include <map>
#include <vector>

struct pt_batch {
  int n;
  std::vector<pt_op *> ops;
  struct Cls {
    int px, py, pz, TX;
    int64_t off, count;
  };
  // One precision's work-list.  Layer tiles: (problem, tile) and (problem, first
  // node) lists, and the scratch that an apply takes from `lay_pool` on its
  // stream (applies on several streams each get their own).
  struct List {
    ptk::BatchProb *d_probs;
    int4 *d_items;
    int2 *d_lay;
    std::vector<Cls> classes;
    int64_t tiles, lay_tiles, lay_nodes, lay_values;
    int coloured;  // problems on coloured tiles
    bool borrowed; // items and lay lists are the other precision's
    // host copies, kept until destroy for the pooled batches' asynchronous uploads
    std::vector<ptk::BatchProb> h;
    std::vector<int4> hitems;
    std::vector<int2> hlay;
  } list[2];  // FP64, FP32
  cudaMemPool_t lay_pool;
  bool own_lay_pool;
  // pooled (server) batches: stream-ordered buffers
  cudaMemPool_t pool;
  cudaStream_t stream;
  template <typename T>
  const List &of() const { return list[sizeof(T) == 4]; }
};

namespace {

// programmatic: a class after the first of one apply may start on the SMs
// the previous class frees; the tile waits in-kernel before writing y (the
// classes of one apply read the same u, K and mask bits)
template <typename T, int TX, bool MASKED>
pt_status batch_launch_cls(const pt_batch::List &b, const pt_batch::Cls &c, const T *const *u, T *const *y, cudaStream_t st,
                           bool programmatic)
{
  constexpr size_t smem = ptk::stream_smem_bytes<T, TX>();
  pt_status as = kernel_attrs((const void *)ptk::a11_stream_batch_kernel<T, TX, MASKED>, smem);
  if (as != PT_OK) return as;
  const ptk::BatchProb *probs = b.d_probs;
  cudaLaunchAttribute pdl[1];
  pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c.count);
  cfg.blockDim = dim3(TX);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = programmatic ? pdl : nullptr;
  cfg.numAttrs = programmatic ? 1 : 0;
  const int4 *items = b.d_items + c.off;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, ptk::a11_stream_batch_kernel<T, TX, MASKED>, probs, items, c.px, c.py,
                                           c.pz, u, y);
  if (e != cudaSuccess) return fail(PT_ERR_CUDA, "batched kernel launch: %s", cudaGetErrorString(e));
  return PT_OK;
}

// Dirichlet rows of every masked problem after the colour passes: y_k = x_k
// (blockIdx.y = problem).
template <typename T>
__global__ void batch_bc_kernel(const ptk::BatchProb *__restrict__ probs, const T *const *__restrict__ uptr,
                                T *const *__restrict__ yptr)
{
  const ptk::BatchProb &p = probs[blockIdx.y];
  if (!p.mask || p.layer) return;
  const T *x = uptr[blockIdx.y];
  T *y = yptr[blockIdx.y];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.nvel; i += (int64_t)gridDim.x * blockDim.x)
    if (p.mask[i]) y[i] = x[i];
}

// The problems on layer tiles: every tile in one launch, every node in a second.
template <typename T, bool MASKED>
pt_status batch_apply_layers(pt_batch *b, const T *const *u, T *const *y, cudaStream_t st)
{
  constexpr size_t smem = ptk::layer_smem_bytes<T, LNT>();
  pt_status as = kernel_attrs((const void *)ptk::a11_layer_batch_kernel<T, LNT, MASKED>, smem);
  if (as != PT_OK) return as;
  const pt_batch::List &l = b->of<T>();
  const ptk::BatchProb *probs = l.d_probs;
  T *scratch = nullptr;
  PT_CUDA(cudaMallocFromPoolAsync((void **)&scratch, sizeof(T) * (size_t)l.lay_values, b->lay_pool, st));
  ptk::a11_layer_batch_kernel<T, LNT, MASKED><<<(unsigned)l.lay_tiles, LNT, smem, st>>>(probs, l.d_lay, u, scratch);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    cudaLaunchAttribute pdl[1];
    pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)l.lay_nodes);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = pdl;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, ptk::layer_gather_batch_kernel<T, LNT, MASKED>, probs,
                           (const int2 *)(l.d_lay + l.lay_tiles), u, (const T *)scratch, y);
  }
  cudaFreeAsync(scratch, st);
  if (e != cudaSuccess) return fail(PT_ERR_CUDA, "batched layer tiles: %s", cudaGetErrorString(e));
  return PT_OK;
}

// MASKED: the MatShell apply of every problem with a mask (columns inside the
// kernel, rows by one more launch; layer tiles set both).
template <typename T, bool MASKED>
pt_status batch_apply(pt_batch *b, const T *const *u, T *const *y, void *stream)
{
  if (!b || !u || !y) return fail(PT_ERR_BAD_ARG, "NULL argument");
  const cudaStream_t st = (cudaStream_t)stream;
  const pt_batch::List &l = b->of<T>();
  if (l.lay_tiles) {
    pt_status s = batch_apply_layers<T, MASKED>(b, u, y, st);
    if (s != PT_OK) return s;
  }
  bool first = true;
  for (const pt_batch::Cls &c : l.classes) {
    pt_status s;
    if (c.TX == 32) s = batch_launch_cls<T, 32, MASKED>(l, c, u, y, st, !first);
    else if (c.TX == 64) s = batch_launch_cls<T, 64, MASKED>(l, c, u, y, st, !first);
    else s = batch_launch_cls<T, 128, MASKED>(l, c, u, y, st, !first);
    if (s != PT_OK) return s;
    first = false;
  }
  if (MASKED && l.coloured) {
    batch_bc_kernel<T><<<dim3(32, (unsigned)b->n), 256, 0, st>>>(l.d_probs, u, y);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(PT_ERR_CUDA, "batched Dirichlet rows: %s", cudaGetErrorString(e));
  }
  return PT_OK;
}

// Launches of one masked apply.
int64_t batch_launches(const pt_batch *b, bool fp32)
{
  const pt_batch::List &l = b->list[fp32];
  return (int64_t)l.classes.size() + (l.lay_tiles ? 2 : 0) + (l.coloured ? 1 : 0);
}

bool batch_on_layers(int kernel) { return kernel == A11_LAYER || kernel == A11_EBE; }

void batch_list(int n, pt_op *const *ops, const int32_t *lz, int32_t tile_x, bool fp32, bool layers, pt_batch::List &l)
{
  // class key: (pass, TX) -> items
  std::map<std::pair<int, int>, std::vector<int4>> cls;
  std::vector<int2> lay_nodes;
  for (int i = 0; i < n; i++) {
    pt_op *op = ops[i];
    const int TX = tile_x ? tile_x : op->TX;
    ptk::BatchProb d;
    d.b = op->box;
    d.ntx = (op->mx + TX - 1) / TX;
    int L = (lz && lz[i] > 0) ? lz[i] : op->LZ;
    if (L > op->mz) L = op->mz;
    d.LZ = L;
    d.nzc = (op->mz + L - 1) / L;
    d.mask = op->has_mask ? op->d_mask : nullptr;
    d.mbits = op->has_mask ? op->d_mbits : nullptr;
    d.nvel = op->nvel;
    // layer tiles unless the caller asks for a z-chunk depth or there is no room
    // for their sums (a box whose own applies use element matrices too: they are
    // not batched)
    const int kernel = fp32 ? op->a11_kernel32 : op->a11_kernel;
    d.layer = layers && batch_on_layers(kernel) && !(lz && lz[i] > 0);
    d.lg = op->lg;
    d.lay_off = l.lay_values;
    d.K = fp32 ? (const void *)op->d_K32 : (const void *)op->d_K;
    l.h.push_back(d);
    if (d.layer) {
      const int64_t nt = op->lg.tiles;
      l.lay_values += nt * ptk::LayerLayout<LNT>::TILE;
      for (int64_t k = 0; k < nt; k++) l.hlay.push_back(make_int2(i, (int)k));
      for (int64_t k = 0; k < (int64_t)op->lg.nodes(); k += ptk::LAYER_GATHER_NODES) lay_nodes.push_back(make_int2(i, (int)k));
      continue;
    }
    l.coloured++;
    for (int zc = 0; zc < d.nzc; zc++)
      for (int ej = 0; ej < op->my; ej++)
        for (int tx = 0; tx < d.ntx; tx++) {
          const int pass = (tx & 1) + 2 * (ej & 1) + 4 * (zc & 1);
          cls[{pass, TX}].push_back(make_int4(i, tx, ej, zc));
        }
  }
  l.lay_tiles = (int64_t)l.hlay.size();
  l.lay_nodes = (int64_t)lay_nodes.size();
  l.hlay.insert(l.hlay.end(), lay_nodes.begin(), lay_nodes.end());
  for (auto &kv : cls) {
    pt_batch::Cls c;
    c.px = kv.first.first & 1; c.py = (kv.first.first >> 1) & 1; c.pz = (kv.first.first >> 2) & 1;
    c.TX = kv.first.second;
    c.off = (int64_t)l.hitems.size();
    c.count = (int64_t)kv.second.size();
    l.hitems.insert(l.hitems.end(), kv.second.begin(), kv.second.end());
    l.classes.push_back(c);
  }
  l.tiles = l.lay_tiles + (int64_t)l.hitems.size();
}

// A list's array on the device: from the batch's pool and asynchronous, or
// cudaMalloc and a synchronous copy.
template <typename V>
cudaError_t batch_upload(const pt_batch *b, V **p, const std::vector<V> &h)
{
  const size_t bytes = sizeof(V) * h.size();
  if (!bytes) return cudaSuccess;
  cudaError_t e = b->pool ? cudaMallocFromPoolAsync((void **)p, bytes, b->pool, b->stream) : cudaMalloc(p, bytes);
  if (e != cudaSuccess) return e;
  return b->pool ? cudaMemcpyAsync(*p, h.data(), bytes, cudaMemcpyHostToDevice, b->stream)
                 : cudaMemcpy(*p, h.data(), bytes, cudaMemcpyHostToDevice);
}

}  // namespace

extern "C" {

// pool == null: cudaMalloc + synchronous upload; else buffers from `pool`
// with asynchronous uploads, both ordered on `stream`.
static pt_status batch_create_impl(int n, pt_op *const *ops, const int32_t *lz, int32_t tile_x, cudaMemPool_t pool,
                                   cudaStream_t stream, pt_batch **out, bool layers = true)
{
  if (!out || n < 1 || !ops) return fail(PT_ERR_BAD_ARG, "need n >= 1 ops");
  if (tile_x != 0 && tile_x != 32 && tile_x != 64 && tile_x != 128)
    return fail(PT_ERR_BAD_ARG, "tile_x must be 0, 32, 64 or 128");
  *out = nullptr;
  for (int i = 0; i < n; i++) {
    pt_op *op = ops[i];
    pt_status s = check_ready(op, true);
    if (s != PT_OK) return s;
    if (!op->full_box) return fail(PT_ERR_UNSUPPORTED, "batch problem %d: one-rank boxes only", i);
    if ((s = ensure_geometry(op)) != PT_OK) return s;
    if (!op->geom_ok) return fail(PT_ERR_BAD_ARG, "batch problem %d has w*eta/detJ <= 0 somewhere", i);
    if (op->has_mask && !op->d_mbits) return fail(PT_ERR_STATE, "batch problem %d: mask without its packed bits", i);
  }
  pt_batch *b = new (std::nothrow) pt_batch();
  if (!b) return fail(PT_ERR_OOM, "host allocation failed");
  b->n = n;
  b->ops.assign(ops, ops + n);
  b->pool = pool;
  b->stream = stream;
  cudaError_t e = cudaSuccess;
  // one list for both precisions (but for K) where every op takes the same tiles in both
  const bool one = std::all_of(ops, ops + n, [](const pt_op *op) {
    return batch_on_layers(op->a11_kernel) == batch_on_layers(op->a11_kernel32);
  });
  for (int f = 0; f < 2; f++) {
    pt_batch::List &l = b->list[f];
    if (f && one) {
      const pt_batch::List &o = b->list[0];
      l.d_items = o.d_items; l.d_lay = o.d_lay;
      l.classes = o.classes;
      l.tiles = o.tiles; l.lay_tiles = o.lay_tiles; l.lay_nodes = o.lay_nodes; l.lay_values = o.lay_values;
      l.coloured = o.coloured;
      l.borrowed = true;
      l.h = o.h;
      for (int i = 0; i < n; i++) l.h[i].K = ops[i]->d_K32;
      if (e == cudaSuccess) e = batch_upload(b, &l.d_probs, l.h);
      break;
    }
    batch_list(n, ops, lz, tile_x, f != 0, layers, l);
    if (e == cudaSuccess) e = batch_upload(b, &l.d_probs, l.h);
    if (e == cudaSuccess) e = batch_upload(b, &l.d_items, l.hitems);
    if (e == cudaSuccess) e = batch_upload(b, &l.d_lay, l.hlay);
  }
  const size_t scratch = std::max(sizeof(double) * (size_t)b->list[0].lay_values, sizeof(float) * (size_t)b->list[1].lay_values);
  if (pool) b->lay_pool = pool;
  else if (scratch) {
    cudaMemPoolProps pp{};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    if (e == cudaSuccess) e = cudaGetDevice(&pp.location.id);
    if (e == cudaSuccess) e = cudaMemPoolCreate(&b->lay_pool, &pp);
    if (e == cudaSuccess) {
      b->own_lay_pool = true;
      uint64_t keep = UINT64_MAX;  // kept from apply to apply, given back with the batch
      e = cudaMemPoolSetAttribute(b->lay_pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    // one apply's scratch is there before the first apply
    void *first = nullptr;
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&first, scratch, b->lay_pool, stream);
    if (e == cudaErrorMemoryAllocation) {  // no room for the sums: all boxes on streaming tiles
      cudaGetLastError();
      pt_batch_destroy(b);
      return batch_create_impl(n, ops, lz, tile_x, pool, stream, out, false);
    }
    if (e == cudaSuccess) e = cudaFreeAsync(first, stream);
  }
  if (e != cudaSuccess) {
    pt_status s = fail(e == cudaErrorMemoryAllocation ? PT_ERR_OOM : PT_ERR_CUDA, "pt_batch_create: %s",
                       cudaGetErrorString(e));
    pt_batch_destroy(b);
    return s;
  }
  *out = b;
  return PT_OK;
}

pt_status pt_batch_create_tiled(int n, pt_op *const *ops, const int32_t *lz, int32_t tile_x, pt_batch **out)
{
  return batch_create_impl(n, ops, lz, tile_x, nullptr, nullptr, out);
}

pt_status pt_batch_create(int n, pt_op *const *ops, const int32_t *lz, pt_batch **out)
{
  return batch_create_impl(n, ops, lz, 0, nullptr, nullptr, out);
}

pt_status pt_batch_destroy(pt_batch *b)
{
  if (!b) return PT_OK;
  for (const pt_batch::List &l : b->list) {
    void *bufs[] = {l.d_probs, l.borrowed ? nullptr : l.d_items, l.borrowed ? nullptr : l.d_lay};
    for (void *p : bufs) {
      if (!p) continue;
      if (b->pool) cudaFreeAsync(p, b->stream);
      else cudaFree(p);
    }
  }
  if (b->own_lay_pool) cudaMemPoolDestroy(b->lay_pool);
  delete b;
  return PT_OK;
}

int64_t pt_batch_launches_per_apply(const pt_batch *b)
{
  return b ? (int64_t)b->list[0].classes.size() + (b->list[0].lay_tiles ? 2 : 0) : 0;
}
int64_t pt_batch_tiles(const pt_batch *b) { return b ? b->list[0].tiles : 0; }

pt_status pt_batch_a11_apply_d(pt_batch *b, const double *const *u, double *const *y, int masked, void *stream)
{
  return masked ? batch_apply<double, true>(b, u, y, stream) : batch_apply<double, false>(b, u, y, stream);
}

pt_status pt_batch_a11_apply_f32_d(pt_batch *b, const float *const *u, float *const *y, int masked, void *stream)
{
  return masked ? batch_apply<float, true>(b, u, y, stream) : batch_apply<float, false>(b, u, y, stream);
}

}  // extern "C"
