// Python bindings of the sm_100a kernels (module tensornet_b200._ext._tn_cuda).
// Storage is owned by torch tensors created on the Python side; the objects here only keep
// raw device pointers (plus a reference to the tensors) so a kernel launch costs one call.
#include <torch/extension.h>
#include <ATen/cuda/CachingHostAllocator.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <vector>

#include "gemm_tcgen05.h"
#include "mlp_fused.h"
#include "tn_ops.h"
#include "tn_types.h"

namespace py = pybind11;

namespace {

template <typename T>
T* ptr_of(const at::Tensor& t) { return reinterpret_cast<T*>(t.data_ptr()); }
template <typename T>
T* ptr_of(int64_t p) { return reinterpret_cast<T*>(static_cast<uintptr_t>(p)); }

// Every binding that launches a kernel fetches the stream exactly once, so this doubles as the
// count of kernels this library has launched (or recorded into a CUDA graph).
std::atomic<long long> g_launches{0};
cudaStream_t cur_stream() {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return at::cuda::getCurrentCUDAStream().stream();
}

void check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  cudaGetLastError();      // told here: the next check of a launch is not to find it again
  throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

tn::SparseOptParams opt_from_dict(const py::dict& d) {
  tn::SparseOptParams o{};
  o.kind = d["kind"].cast<int>();
  o.lr = d["lr"].cast<float>();
  o.eps = d["eps"].cast<float>();
  o.beta1 = d["beta1"].cast<float>();
  o.beta2 = d["beta2"].cast<float>();
  o.initial_g2sum = d["initial_g2sum"].cast<float>();
  o.initial_scale = d["initial_scale"].cast<float>();
  o.ftrl_beta = d["ftrl_beta"].cast<float>();
  o.lambda1 = d["lambda1"].cast<float>();
  o.lambda2 = d["lambda2"].cast<float>();
  o.zero_init = d["zero_init"].cast<int>();
  o.seed = d["seed"].cast<uint64_t>();
  return o;
}

tn::TableView table_from_dict(const py::dict& d) {
  tn::TableView t{};
  t.keys = ptr_of<unsigned long long>(d["keys"].cast<at::Tensor>());
  t.slots = ptr_of<int>(d["slots"].cast<at::Tensor>());
  t.rows = ptr_of<float>(d["rows"].cast<at::Tensor>());
  t.row_keys = ptr_of<unsigned long long>(d["row_keys"].cast<at::Tensor>());
  t.row_tag = ptr_of<unsigned long long>(d["row_tag"].cast<at::Tensor>());
  t.n_rows = ptr_of<int>(d["n_rows"].cast<at::Tensor>());
  int64_t cap = d["keys"].cast<at::Tensor>().numel();
  TORCH_CHECK(cap > 0 && (cap & (cap - 1)) == 0, "table capacity must be a power of two");
  t.cap_mask = (unsigned)(cap - 1);
  t.row_cap = (int)d["row_keys"].cast<at::Tensor>().numel();
  t.dim = d["dim"].cast<int>();
  t.stride = d["stride"].cast<int>();
  t.use_cvm = d["use_cvm"].cast<int>();
  return t;
}

// One embedding table + its exchange buffers.
struct SparseCtx {
  tn::SparseCommView c{};
  tn::TableView t{};
  tn::SparseOptParams o{};
  int pull_lanes = 1, push_lanes = 1;
  int tile_rows = 0;   // staged row return of the pull (0 = rows go straight to the requester's matrix)
  py::dict keep;   // keeps the tensors alive
  at::Tensor tbl_dev;  // the table descriptor in device memory (what launches inside CUDA graphs read)

  void upload_table() {
    if (!tbl_dev.defined()) {
      at::Tensor rows = keep["table"].cast<py::dict>()["rows"].cast<at::Tensor>();
      tbl_dev = at::empty({(int64_t)((sizeof(tn::TableView) + 7) / 8)}, at::TensorOptions().dtype(at::kLong).device(rows.device()));
    }
    // stream-ordered with the launches around it; the source is copied out before the call returns (pageable memory)
    check(cudaMemcpyAsync(tbl_dev.data_ptr(), &t, sizeof(tn::TableView), cudaMemcpyHostToDevice, at::cuda::getCurrentCUDAStream().stream()),
          "table descriptor upload");
  }

  SparseCtx(py::dict table, py::dict comm, py::dict opt) {
    keep["table"] = table; keep["comm"] = comm;
    t = table_from_dict(table);
    upload_table();
    o = opt_from_dict(opt);
    c.world = comm["world"].cast<int>();
    c.rank = comm["rank"].cast<int>();
    c.capo = comm["capo"].cast<int>();
    c.gstride = comm["gstride"].cast<int>();
    c.ustride = comm["ustride"].cast<int>();
    TORCH_CHECK(c.world >= 1 && c.world <= tn::kMaxWorld, "world must be 1..8");
    TORCH_CHECK(c.capo % 4 == 0, "segment capacity must be a multiple of 4");
    auto inbox = comm["inbox_ids"].cast<std::vector<int64_t>>();
    auto gU_peer = comm["gU_peer"].cast<std::vector<int64_t>>();
    auto cnts_peer = comm["cnts_peer"].cast<std::vector<int64_t>>();
    auto U = comm["U"].cast<std::vector<int64_t>>();
    auto sig = comm["sig"].cast<std::vector<int64_t>>();
    TORCH_CHECK((int)inbox.size() == c.world && (int)gU_peer.size() == c.world && (int)cnts_peer.size() == c.world && (int)U.size() == c.world &&
                    (int)sig.size() == c.world, "peer pointer tables must have `world` entries");
    for (int p = 0; p < c.world; ++p) {
      c.inbox_ids[p] = ptr_of<unsigned long long>(inbox[p]);
      c.gU_peer[p] = ptr_of<float>(gU_peer[p]);
      c.cnts_peer[p] = ptr_of<float>(cnts_peer[p]);
      c.U[p] = ptr_of<float>(U[p]);
      c.sig[p] = ptr_of<unsigned long long>(sig[p]);
    }
    c.stage_ids = ptr_of<unsigned long long>(comm["stage_ids"].cast<at::Tensor>());
    c.gU = ptr_of<float>(comm["gU"].cast<at::Tensor>());
    c.cnts = ptr_of<float>(comm["cnts"].cast<at::Tensor>());
    c.cnt = ptr_of<int>(comm["cnt"].cast<at::Tensor>());
    c.cnt_saved = ptr_of<int>(comm["cnt_saved"].cast<at::Tensor>());
    c.req_n = ptr_of<int>(comm["req_n"].cast<at::Tensor>());
    c.req_row = ptr_of<int>(comm["req_row"].cast<at::Tensor>());
    c.req_ou = ptr_of<int>(comm["req_ou"].cast<at::Tensor>());
    c.ou_row = ptr_of<int>(comm["ou_row"].cast<at::Tensor>());
    c.ocount = ptr_of<int>(comm["ocount"].cast<at::Tensor>());
    c.acc = ptr_of<float>(comm["acc"].cast<at::Tensor>());
    at::Tensor ddk = comm["dd_keys"].cast<at::Tensor>();
    int64_t ddcap = ddk.numel();
    TORCH_CHECK(ddcap >= 2 && (ddcap & (ddcap - 1)) == 0, "dedup scratch must be a power of two");
    c.dd_keys = ptr_of<unsigned long long>(ddk);
    c.dd_vals = ptr_of<int>(comm["dd_vals"].cast<at::Tensor>());
    c.dd_mask = (unsigned)(ddcap - 1);
    c.epoch = ptr_of<unsigned long long>(comm["epoch"].cast<at::Tensor>());
    c.bar = ptr_of<unsigned>(comm["bar"].cast<at::Tensor>());
    c.status = ptr_of<int>(comm["status"].cast<at::Tensor>());
    c.wait_ns = comm["wait_ns"].cast<uint64_t>();
    c.prof = comm.contains("prof") && !comm["prof"].is_none() ? ptr_of<unsigned long long>(comm["prof"].cast<at::Tensor>()) : nullptr;
    pull_lanes = tn::lanes_for_width_host((c.ustride + 3) / 4);   // each lane keeps up to four 16-byte chunks in flight
    {
      // Lanes per row in the row update.  Fewer lanes per row = more rows in flight per warp, which is what the
      // update is short of (dependent random accesses): with 1 M ids per batch, two 16-byte chunks per lane take the
      // push from 169 to 131 us at dim 64 and four from 318 to 233 us at dim 128; short rows (dim 20) are best at one.
      const int cpl = t.dim >= 128 ? 4 : (t.dim >= 32 ? 2 : 1);
      push_lanes = tn::lanes_for_width_host((t.dim + cpl - 1) / cpl);
    }
    if (!comm.contains("staged_return") || comm["staged_return"].cast<bool>()) {
      // rows per tile: whole 128-byte lines per tile, about 4 KiB of shared memory per warp at most
      int tr = 32;
      while (tr > 8 && tr * c.ustride * 4 > 4096) tr >>= 1;
      const int rpp = 32 / pull_lanes;
      const bool fits = (size_t)tr * c.ustride * 4 * 32 <= 160 * 1024;
      if (fits && tr % rpp == 0 && c.capo % tr == 0 && (tr * c.ustride * 4) % 128 == 0) tile_rows = tr;
    }
  }

  void set_opt(py::dict opt) { o = opt_from_dict(opt); }
  // The shard's arrays were replaced (growth, compaction): launches already recorded in CUDA graphs pick the new ones up.
  void set_table(py::dict table) { keep["table"] = table; t = table_from_dict(table); upload_table(); }

  // One GPU: the pull is ordinary kernels, and pooling reads the rows where they are (staged returns keep the exchange kernel).
  bool in_place() const { return c.world == 1 && tile_rows == 0; }

  // `req`: rows of the batch's distinct signs, for a batch whose pull started ahead of its step (in place only)
  int* req_ptr(const c10::optional<at::Tensor>& req) const {
    if (!req.has_value()) return c.req_row;
    TORCH_CHECK(in_place() && req->is_cuda() && req->scalar_type() == at::kInt && req->numel() >= c.capo, "req: int32, one per distinct sign");
    return ptr_of<int>(*req);
  }
  tn::PullArgs pull_args(const at::Tensor& ids, const at::Tensor& inverse, const c10::optional<at::Tensor>& req) const {
    TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous(), "ids: contiguous int64 CUDA tensor");
    TORCH_CHECK(inverse.scalar_type() == at::kInt && inverse.numel() >= ids.numel(), "inverse: int32, one per id");
    tn::PullArgs a{};
    a.c = c; a.tbl = t; a.opt = o;
    a.c.req_row = req_ptr(req);
    a.tbl_dev = reinterpret_cast<const tn::TableView*>(tbl_dev.data_ptr());
    a.ids = ptr_of<const long long>(ids);
    a.n_ids = (int)ids.numel();
    a.inverse = ptr_of<int>(inverse);
    a.lanes = pull_lanes;
    return a;
  }

  // The part of a batch's pull that needs only its ids, ahead of its step (plain kernels on the current stream).
  void front(at::Tensor ids, at::Tensor inverse, c10::optional<at::Tensor> req) {
    c10::cuda::CUDAGuard guard(ids.device());
    tn::PullArgs a = pull_args(ids, inverse, req);
    a.training = 1;
    a.front_done = 1;
    check(in_place() ? tn::launch_sparse_pull_local_front(a, cur_stream()) : tn::launch_sparse_pull_front(a, cur_stream()),
          "sparse_pull_front launch");
    g_launches.fetch_add(1, std::memory_order_relaxed);      // two kernels
  }

  static const int* count_ptr(const c10::optional<at::Tensor>& n_dev) {
    if (!n_dev.has_value()) return nullptr;
    TORCH_CHECK(n_dev->is_cuda() && n_dev->scalar_type() == at::kInt && n_dev->numel() == 1, "n_dev: one int32 on the device");
    return ptr_of<const int>(*n_dev);
  }
  tn::PullArgs batch_args(const at::Tensor& ids, const at::Tensor& inverse, const c10::optional<at::Tensor>& labels, int label_mod,
                          bool training, bool lookup_only, bool front_done, const c10::optional<at::Tensor>& n_dev,
                          const c10::optional<at::Tensor>& req) const {
    tn::PullArgs a = pull_args(ids, inverse, req);
    a.n_dev = count_ptr(n_dev);
    a.labels = labels.has_value() ? ptr_of<const float>(*labels) : nullptr;
    a.label_mod = label_mod;
    a.training = training ? 1 : 0;
    a.lookup_only = lookup_only ? 1 : 0;
    TORCH_CHECK(!(training && lookup_only), "a training pull creates rows; lookup_only is for inference");
    a.front_done = front_done ? 1 : 0;
    return a;
  }
  // `rows`: the pulled rows are wanted in the per-batch matrix (always the case where they are not read in place)
  void pull(at::Tensor ids, at::Tensor inverse, c10::optional<at::Tensor> labels, int label_mod, bool training, bool lookup_only,
            bool front_done, c10::optional<at::Tensor> n_dev, bool rows, c10::optional<at::Tensor> req) {
    c10::cuda::CUDAGuard guard(ids.device());
    tn::PullArgs a = batch_args(ids, inverse, labels, label_mod, training, lookup_only, front_done, n_dev, req);
    if (in_place()) {
      check(tn::launch_sparse_pull_local(&a, 1, cur_stream()), "sparse_pull_local launch");
      if (!front_done) g_launches.fetch_add(1, std::memory_order_relaxed);
      if (rows) check(tn::launch_sparse_pull_local_rows(a, cur_stream()), "sparse_pull_local_rows launch");
      return;
    }
    a.tile_rows = tile_rows;
    long long work = (long long)a.n_ids * (pull_lanes > 4 ? pull_lanes / 2 : 2);
    if (work > (1ll << 30)) work = 1ll << 30;
    check(tn::launch_sparse_pull(a, (int)work, cur_stream()), "sparse_pull_fused launch");
  }

  // The rows of the last pull as the pooling kernels are to read them.
  // `direct`: positions are rows (lookup_many).
  tn::RowSource source(const c10::optional<at::Tensor>& req, bool direct) const {
    tn::RowSource s{};
    s.U = c.U[c.rank];
    s.ustride = c.ustride;
    TORCH_CHECK(!direct || in_place(), "direct rows: one GPU");
    if (in_place()) {
      s.row_of = direct ? nullptr : req_ptr(req);
      s.tbl = reinterpret_cast<const tn::TableView*>(tbl_dev.data_ptr());
    }
    s.stride = t.stride;
    s.dim = t.dim;
    s.cvm = !t.use_cvm ? 0 : o.kind == tn::kAdaGrad ? 1 : 2;
    return s;
  }

  // `dense`: the dense step of the same training step (DenseCtx::rider_args), carried by a few CTAs of this launch.
  void push(int64_t work_hint, int max_ctas, const tn::DenseStepArgs* dense, const c10::optional<at::Tensor>& req) {
    tn::PushArgs a{};
    a.c = c; a.tbl = t; a.opt = o; a.lanes = push_lanes;
    a.c.req_row = req_ptr(req);
    a.tbl_dev = reinterpret_cast<const tn::TableView*>(tbl_dev.data_ptr());
    long long work = work_hint * push_lanes;
    if (work > (1ll << 30)) work = 1ll << 30;
    check(tn::launch_sparse_push(a, (int)work, max_ctas, dense, cur_stream()), "sparse_push_fused launch");
  }
};

struct DenseCtx {
  tn::DenseStepArgs a{};
  py::dict keep;
  DenseCtx(py::dict d) {
    keep = d;
    a.opt.kind = d["kind"].cast<int>();
    a.opt.beta1 = d["beta1"].cast<float>();
    a.opt.beta2 = d["beta2"].cast<float>();
    a.opt.eps = d["eps"].cast<float>();
    a.opt.grad_decay = d["grad_decay"].cast<float>();
    a.opt.mom_decay = d["mom_decay"].cast<float>();
    a.opt.state = ptr_of<float>(d["state"].cast<at::Tensor>());
    a.n = d["n"].cast<long long>();
    a.chunk = d["chunk"].cast<long long>();
    a.world = d["world"].cast<int>();
    a.rank = d["rank"].cast<int>();
    a.grad_scale = d["grad_scale"].cast<float>();
    // small arrays: the owner re-zeroes every replica's gradient through the switch (no extra grid barrier);
    // large ones: each GPU clears its own replica after the closing barrier (no NVLink bytes)
    a.gated = d.contains("gated") ? d["gated"].cast<int>() : 0;
    a.zero_local = d.contains("zero_local") ? d["zero_local"].cast<int>() : (a.world > 1 && a.n > (1ll << 21) ? 1 : 0);
    auto W = d["W"].cast<std::vector<int64_t>>();
    auto G = d["G"].cast<std::vector<int64_t>>();
    auto Wb = d["Wb"].cast<std::vector<int64_t>>();
    auto sig = d["sig"].cast<std::vector<int64_t>>();
    TORCH_CHECK((int)W.size() == a.world && (int)G.size() == a.world && (int)Wb.size() == a.world, "peer tables");
    for (int p = 0; p < a.world; ++p) {
      a.W[p] = ptr_of<float>(W[p]); a.G[p] = ptr_of<float>(G[p]); a.Wb[p] = ptr_of<void>(Wb[p]);
      a.sig[p] = p < (int)sig.size() ? ptr_of<unsigned long long>(sig[p]) : nullptr;
    }
    a.W_mc = ptr_of<float>(d["W_mc"].cast<int64_t>());
    a.G_mc = ptr_of<float>(d["G_mc"].cast<int64_t>());
    a.Wb_mc = ptr_of<void>(d["Wb_mc"].cast<int64_t>());
    a.s0 = ptr_of<float>(d["s0"].cast<at::Tensor>());
    a.s1 = ptr_of<float>(d["s1"].cast<at::Tensor>());
    a.s2 = d.contains("s2") && !d["s2"].is_none() ? ptr_of<float>(d["s2"].cast<at::Tensor>()) : nullptr;
    a.epoch = ptr_of<unsigned long long>(d["epoch"].cast<at::Tensor>());
    a.bar = ptr_of<unsigned>(d["bar"].cast<at::Tensor>());
    a.status = ptr_of<int>(d["status"].cast<at::Tensor>());
    a.wait_ns = d["wait_ns"].cast<uint64_t>();
  }
  void step(bool skip_open) {
    tn::DenseStepArgs b = a;
    b.skip_open = skip_open ? 1 : 0;
    check(tn::launch_dense_step(b, cur_stream()), "dense step launch");
  }
  // Arguments for a launch in which the sparse push kernel carries this step: the opening "gradients ready"
  // barrier is always run (the carrying CTAs start together with the push, before any peer has been heard from).
  tn::DenseStepArgs rider_args() const {
    tn::DenseStepArgs b = a;
    b.skip_open = 0;
    return b;
  }
  void set_gated(bool g) { a.gated = g ? 1 : 0; }
  void set_max_ctas(int n) { a.max_ctas = n; }
};

// Device-resident batch-norm table and the per-step kernels of the layer.
struct BnCtx {
  tn::BnTableView t{};
  tn::BnSyncView s{};
  bool has_sync = false;
  double* batch = nullptr;     // [3][C] per-step scratch, kept zero between steps
  double* scratch = nullptr;   // [3][C] sum of the peers' increments during an exchange
  py::dict keep;
  BnCtx(py::dict d) {
    keep = d;
    t.C = d["C"].cast<int>();
    t.pctr = d["pctr"].cast<int>();
    t.moment = d["moment"].cast<double>();
    t.max_count = d["max_count"].cast<long long>();
    t.total_sum = ptr_of<double>(d["total_sum"].cast<at::Tensor>());
    t.total_sum_err = ptr_of<double>(d["total_sum_err"].cast<at::Tensor>());
    t.total_sq = ptr_of<double>(d["total_sq"].cast<at::Tensor>());
    t.total_sq_err = ptr_of<double>(d["total_sq_err"].cast<at::Tensor>());
    t.total_count = ptr_of<double>(d["total_count"].cast<at::Tensor>());
    t.inc = ptr_of<double>(d["inc"].cast<at::Tensor>());
    t.mean = ptr_of<float>(d["mean"].cast<at::Tensor>());
    t.var = ptr_of<float>(d["var"].cast<at::Tensor>());
    batch = ptr_of<double>(d["batch"].cast<at::Tensor>());
    scratch = ptr_of<double>(d["scratch"].cast<at::Tensor>());
    s.world = d["world"].cast<int>();
    s.rank = d["rank"].cast<int>();
    if (s.world > 1) {
      auto inc = d["inc_ptrs"].cast<std::vector<int64_t>>();
      auto sig = d["sig_ptrs"].cast<std::vector<int64_t>>();
      TORCH_CHECK((int)inc.size() == s.world && (int)sig.size() == s.world, "peer tables");
      for (int p = 0; p < s.world; ++p) { s.inc[p] = ptr_of<const double>(inc[p]); s.sig[p] = ptr_of<unsigned long long>(sig[p]); }
      s.epoch = ptr_of<unsigned long long>(d["epoch"].cast<at::Tensor>());
      s.status = ptr_of<int>(d["status"].cast<at::Tensor>());
      s.wait_ns = d["wait_ns"].cast<uint64_t>();
      has_sync = true;
    }
  }
  // [h (bf16, first nh columns) | x (fp32)], or x alone
  tn::BnInput input(const c10::optional<at::Tensor>& h, int nh, const at::Tensor& x) const {
    tn::BnInput in{};
    TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2 && x.size(1) == t.C - nh && x.stride(1) == 1, "x must be fp32 [B, C]");
    in.x = ptr_of<float>(x);
    in.ldx = (int)x.stride(0);
    if (h.has_value()) {
      TORCH_CHECK(h->is_cuda() && h->scalar_type() == at::kBFloat16 && h->is_contiguous() && h->dim() == 2 && h->size(0) == x.size(0) && h->size(1) >= nh,
                  "h must be contiguous bf16 [B, >= nh]");
      in.h = h->data_ptr();
      in.ldh = (int)h->size(1);
      in.nh = nh;
    }
    return in;
  }
  // sums of one batch -> totals, increments (or none pending: `drop_inc`) and moments (two launches)
  void push(at::Tensor x, bool centered, bool drop_inc, c10::optional<at::Tensor> h, int nh) {
    const tn::BnInput in = input(h, h.has_value() ? nh : 0, x);
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_batch_stats(in, (int)x.size(0), t.C, centered ? t.mean : nullptr, batch, cur_stream());
    tn::launch_bn_table_append(t, batch, drop_inc, cur_stream());
  }
  void join_fwd(at::Tensor h, int nh, at::Tensor x, c10::optional<at::Tensor> gamma, c10::optional<at::Tensor> beta, double eps, at::Tensor z,
                at::Tensor moments) {
    const tn::BnInput in = input(h, nh, x);
    TORCH_CHECK(z.scalar_type() == at::kBFloat16 && z.is_contiguous() && z.size(1) % 2 == 0 && z.size(1) > t.C, "join: z");
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_join_fwd(in, (int)x.size(0), t.C, t.mean, t.var, gamma ? ptr_of<float>(*gamma) : nullptr, beta ? ptr_of<float>(*beta) : nullptr,
                           (float)eps, z.data_ptr(), (int)z.size(1), ptr_of<float>(moments), ptr_of<float>(moments) + t.C, cur_stream());
  }
  // push and join_fwd of one batch, in one launch where it fits
  void join_train(at::Tensor h, int nh, at::Tensor x, c10::optional<at::Tensor> gamma, c10::optional<at::Tensor> beta, double eps, bool drop_inc,
                  at::Tensor z, at::Tensor moments) {
    if (!tn::bn_join_train_fits((int)x.size(0), t.C, (int)z.size(1))) {
      push(x, false, drop_inc, h, nh);
      return join_fwd(h, nh, x, gamma, beta, eps, z, moments);
    }
    const tn::BnInput in = input(h, nh, x);
    TORCH_CHECK(z.scalar_type() == at::kBFloat16 && z.is_contiguous() && z.size(0) == x.size(0) && z.size(1) > t.C, "join: z");
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_join_train(t, in, (int)x.size(0), gamma ? ptr_of<float>(*gamma) : nullptr, beta ? ptr_of<float>(*beta) : nullptr, (float)eps,
                             drop_inc, z.data_ptr(), (int)z.size(1), ptr_of<float>(moments), ptr_of<float>(moments) + t.C, batch, cur_stream());
  }
  void join_bwd(at::Tensor dz, at::Tensor h, int nh, at::Tensor x, at::Tensor moments, c10::optional<at::Tensor> gamma, double eps, bool mask,
                c10::optional<at::Tensor> gh, c10::optional<at::Tensor> gx, c10::optional<at::Tensor> gg, c10::optional<at::Tensor> gb) {
    const tn::BnInput in = input(h, nh, x);
    TORCH_CHECK(dz.scalar_type() == at::kBFloat16 && dz.is_contiguous() && dz.size(1) >= t.C, "join: dz");
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_join_bwd(dz.data_ptr(), (int)dz.size(1), in, (int)x.size(0), t.C, ptr_of<float>(moments), ptr_of<float>(moments) + t.C,
                           gamma ? ptr_of<float>(*gamma) : nullptr, (float)eps, mask ? 1 : 0, gh ? gh->data_ptr() : nullptr,
                           gx ? ptr_of<float>(*gx) : nullptr, gx ? (int)gx->stride(0) : 0, gg ? ptr_of<float>(*gg) : nullptr,
                           gb ? ptr_of<float>(*gb) : nullptr, cur_stream());
  }
  // fold a record the host has staged in `batch`
  void append_staged() { tn::launch_bn_table_append(t, batch, false, cur_stream()); }
  void refresh() { tn::launch_bn_table_refresh(t, cur_stream()); }
  void sync() {
    if (has_sync) tn::launch_bn_table_sync(t, s, scratch, cur_stream());
  }
  void apply_fwd(at::Tensor x, at::Tensor mean, at::Tensor var, c10::optional<at::Tensor> gamma, c10::optional<at::Tensor> beta, double eps,
                 at::Tensor y) {
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_apply_fwd(ptr_of<float>(x), (int)x.stride(0), (int)x.size(0), t.C, ptr_of<float>(mean), ptr_of<float>(var), gamma ? ptr_of<float>(*gamma) : nullptr,
                            beta ? ptr_of<float>(*beta) : nullptr, (float)eps, ptr_of<float>(y), (int)y.stride(0), cur_stream());
  }
  void apply_bwd(at::Tensor dy, at::Tensor x, at::Tensor mean, at::Tensor var, c10::optional<at::Tensor> gamma, double eps,
                 c10::optional<at::Tensor> dx, c10::optional<at::Tensor> gg, c10::optional<at::Tensor> gb) {
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_bn_apply_bwd(ptr_of<float>(dy), (int)dy.stride(0), ptr_of<float>(x), (int)x.stride(0), (int)x.size(0), t.C,
                            ptr_of<float>(mean), ptr_of<float>(var),
                            gamma ? ptr_of<float>(*gamma) : nullptr, (float)eps, dx ? ptr_of<float>(*dx) : nullptr,
                            dx ? (int)dx->stride(0) : 0, gg ? ptr_of<float>(*gg) : nullptr, gb ? ptr_of<float>(*gb) : nullptr, cur_stream());
  }
};

// Device address of a host tensor that kernels may read in place (page-locked and mapped), else null.
const void* mapped_host_ptr(const at::Tensor& t) {
  if (t.is_cuda() || t.numel() == 0 || !t.is_contiguous()) return nullptr;
  const char* p = static_cast<const char*>(t.data_ptr());
  cudaPointerAttributes at;          // one question to the driver, whether it is page-locked and where a kernel finds it
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  const char* d = static_cast<const char*>(at.devicePointer);
  if (at.type != cudaMemoryTypeHost || d == nullptr) return nullptr;
  // Its last byte too, where that lies on another page: somebody may have registered no more than the pages that it begins in, and
  // a kernel would read on behind them.
  const char* last = p + t.nbytes() - 1;
  if (reinterpret_cast<uintptr_t>(p) >> 12 == reinterpret_cast<uintptr_t>(last) >> 12) return d;
  if (cudaPointerGetAttributes(&at, last) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  return at.type == cudaMemoryTypeHost && at.devicePointer == d + t.nbytes() - 1 ? d : nullptr;
}

// InferenceEngine's request path: lookup + pooling, the layers of the tower, head and sigmoid, launched from one call.
// Holds the dictionary's descriptor; weights come with every call (training may have re-pointed them).
struct ServeCtx {
  tn::TableView t{};
  py::dict keep;
  int S, combiner;
  std::vector<int> dims;           // tower widths, input first
  bool relu_last;
  ServeCtx(py::dict table, int S_, int combiner_, std::vector<int> dims_, bool relu_last_)
      : keep(table), S(S_), combiner(combiner_), dims(std::move(dims_)), relu_last(relu_last_) {
    t = table_from_dict(table);
    TORCH_CHECK(t.dim % 4 == 0 && t.stride % 4 == 0, "serving: dim must be a multiple of 4");
    TORCH_CHECK(dims.size() >= 2 && dims.size() <= (size_t)tn::kServeMaxLayers + 1 && dims[0] == S * t.dim, "serving: tower input width");
  }
  static int pad8(int n) { return (n + 7) / 8 * 8; }
  struct CopyLane { cudaStream_t stream = nullptr; cudaEvent_t begin = nullptr, end = nullptr, read = nullptr; };
  // one per thread and device: threads that serve side by side do not wait for one another's copies
  static CopyLane& copy_lane(int device) {
    static thread_local CopyLane lanes[64];
    CopyLane& c = lanes[device & 63];
    if (c.stream == nullptr) {
      check(cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking), "serving: stream");
      check(cudaEventCreateWithFlags(&c.begin, cudaEventDisableTiming), "serving: event");
      check(cudaEventCreateWithFlags(&c.end, cudaEventDisableTiming), "serving: event");
      check(cudaEventCreateWithFlags(&c.read, cudaEventDisableTiming), "serving: event");
    }
    return c;
  }

  // `weights`: fp32 [N, pad8(K + 1)] per layer; `shadows`: their bf16 copies when something keeps them current, else empty.
  // Nothing comes back for weights of another kind, or that do not start on 16 bytes, which the kernels' loads ask for.
  // `wait_read`: return only when page-locked ids and offsets have been read, so that the caller may fill them again.
  c10::optional<at::Tensor> forward(at::Tensor ids, c10::optional<at::Tensor> offsets, int B, const std::vector<at::Tensor>& weights,
                                    const std::vector<at::Tensor>& shadows, at::Tensor head_w, at::Tensor status, bool wait_read) {
    const int L = (int)dims.size() - 1;
    const bool cast_needed = shadows.empty();
    if (!head_w.is_cuda() || !head_w.is_contiguous() || head_w.scalar_type() != at::kFloat) return c10::nullopt;
    for (const at::Tensor& w : weights)
      if (!w.is_cuda() || !w.is_contiguous() || w.scalar_type() != at::kFloat) return c10::nullopt;
    TORCH_CHECK((int)weights.size() == L && (cast_needed || (int)shadows.size() == L) && head_w.numel() == dims[L] + 1, "serving: weights");
    TORCH_CHECK(ids.scalar_type() == at::kLong && ids.is_contiguous() && B >= 1, "serving: contiguous int64 ids");
    TORCH_CHECK(offsets.has_value() ? offsets->numel() == (int64_t)S * B + 1 && offsets->is_contiguous() && offsets->scalar_type() == at::kInt
                                    : ids.numel() == (int64_t)S * B, "serving: one bag per slot and example");
    for (const at::Tensor& w : cast_needed ? weights : shadows)
      if (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15) return c10::nullopt;
    c10::cuda::CUDAGuard guard(head_w.device());
    const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
    const auto dev = head_w.device();
    // Ids and offsets: small ones in place when the kernels can reach them (a copy costs its launch and a wait, 3 us);
    // beyond that the copy engine is the faster reader (44 against 22 GB/s at 819 KB).
    const bool on_host = !ids.is_cuda() && ids.numel() > 0;
    const size_t in_bytes = (size_t)ids.numel() * 8 + (offsets.has_value() ? (size_t)offsets->numel() * 4 : 0);
    at::Tensor hold_ids = ids, hold_off = offsets.has_value() ? *offsets : at::Tensor();
    const bool off_host = hold_off.defined() && !hold_off.is_cuda();
    const void *mid = nullptr, *moff = nullptr;
    if (in_bytes <= 128 * 1024) {
      if (on_host) mid = mapped_host_ptr(ids);
      if (off_host) moff = mapped_host_ptr(hold_off);
    }
    const bool copy_ids = on_host && !mid, copy_off = off_host && !moff;
    if (copy_ids) hold_ids = at::empty(ids.sizes(), ids.options().device(dev));
    if (copy_off) hold_off = at::empty(hold_off.sizes(), hold_off.options().device(dev));
    const long long* pid = static_cast<const long long*>(mid ? mid : hold_ids.data_ptr());
    const int* poff = hold_off.defined() ? static_cast<const int*>(moff ? moff : hold_off.data_ptr()) : nullptr;
    const bool skinny = B <= tn::kServeSkinnyRows;
    // one workspace: activations, row indices and offsets of a ragged request, bf16 weights
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    std::vector<size_t> at_act(L + 1), at_w(L);
    size_t bytes = 0;
    for (int l = 0; l <= L; ++l) { at_act[l] = bytes; bytes += up((size_t)B * pad8(dims[l] + 1) * 2); }
    size_t at_rows = 0, at_off = 0;
    if (poff) { at_rows = bytes; bytes += up((size_t)ids.numel() * 4); at_off = bytes; bytes += up(((size_t)S * B + 1) * 4); }
    const bool cast_now = cast_needed && !skinny;
    if (cast_now)
      for (int l = 0; l < L; ++l) { at_w[l] = bytes; bytes += up((size_t)weights[l].numel() * 2); }
    at::Tensor ws = at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(dev));
    at::Tensor prob = at::empty({B}, at::TensorOptions().dtype(at::kFloat).device(dev));
    uint8_t* w0 = static_cast<uint8_t*>(ws.data_ptr());
    for (int l = 0; l < L; ++l) {
      const at::Tensor& w = cast_needed ? weights[l] : shadows[l];
      TORCH_CHECK(w.is_cuda() && w.dim() == 2 && w.is_contiguous() && w.size(0) == dims[l + 1] && w.size(1) == pad8(dims[l] + 1) &&
                      w.scalar_type() == (cast_needed ? at::kFloat : at::kBFloat16),
                  "serving: layer ", l, " weights");
    }
    cudaEvent_t read = nullptr;                // behind the last reader of page-locked memory
    bool pinned = mid != nullptr || moff != nullptr;
    if (copy_ids || copy_off) {
      // on a stream of its own: the weights are converted meanwhile
      CopyLane& cl = copy_lane(dev.index());
      const bool side = cast_now;
      const cudaStream_t cs = side ? cl.stream : st;
      if (side) {
        check(cudaEventRecord(cl.begin, st), "serving: event");        // the buffers' former users are done
        check(cudaStreamWaitEvent(cs, cl.begin, 0), "serving: wait");
      }
      auto put = [&](const at::Tensor& d, const at::Tensor& h) {
        check(cudaMemcpyAsync(d.data_ptr(), h.data_ptr(), h.nbytes(), cudaMemcpyHostToDevice, cs), "serving: copy");
        if (h.is_pinned()) {
          pinned = true;
          at::getHostAllocator(at::kCUDA)->record_event(const_cast<void*>(h.storage().data()), h.storage().data_ptr().get_context(),
                                                        c10::cuda::getStreamFromExternal(cs, dev.index()).unwrap());
        }
      };
      if (copy_ids) put(hold_ids, ids);
      if (copy_off) put(hold_off, *offsets);
      if (side) check(cudaEventRecord(cl.end, cs), "serving: event");
      if (wait_read && pinned) {
        read = side ? cl.end : cl.read;
        if (!side) check(cudaEventRecord(cl.read, st), "serving: event");
      }
    }
    if (cast_now) {
      tn::ServeCast c{};
      c.n = L;
      for (int l = 0; l < L; ++l) { c.src[l] = ptr_of<const float>(weights[l]); c.dst[l] = w0 + at_w[l]; c.n8[l] = weights[l].numel() / 8; }
      tn::launch_serve_cast(c, st);
      if (copy_ids || copy_off) check(cudaStreamWaitEvent(st, copy_lane(dev.index()).end, 0), "serving: wait");
    }
    // behind a copy the lookup is launched the ordinary way; the conversion is then complete anyway
    const bool behind_cast = cast_now && !copy_ids && !copy_off;
    const int ld0 = pad8(dims[0] + 1);
    const bool in_place = mid != nullptr || moff != nullptr;
    if (wait_read && in_place) read = copy_lane(dev.index()).read;
    if (poff)
      tn::launch_serve_lookup_ragged(t, pid, (int)ids.numel(), poff, B, S, combiner, reinterpret_cast<int*>(w0 + at_rows),
                                     moff ? reinterpret_cast<int*>(w0 + at_off) : nullptr, w0 + at_act[0], ld0, dims[0], behind_cast,
                                     wait_read && in_place ? read : nullptr, st);
    else
      tn::launch_serve_lookup_single(t, pid, B, S, w0 + at_act[0], ld0, dims[0], behind_cast, wait_read && in_place ? read : nullptr, st);
    // host memory read in place must not be handed out again before the kernels are done with it
    for (const at::Tensor* h : {mid ? &hold_ids : nullptr, moff ? &hold_off : nullptr})
      if (h != nullptr)
        at::getHostAllocator(at::kCUDA)->record_event(const_cast<void*>(h->storage().data()), h->storage().data_ptr().get_context(),
                                                      at::cuda::getCurrentCUDAStream().unwrap());
    for (int l = 0; l < L; ++l) {
      const int N = dims[l + 1], K = dims[l] + 1, ldx = pad8(K), ldy = pad8(N + 1), relu = relu_last || l < L - 1;
      void *x = w0 + at_act[l], *y = w0 + at_act[l + 1];
      const void* w = cast_now ? (const void*)(w0 + at_w[l]) : (cast_needed ? weights[l].data_ptr() : shadows[l].data_ptr());
      if (skinny) {
        tn::launch_serve_skinny(x, ldx, w, cast_needed ? 1 : 0, ldx, B, N, K, relu, y, ldy, ldy, st);
      } else {
        tn::GemmDesc d;
        d.M = B; d.N = N; d.K = K; d.A = x; d.B = w; d.lda = ldx; d.ldb = ldx; d.C = y; d.ldc = ldy; d.relu = relu;
        d.ones_col = N; d.n_store = ldy; d.split_k = 1; d.status = ptr_of<int>(status);
        const char* err = tn::gemm_bf16(d, st);
        if (err) throw std::runtime_error(err);
      }
    }
    tn::launch_serve_head(w0 + at_act[L], pad8(dims[L] + 1), B, dims[L] + 1, ptr_of<const float>(head_w), ptr_of<float>(prob), st);
    check(cudaGetLastError(), "serving launch");
    g_launches.fetch_add(L + 2 + (cast_now ? 1 : 0) + (poff ? 1 : 0), std::memory_order_relaxed);
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (read != nullptr) check(cudaStreamIsCapturing(st, &capturing), "serving: stream");
    if (read != nullptr && capturing == cudaStreamCaptureStatusNone) {
      py::gil_scoped_release others_may_run;
      check(cudaEventSynchronize(read), "serving: inputs");
    }
    return prob;
  }
};

// A metric-sum buffer is fp32[4] or fp32[4 + 2 * nbins]: the tail holds the two u32 prediction histograms of the AUC.
static int hist_bins(const at::Tensor& sums) {
  TORCH_CHECK(sums.scalar_type() == at::kFloat && sums.is_contiguous() && sums.numel() >= 4 && (sums.numel() - 4) % 2 == 0,
              "metric sums must be fp32[4] or fp32[4 + 2 * nbins]");
  return (int)((sums.numel() - 4) / 2);
}

void gemm(at::Tensor A, at::Tensor B, at::Tensor C, int M, int N, int K, int lda, int ldb, int ldc, bool a_mn, bool b_mn,
          bool accumulate, bool relu, c10::optional<at::Tensor> bias, c10::optional<at::Tensor> mask_aux,
          c10::optional<at::Tensor> had_x0, c10::optional<at::Tensor> had_xl, int ld_aux, int ones_col, int n_store,
          int split_k, int BN, at::Tensor status, c10::optional<at::Tensor> prof, c10::optional<at::Tensor> gate_flags,
          c10::optional<at::Tensor> gate_epoch, int gate_world, uint64_t gate_wait_ns, int m_halves, c10::optional<at::Tensor> aux_out, int cluster_k) {
  TORCH_CHECK(A.is_cuda() && B.is_cuda() && C.is_cuda(), "gemm: CUDA tensors");
  TORCH_CHECK(A.scalar_type() == at::kBFloat16 && B.scalar_type() == at::kBFloat16, "gemm: bf16 operands");
  c10::cuda::CUDAGuard guard(A.device());
  tn::GemmDesc d;
  d.M = M; d.N = N; d.K = K; d.A = A.data_ptr(); d.B = B.data_ptr(); d.lda = lda; d.ldb = ldb;
  d.a_mn = a_mn; d.b_mn = b_mn; d.C = C.data_ptr(); d.ldc = ldc;
  d.out_f32 = C.scalar_type() == at::kFloat;
  TORCH_CHECK(d.out_f32 || C.scalar_type() == at::kBFloat16, "gemm: C must be fp32 or bf16");
  d.accumulate = accumulate; d.relu = relu;
  d.bias = bias.has_value() ? ptr_of<const float>(*bias) : nullptr;
  d.mask_aux = mask_aux.has_value() ? mask_aux->data_ptr() : nullptr;
  d.had_x0 = had_x0.has_value() ? had_x0->data_ptr() : nullptr;
  d.had_xl = had_xl.has_value() ? had_xl->data_ptr() : nullptr;
  d.ld_aux = ld_aux; d.ones_col = ones_col; d.n_store = n_store; d.split_k = split_k; d.BN = BN;
  d.status = ptr_of<int>(status);
  d.prof = prof.has_value() ? ptr_of<unsigned long long>(*prof) : nullptr;
  d.m_halves = m_halves;
  d.cluster_k = cluster_k;
  if (aux_out.has_value()) {
    TORCH_CHECK(aux_out->scalar_type() == at::kBFloat16 && aux_out->stride(0) == ld_aux, "gemm: aux_out must be bf16 with row stride ld_aux");
    d.aux_out = aux_out->data_ptr();
  }
  if (gate_flags.has_value()) {
    TORCH_CHECK(gate_epoch.has_value() && gate_world >= 1 && gate_world <= tn::kMaxWorld, "gemm: gate wants flags, epoch and a world size");
    d.gate_flags = ptr_of<const unsigned long long>(*gate_flags);
    d.gate_epoch = ptr_of<const unsigned long long>(*gate_epoch);
    d.gate_world = gate_world;
    d.gate_wait_ns = gate_wait_ns;
  }
  const char* err = tn::gemm_bf16(d, cur_stream());
  if (err) throw std::runtime_error(err);
}

// One-kernel MLP chain.  weights[i]: bf16 [N_i, ld]; outs[i]: bf16 [M, ld_out_i] (forward: activations; backward: input
// gradients); masks[i] (backward): the activation whose ReLU the gradient passes through, or None.
tn::MlpChainDesc chain_desc(bool backward, const at::Tensor& x, int in_cols, const std::vector<at::Tensor>& weights,
                            const std::vector<int>& n_rows, const std::vector<int>& k_cols, const std::vector<at::Tensor>& outs,
                            const std::vector<int>& relu, const std::vector<int>& n_valid,
                            const std::vector<c10::optional<at::Tensor>>& masks, const at::Tensor& status) {
  const int L = (int)weights.size();
  TORCH_CHECK(L >= 1 && L <= tn::kMlpMaxLayers && (int)outs.size() == L && (int)n_rows.size() == L && (int)k_cols.size() == L,
              "mlp_chain: 1..4 layers with one output each");
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1, "mlp_chain: input must be a bf16 matrix");
  tn::MlpChainDesc d;
  d.L = L; d.M = (int)x.size(0); d.backward = backward ? 1 : 0;
  d.in = x.data_ptr(); d.in_cols = in_cols; d.ld_in = (int)x.stride(0);
  d.status = ptr_of<int>(status);
  for (int i = 0; i < L; ++i) {
    const at::Tensor& w = weights[i];
    const at::Tensor& o = outs[i];
    TORCH_CHECK(w.scalar_type() == at::kBFloat16 && w.dim() == 2 && w.stride(1) == 1, "mlp_chain: weights must be bf16 matrices");
    TORCH_CHECK(o.scalar_type() == at::kBFloat16 && o.dim() == 2 && o.stride(1) == 1 && o.size(0) == x.size(0), "mlp_chain: bad output");
    TORCH_CHECK(n_rows[i] <= w.size(0) && k_cols[i] <= w.stride(0), "mlp_chain: layer shape exceeds the weight matrix");
    tn::MlpChainLayer& l = d.layer[i];
    l.w = w.data_ptr(); l.n_rows = n_rows[i]; l.k_cols = k_cols[i]; l.ldw = (int)w.stride(0);
    l.out = o.data_ptr(); l.ld_out = (int)o.stride(0);
    l.relu = i < (int)relu.size() ? relu[i] : 0;
    l.n_valid = i < (int)n_valid.size() ? n_valid[i] : 0;
    if (i < (int)masks.size() && masks[i].has_value()) {
      const at::Tensor& mk = *masks[i];
      TORCH_CHECK(mk.scalar_type() == at::kBFloat16 && mk.dim() == 2 && mk.size(0) == x.size(0), "mlp_chain: bad mask");
      l.mask = mk.data_ptr(); l.ld_mask = (int)mk.stride(0);
    }
  }
  return d;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<SparseCtx>(m, "SparseCtx")
      .def(py::init<py::dict, py::dict, py::dict>())
      .def("set_opt", &SparseCtx::set_opt)
      .def("set_table", &SparseCtx::set_table)
      .def("pull", &SparseCtx::pull, py::arg("ids"), py::arg("inverse"), py::arg("labels"), py::arg("label_mod"), py::arg("training"),
           py::arg("lookup_only") = false, py::arg("front_done") = false, py::arg("n_dev") = py::none(), py::arg("rows") = true,
           py::arg("req") = py::none())
      .def("push", [](SparseCtx& self, int64_t work_hint, int max_ctas, py::object dense, c10::optional<at::Tensor> req) {
        if (dense.is_none()) { self.push(work_hint, max_ctas, nullptr, req); return; }
        const tn::DenseStepArgs d = dense.cast<DenseCtx&>().rider_args();
        self.push(work_hint, max_ctas, &d, req);
      }, py::arg("work_hint"), py::arg("max_ctas") = 0, py::arg("dense") = py::none(), py::arg("req") = py::none())
      .def("front", &SparseCtx::front, py::arg("ids"), py::arg("inverse"), py::arg("req") = py::none())
      .def("in_place", &SparseCtx::in_place)
      // in-place pulls of different tables side by side: all of them behind a front (`front_done`) or none
      .def_static("pull_many", [](std::vector<SparseCtx*> ctx, std::vector<at::Tensor> ids, std::vector<at::Tensor> inverse,
                                  std::vector<c10::optional<at::Tensor>> labels, std::vector<int> label_mod, std::vector<bool> training,
                                  bool front_done, std::vector<c10::optional<at::Tensor>> n_dev, std::vector<c10::optional<at::Tensor>> req) {
        const size_t n = ctx.size();
        TORCH_CHECK(n >= 1 && n <= (size_t)tn::kMaxPullBatch && ids.size() == n && inverse.size() == n && labels.size() == n &&
                        label_mod.size() == n && training.size() == n && n_dev.size() == n && req.size() == n, "pull_many: one entry per pull");
        c10::cuda::CUDAGuard guard(ids[0].device());
        tn::PullArgs batch[tn::kMaxPullBatch];
        for (size_t k = 0; k < n; ++k) {
          TORCH_CHECK(ctx[k]->in_place(), "pull_many: in-place pulls only");
          for (size_t j = 0; j < k; ++j) TORCH_CHECK(ctx[j]->t.keys != ctx[k]->t.keys, "pull_many: different tables");
          batch[k] = ctx[k]->batch_args(ids[k], inverse[k], labels[k], label_mod[k], training[k], false, front_done, n_dev[k], req[k]);
        }
        check(tn::launch_sparse_pull_local(batch, (int)n, cur_stream()), "sparse_pull_local launch");
        if (!front_done) g_launches.fetch_add(1, std::memory_order_relaxed);
      })
      // the rows of the ids of up to two tables (one GPU); nothing is counted
      .def_static("lookup_many", [](std::vector<SparseCtx*> ctx, std::vector<at::Tensor> ids, std::vector<at::Tensor> rows,
                                    std::vector<c10::optional<at::Tensor>> n_dev, bool lookup_only) {
        const size_t n = ctx.size();
        TORCH_CHECK(n >= 1 && n <= (size_t)tn::kMaxPullBatch && ids.size() == n && rows.size() == n && n_dev.size() == n, "lookup_many: one entry per lookup");
        c10::cuda::CUDAGuard guard(ids[0].device());
        tn::PullArgs batch[tn::kMaxPullBatch];
        for (size_t k = 0; k < n; ++k) {
          TORCH_CHECK(ctx[k]->in_place(), "lookup_many: one GPU only");
          for (size_t j = 0; j < k; ++j) TORCH_CHECK(ctx[j]->t.keys != ctx[k]->t.keys, "lookup_many: different tables");
          batch[k] = ctx[k]->batch_args(ids[k], rows[k], c10::nullopt, 0, false, lookup_only, false, n_dev[k], c10::nullopt);
        }
        check(tn::launch_sparse_lookup(batch, (int)n, cur_stream()), "sparse_lookup launch");
        if (!lookup_only) g_launches.fetch_add(2, std::memory_order_relaxed);
      })
      .def("pool_fwd", [](SparseCtx& self, at::Tensor inverse, c10::optional<at::Tensor> offsets, int B, int S, int combiner, at::Tensor out,
                          c10::optional<at::Tensor> req, bool direct) {
        c10::cuda::CUDAGuard guard(out.device());
        const int pd = self.t.dim + 2 * self.t.use_cvm;
        TORCH_CHECK(out.scalar_type() == at::kFloat && out.is_contiguous() && out.numel() == (int64_t)B * S * pd, "pool_fwd: out must be fp32 [B, S * width]");
        tn::launch_pool_fwd(self.source(req, direct), ptr_of<int>(inverse), offsets ? ptr_of<int>(*offsets) : nullptr, B, S, pd, combiner,
                            ptr_of<float>(out), S * pd, cur_stream());
      }, py::arg("inverse"), py::arg("offsets"), py::arg("B"), py::arg("S"), py::arg("combiner"), py::arg("out"), py::arg("req"),
         py::arg("direct") = false)
      .def("seq_fwd", [](SparseCtx& self, at::Tensor inverse, at::Tensor offsets, int B, int T, at::Tensor out, at::Tensor lengths,
                         c10::optional<at::Tensor> req) {
        c10::cuda::CUDAGuard guard(out.device());
        tn::launch_seq_fwd(self.source(req, false), ptr_of<int>(inverse), ptr_of<int>(offsets), B, T, self.t.dim + 2 * self.t.use_cvm,
                           ptr_of<float>(out), ptr_of<int>(lengths), cur_stream());
      })
      .def("embed_input_fwd", [](SparseCtx& self, at::Tensor inverse, c10::optional<at::Tensor> offsets, int B, int S, int D, int combiner,
                                 c10::optional<at::Tensor> dense, at::Tensor X0, c10::optional<at::Tensor> E, c10::optional<at::Tensor> fm,
                                 c10::optional<at::Tensor> fsum, int lin_col, c10::optional<at::Tensor> Lout, c10::optional<at::Tensor> req, bool direct) {
        c10::cuda::CUDAGuard guard(X0.device());
        auto f32 = [](const c10::optional<at::Tensor>& t, int64_t n) { return !t || (t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() >= n); };
        const int pd = self.t.dim + 2 * self.t.use_cvm;
        TORCH_CHECK(D >= 1 && D <= pd && lin_col < self.t.dim && (!offsets || offsets->numel() >= (int64_t)B * S + 1) &&
                        (offsets || inverse.numel() >= (int64_t)B * S), "embed_input: slots");
        TORCH_CHECK(X0.scalar_type() == at::kBFloat16 && X0.dim() == 2 && X0.stride(1) == 1 && X0.size(0) == B && (!E || (f32(E, 0) && E->dim() == 2 && E->size(0) == B)) &&
                        f32(fm, B) && f32(fsum, (int64_t)B * ((D + 3) / 4 * 4)) && f32(Lout, (int64_t)B * S) &&
                        (!dense || (dense->scalar_type() == at::kFloat && dense->dim() == 2 && dense->stride(1) == 1 && dense->size(0) == B)),
                    "embed_input: outputs or dense features");
        tn::EmbedInput a = {};
        a.inverse = ptr_of<int>(inverse); a.offsets = offsets ? ptr_of<int>(*offsets) : nullptr;
        a.B = B; a.S = S; a.D = D; a.combiner = combiner;
        a.dense = dense ? ptr_of<float>(*dense) : nullptr;
        a.Dd = dense ? (int)dense->size(1) : 0; a.ld_dense = dense ? (int)dense->stride(0) : 0;
        a.X0 = X0.data_ptr(); a.ld = (int)X0.stride(0);
        a.E = E ? ptr_of<float>(*E) : nullptr; a.ldE = E ? (int)E->size(1) : 0; a.fm = fm ? ptr_of<float>(*fm) : nullptr; a.fsum = fsum ? ptr_of<float>(*fsum) : nullptr;
        a.Lout = Lout ? ptr_of<float>(*Lout) : nullptr; a.lin_col = Lout ? lin_col : -1;
        if (const char* err = tn::launch_embed_input_fwd(self.source(req, direct), a, cur_stream())) throw std::runtime_error(err);
      });
  py::class_<ServeCtx>(m, "ServeCtx")
      .def(py::init<py::dict, int, int, std::vector<int>, bool>())
      .def("forward", &ServeCtx::forward);
  py::class_<BnCtx>(m, "BnCtx")
      .def(py::init<py::dict>())
      .def("push", &BnCtx::push, py::arg("x"), py::arg("centered"), py::arg("drop_inc") = false, py::arg("h") = py::none(), py::arg("nh") = 0)
      .def("append_staged", &BnCtx::append_staged)
      .def("refresh", &BnCtx::refresh)
      .def("sync", &BnCtx::sync)
      .def("apply_fwd", &BnCtx::apply_fwd)
      .def("join_train", &BnCtx::join_train)
      .def("join_fwd", &BnCtx::join_fwd)
      .def("join_bwd", &BnCtx::join_bwd)
      .def("apply_bwd", &BnCtx::apply_bwd);
  py::class_<DenseCtx>(m, "DenseCtx").def(py::init<py::dict>()).def("step", &DenseCtx::step, py::arg("skip_open") = false).def("set_gated", &DenseCtx::set_gated).def("set_max_ctas", &DenseCtx::set_max_ctas);
  m.def("dense_ctas_per_sm", [] { return tn::dense_step_ctas_per_sm(); });
  m.def("mlp_chain", [](bool backward, at::Tensor x, int in_cols, std::vector<at::Tensor> weights, std::vector<int> n_rows,
                        std::vector<int> k_cols, std::vector<at::Tensor> outs, std::vector<int> relu, std::vector<int> n_valid,
                        std::vector<c10::optional<at::Tensor>> masks, at::Tensor status, c10::optional<at::Tensor> gate_flags,
                        c10::optional<at::Tensor> gate_epoch, int gate_world, uint64_t gate_wait_ns, bool probe_only,
                        c10::optional<at::Tensor> prof, int split) {
    c10::cuda::CUDAGuard guard(x.device());
    tn::MlpChainDesc d = chain_desc(backward, x, in_cols, weights, n_rows, k_cols, outs, relu, n_valid, masks, status);
    d.split = split;
    if (prof.has_value()) {
      TORCH_CHECK(prof->scalar_type() == at::kLong && prof->numel() >= 16, "mlp_chain: prof must be int64[16]");
      d.prof = ptr_of<unsigned long long>(*prof);
    }
    if (gate_flags.has_value()) {
      d.gate_flags = ptr_of<const unsigned long long>(*gate_flags);
      d.gate_epoch = ptr_of<const unsigned long long>(*gate_epoch);
      d.gate_world = gate_world;
      d.gate_wait_ns = gate_wait_ns;
    }
    if (probe_only) {
      const char* why = tn::mlp_chain_supported(d);
      return std::string(why ? why : "");
    }
    const char* err = tn::mlp_chain(d, cur_stream());
    if (err) throw std::runtime_error(err);
    return std::string();
  }, py::arg("backward"), py::arg("x"), py::arg("in_cols"), py::arg("weights"), py::arg("n_rows"), py::arg("k_cols"), py::arg("outs"),
     py::arg("relu"), py::arg("n_valid"), py::arg("masks"), py::arg("status"), py::arg("gate_flags") = py::none(),
     py::arg("gate_epoch") = py::none(), py::arg("gate_world") = 0, py::arg("gate_wait_ns") = 0, py::arg("probe_only") = false, py::arg("prof") = py::none(), py::arg("split") = 0,
     "a whole MLP tower (forward, or the input-gradient chain of the backward pass) in one kernel");
  m.def("gemm", &gemm, py::arg("A"), py::arg("B"), py::arg("C"), py::arg("M"), py::arg("N"), py::arg("K"), py::arg("lda"),
        py::arg("ldb"), py::arg("ldc"), py::arg("a_mn"), py::arg("b_mn"), py::arg("accumulate"), py::arg("relu"), py::arg("bias"),
        py::arg("mask_aux"), py::arg("had_x0"), py::arg("had_xl"), py::arg("ld_aux"), py::arg("ones_col"), py::arg("n_store"),
        py::arg("split_k"), py::arg("BN"), py::arg("status"), py::arg("prof") = py::none(),
        py::arg("gate_flags") = py::none(), py::arg("gate_epoch") = py::none(), py::arg("gate_world") = 0, py::arg("gate_wait_ns") = 0,
        py::arg("m_halves") = 0, py::arg("aux_out") = py::none(), py::arg("cluster_k") = 0);
  m.def("launch_count", []() { return g_launches.load(); });

  // ---- per-step host path of a replayed training step --------------------------------------------
  // One call instead of a dozen Python-level stream / event / copy calls: wait (on the copy stream) until the replay
  // that last read these input buffers is over, copy the step's inputs host -> device, record their arrival and make
  // the compute stream wait for it.  Streams and events come as the handles torch exposes (cuda_stream, cuda_event).
  m.def("stage_inputs", [](std::vector<at::Tensor> dsts, std::vector<at::Tensor> srcs, int64_t copy_stream, int64_t main_stream,
                           int64_t done_event, int64_t copied_event, int64_t read_event) {
    TORCH_CHECK(dsts.size() == srcs.size(), "stage_inputs: one source per destination");
    if (dsts.empty()) return;
    c10::cuda::CUDAGuard guard(dsts[0].device());
    cudaStream_t cs = reinterpret_cast<cudaStream_t>(copy_stream), ms = reinterpret_cast<cudaStream_t>(main_stream);
    if (done_event) check(cudaStreamWaitEvent(cs, reinterpret_cast<cudaEvent_t>(done_event), 0), "cudaStreamWaitEvent");
    // the loss of the step that last used this buffer set has been read back (it lives in the same captured memory)
    if (read_event) check(cudaStreamWaitEvent(cs, reinterpret_cast<cudaEvent_t>(read_event), 0), "cudaStreamWaitEvent");
    // Small leaves in page-locked memory go together, read by a kernel; larger ones, for which the copy engine is the faster reader,
    // one copy each.  (Up to 256 KB a kernel's 22 to 30 GB/s are no slower than a copy's rate with its 2 us to the next one.  One or
    // two leaves stay copies: a kernel then saves at most one of them, and it takes turns with those of the step: with two leaves
    // of 16 KB beside 2 MB of ids a Deep&Cross step took 252 us in place of 246.)
    constexpr int64_t kSmall = 256 * 1024;
    tn::StagePieces pieces;
    std::vector<size_t> small;
    std::vector<const void*> seen;
    for (size_t i = 0; i < dsts.size(); ++i) {
      const at::Tensor& d = dsts[i];
      const at::Tensor& h = srcs[i];
      // a vector may be shorter than its static buffer (ids of a batch with ragged slots)
      TORCH_CHECK(d.is_cuda() && !h.is_cuda() && d.is_contiguous() && h.is_contiguous() && d.scalar_type() == h.scalar_type() &&
                      (d.nbytes() == h.nbytes() || (d.dim() == 1 && h.dim() == 1 && h.nbytes() <= d.nbytes())),
                  "stage_inputs: leaf ", i, " must be a contiguous host tensor of the static buffer's type and size");
      const void* p = (int64_t)h.nbytes() <= kSmall ? mapped_host_ptr(h) : nullptr;
      if (p == nullptr) continue;
      small.push_back(i);
      seen.push_back(p);
    }
    if (small.size() < 3) { small.clear(); seen.clear(); }
    size_t next = 0;
    for (size_t i = 0; i < dsts.size(); ++i) {
      const at::Tensor& d = dsts[i];
      const at::Tensor& h = srcs[i];
      if (h.nbytes() == 0) continue;
      if (next < small.size() && small[next] == i) { ++next; continue; }
      check(cudaMemcpyAsync(d.data_ptr(), h.data_ptr(), h.nbytes(), cudaMemcpyHostToDevice, cs), "cudaMemcpyAsync");
    }
    for (size_t at = 0; at < small.size(); at += tn::kStagePieces) {
      pieces.n = 0;
      for (size_t k = at; k < small.size() && k < at + tn::kStagePieces; ++k) {
        pieces.src[pieces.n] = seen[k];
        pieces.dst[pieces.n] = dsts[small[k]].data_ptr();
        pieces.bytes[pieces.n++] = (int)srcs[small[k]].nbytes();
      }
      check(tn::launch_stage_inputs(pieces, cs), "stage_inputs launch");
      g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    // a page-locked source from torch's host allocator must not be handed out again before it has been read
    // (what Tensor.copy_(non_blocking=True) does behind the scenes); a no-op for other host memory
    next = 0;
    auto* hosts = at::getHostAllocator(at::kCUDA);
    const c10::Stream on = c10::cuda::getStreamFromExternal(cs, dsts[0].device().index()).unwrap();
    for (size_t i = 0; i < dsts.size(); ++i) {
      const bool in_kernel = next < small.size() && small[next] == i;
      if (in_kernel) ++next;
      const at::Tensor& h = srcs[i];
      if (h.nbytes() == 0 || !(in_kernel || h.is_pinned())) continue;
      const at::DataPtr& mem = h.storage().data_ptr();
      hosts->record_event(const_cast<void*>(mem.get()), mem.get_context(), on);
    }
    check(cudaEventRecord(reinterpret_cast<cudaEvent_t>(copied_event), cs), "cudaEventRecord");
    check(cudaStreamWaitEvent(ms, reinterpret_cast<cudaEvent_t>(copied_event), 0), "cudaStreamWaitEvent");
  });
  // Numbers of ids of the ragged columns of a batch in host memory (values, offsets in turn), or an empty list when a
  // column's last offset is not the length of its values: a Python-level read of every last offset costs more than the
  // staging itself for batches of dozens of columns.
  m.def("ragged_lengths", [](std::vector<at::Tensor> cols) {
    std::vector<int64_t> n;
    for (size_t i = 0; i + 1 < cols.size(); i += 2) {
      const at::Tensor &v = cols[i], &o = cols[i + 1];
      int64_t last = -1;
      if (v.dim() == 1 && o.dim() == 1 && !o.is_cuda() && o.numel() >= 1) {
        const char* p = static_cast<const char*>(o.data_ptr()) + (o.numel() - 1) * o.stride(0) * o.element_size();
        if (o.scalar_type() == at::kInt) last = *reinterpret_cast<const int*>(p);
        else if (o.scalar_type() == at::kLong) last = *reinterpret_cast<const int64_t*>(p);
      }
      if (last != v.numel()) return std::vector<int64_t>();
      n.push_back(last);
    }
    return n;
  });
  // 4-byte device scalar -> slot of a pinned ring, then an event behind it (the loss of a step on its way to the host)
  // `wait_event` != 0: the copy runs on a stream of its own behind that event (the end of the step), so the compute
  // stream carries nothing between two replayed steps.
  m.def("read_scalar_async", [](at::Tensor pinned, int64_t slot, at::Tensor src, int64_t stream, int64_t event, int64_t wait_event) {
    TORCH_CHECK(!pinned.is_cuda() && pinned.scalar_type() == at::kFloat && slot >= 0 && slot < pinned.numel(), "bad ring slot");
    TORCH_CHECK(src.is_cuda() && src.scalar_type() == at::kFloat && src.numel() == 1, "source: one float on the device");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (wait_event) check(cudaStreamWaitEvent(st, reinterpret_cast<cudaEvent_t>(wait_event), 0), "cudaStreamWaitEvent");
    check(cudaMemcpyAsync(pinned.data_ptr<float>() + slot, src.data_ptr(), sizeof(float), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
    check(cudaEventRecord(reinterpret_cast<cudaEvent_t>(event), st), "cudaEventRecord");
  });

  // ---- CUDA IPC peer memory (fallback transport for the symmetric heap) --------------------------
  m.def("ipc_alloc", [](int64_t nbytes) {
    void* p = nullptr;
    check(cudaMalloc(&p, (size_t)nbytes), "cudaMalloc");
    check(cudaMemset(p, 0, (size_t)nbytes), "cudaMemset");
    cudaIpcMemHandle_t h;
    check(cudaIpcGetMemHandle(&h, p), "cudaIpcGetMemHandle");
    return py::make_tuple((int64_t)reinterpret_cast<uintptr_t>(p), py::bytes(reinterpret_cast<const char*>(&h), sizeof(h)));
  });
  m.def("ipc_open", [](py::bytes handle) {
    std::string hs = handle;
    TORCH_CHECK(hs.size() == sizeof(cudaIpcMemHandle_t), "bad IPC handle size");
    cudaIpcMemHandle_t h;
    std::memcpy(&h, hs.data(), sizeof(h));
    void* p = nullptr;
    check(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess), "cudaIpcOpenMemHandle");
    return (int64_t)reinterpret_cast<uintptr_t>(p);
  });
  m.def("ipc_close", [](int64_t p) { cudaIpcCloseMemHandle(ptr_of<void>(p)); });
  m.def("ipc_free", [](int64_t p) { cudaFree(ptr_of<void>(p)); });
  m.def("tensor_from_ptr", [](int64_t p, int64_t nbytes, int device) {
    auto opts = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device);
    return at::from_blob(ptr_of<void>(p), {nbytes}, opts);
  });

  m.def("expand_bag_labels", [](at::Tensor y, at::Tensor offsets, int S, at::Tensor out) {
    TORCH_CHECK(y.scalar_type() == at::kFloat && y.is_contiguous() && offsets.scalar_type() == at::kInt && offsets.is_contiguous() &&
                    offsets.numel() == y.numel() * S + 1 && out.scalar_type() == at::kFloat && out.is_contiguous(), "expand_bag_labels");
    c10::cuda::CUDAGuard guard(y.device());
    tn::launch_expand_bag_labels(ptr_of<float>(y), ptr_of<int>(offsets), (int)y.numel(), (int)y.numel() * S, ptr_of<float>(out),
                                 (int)out.numel(), cur_stream());
  });
  m.def("pack_columns", [](std::vector<at::Tensor> values, std::vector<c10::optional<at::Tensor>> offsets, std::vector<int> lens, int B,
                           at::Tensor out_values, at::Tensor out_offsets) {
    const int S = (int)values.size();
    TORCH_CHECK(S >= 1 && (int)offsets.size() == S && (int)lens.size() == S && B >= 1 && out_values.scalar_type() == at::kLong &&
                    out_values.is_contiguous() && out_offsets.scalar_type() == at::kInt && out_offsets.is_contiguous() &&
                    out_offsets.numel() == (int64_t)S * B + 1, "pack_columns");
    c10::cuda::CUDAGuard guard(out_values.device());
    for (int s0 = 0; s0 < S; s0 += tn::kPackColumns) {
      tn::PackColumns a{};
      a.n = std::min(tn::kPackColumns, S - s0); a.B = B; a.first = s0;
      a.out_values = ptr_of<long long>(out_values); a.out_offsets = ptr_of<int>(out_offsets); a.total_room = out_values.numel();
      for (int c = 0; c < a.n; ++c) {
        const at::Tensor& v = values[s0 + c];
        TORCH_CHECK(v.is_cuda() && v.is_contiguous() && (v.scalar_type() == at::kLong || v.scalar_type() == at::kInt), "pack_columns: ids");
        a.values[c] = v.data_ptr(); a.val64[c] = v.scalar_type() == at::kLong; a.room[c] = (int)v.numel(); a.len[c] = lens[s0 + c];
        if (offsets[s0 + c].has_value()) {
          const at::Tensor& o = *offsets[s0 + c];
          TORCH_CHECK(o.is_cuda() && o.is_contiguous() && o.numel() == B + 1 && (o.scalar_type() == at::kLong || o.scalar_type() == at::kInt),
                      "pack_columns: offsets");
          a.offsets[c] = o.data_ptr(); a.off64[c] = o.scalar_type() == at::kLong;
        }
      }
      tn::launch_pack_columns(a, cur_stream());
    }
  });
  m.def("pool_fwd", [](at::Tensor U, int ustride, at::Tensor inverse, c10::optional<at::Tensor> offsets, int B, int S, int pd,
                       int combiner, at::Tensor out, int out_ld) {
    c10::cuda::CUDAGuard guard(U.device());
    TORCH_CHECK(ustride % 4 == 0 && reinterpret_cast<uintptr_t>(U.data_ptr()) % 16 == 0, "pool_fwd: rows of U must be whole 16-byte pieces");
    tn::RowSource src{};
    src.U = ptr_of<float>(U);
    src.ustride = ustride;
    tn::launch_pool_fwd(src, ptr_of<int>(inverse), offsets ? ptr_of<int>(*offsets) : nullptr, B, S, pd,
                        combiner, ptr_of<float>(out), out_ld, cur_stream());
  });
  m.def("pool_bwd", [](at::Tensor gU, int gstride, at::Tensor inverse, c10::optional<at::Tensor> offsets, int B, int S, int pd,
                       int dim, int combiner, at::Tensor gout, int gout_ld) {
    c10::cuda::CUDAGuard guard(gU.device());
    TORCH_CHECK(gstride % 4 == 0 && reinterpret_cast<uintptr_t>(gU.data_ptr()) % 16 == 0, "pool_bwd: rows of gU must be whole 16-byte pieces");
    tn::launch_pool_bwd(ptr_of<float>(gU), gstride, ptr_of<int>(inverse), offsets ? ptr_of<int>(*offsets) : nullptr, B, S, pd,
                        dim, combiner, ptr_of<float>(gout), gout_ld, cur_stream());
  });
  m.def("seq_bwd", [](at::Tensor gU, int gstride, at::Tensor inverse, at::Tensor offsets, int B, int T, int pd, int dim,
                      at::Tensor gout) {
    c10::cuda::CUDAGuard guard(gU.device());
    tn::launch_seq_bwd(ptr_of<float>(gU), gstride, ptr_of<int>(inverse), ptr_of<int>(offsets), B, T, pd, dim,
                       ptr_of<float>(gout), cur_stream());
  });
  m.def("table_insert_keys", [](py::dict table, at::Tensor keys, at::Tensor out_rows, at::Tensor status) {
    c10::cuda::CUDAGuard guard(keys.device());
    tn::launch_table_insert_keys(table_from_dict(table), ptr_of<long long>(keys), (int)keys.numel(), ptr_of<int>(out_rows),
                                 ptr_of<int>(status), cur_stream());
  });
  m.def("table_lookup", [](py::dict table, at::Tensor keys, at::Tensor out_rows) {
    c10::cuda::CUDAGuard guard(keys.device());
    tn::launch_table_lookup(table_from_dict(table), ptr_of<long long>(keys), (int)keys.numel(), ptr_of<int>(out_rows), cur_stream());
  });
  m.def("table_rebuild_index", [](py::dict table, int n, at::Tensor status) {
    tn::TableView t = table_from_dict(table);
    TORCH_CHECK(n >= 0 && n <= t.row_cap, "table_rebuild_index: more rows than the slab holds");
    c10::cuda::CUDAGuard guard(status.device());
    tn::launch_table_rebuild_index(t, n, ptr_of<int>(status), cur_stream());
  }, "fill an all-empty key array from the signs of rows [0, n)");
  m.def("table_keep_mask", [](py::dict table, int kind, bool evict, float show_threshold, int no_show_days, int logic, int n,
                              at::Tensor keep) {
    TORCH_CHECK(keep.scalar_type() == at::kByte && keep.numel() >= n, "table_keep_mask: keep must be uint8[n]");
    tn::ExportRule rule{evict ? 1 : 0, show_threshold, no_show_days, logic};
    c10::cuda::CUDAGuard guard(keep.device());
    tn::launch_table_keep_mask(table_from_dict(table), kind, rule, n, keep.data_ptr<unsigned char>(), cur_stream());
  }, "keep[r] = 0 for the rows the save-time eviction rule drops");
  m.def("table_decay", [](py::dict table, int kind, float rate, int delta_days) {
    tn::launch_table_decay(table_from_dict(table), kind, rate, delta_days, cur_stream());
  });
  m.def("table_export", [](py::dict table, int kind, bool evict, float show_threshold, int no_show_days, int logic, int r0, int r1,
                           at::Tensor counts, at::Tensor cursors, at::Tensor out_keys, at::Tensor out_rows) {
    TORCH_CHECK(counts.numel() >= 8 && cursors.numel() >= 8 && out_rows.dim() == 2 && out_rows.is_contiguous(), "table_export buffers");
    TORCH_CHECK(out_keys.numel() >= r1 - r0 && out_rows.size(0) >= r1 - r0, "table_export: staging buffers smaller than the row range");
    tn::ExportRule rule{evict ? 1 : 0, show_threshold, no_show_days, logic};
    c10::cuda::CUDAGuard guard(out_rows.device());
    tn::launch_table_export(table_from_dict(table), kind, rule, r0, r1, ptr_of<int>(counts), ptr_of<int>(cursors),
                            ptr_of<unsigned long long>(out_keys), ptr_of<float>(out_rows), (int)out_rows.size(1), cur_stream());
    g_launches.fetch_add(1, std::memory_order_relaxed);
  }, "filter rows [r0, r1) by the save-time eviction rule and pack them grouped by block file");
  m.def("fm_fwd", [](at::Tensor E, int ld, int B, int F, int D, at::Tensor out) {
    c10::cuda::CUDAGuard guard(E.device());
    tn::launch_fm_fwd(ptr_of<float>(E), ld, B, F, D, ptr_of<float>(out), cur_stream());
  });
  m.def("fm_bwd", [](at::Tensor E, int ld, int B, int F, int D, at::Tensor gout, at::Tensor gE, int gld, bool accumulate) {
    c10::cuda::CUDAGuard guard(E.device());
    tn::launch_fm_bwd(ptr_of<float>(E), ld, B, F, D, ptr_of<float>(gout), ptr_of<float>(gE), gld, accumulate, cur_stream());
  });
  auto concat_like = [](bool split) {
    return [split](std::vector<c10::optional<at::Tensor>> pieces, std::vector<int> widths, std::vector<int> lds, at::Tensor out,
                   int B, int ld_out, int ones_col) {
      TORCH_CHECK(pieces.size() <= (size_t)tn::kMaxPieces && pieces.size() == widths.size() && lds.size() == widths.size(),
                  "concat: at most 6 pieces");
      c10::cuda::CUDAGuard guard(out.device());
      tn::ConcatArgs a{};
      a.B = B; a.n_pieces = (int)pieces.size(); a.out = out.data_ptr(); a.ld_out = ld_out; a.ones_col = ones_col;
      for (size_t p = 0; p < pieces.size(); ++p) {
        a.width[p] = widths[p]; a.ld[p] = lds[p];
        if (pieces[p].has_value()) {
          a.ptr[p] = pieces[p]->data_ptr();
          a.is_bf16[p] = pieces[p]->scalar_type() == at::kBFloat16;
          TORCH_CHECK(a.is_bf16[p] || pieces[p]->scalar_type() == at::kFloat, "concat: fp32 or bf16 pieces");
        } else {
          a.ptr[p] = nullptr; a.is_bf16[p] = 0;
        }
      }
      if (split) tn::launch_split_cast(a, cur_stream()); else tn::launch_concat_cast(a, cur_stream());
    };
  };
  m.def("concat_cast", concat_like(false));
  m.def("split_cast", concat_like(true));
  m.def("gemv_fwd", [](at::Tensor Z, int ld, int B, int K, at::Tensor w, at::Tensor y) {
    c10::cuda::CUDAGuard guard(Z.device());
    tn::launch_gemv_fwd(Z.data_ptr(), ld, B, K, ptr_of<float>(w), ptr_of<float>(y), cur_stream());
  });
  m.def("gemv_bwd", [](at::Tensor Z, int ld, int B, int K, at::Tensor w, at::Tensor dy, at::Tensor dZ, at::Tensor gw, int relu_cols) {
    c10::cuda::CUDAGuard guard(Z.device());
    tn::launch_gemv_bwd(Z.data_ptr(), ld, B, K, ptr_of<float>(w), ptr_of<float>(dy), dZ.data_ptr(), ptr_of<float>(gw), relu_cols,
                        cur_stream());
  });
  m.def("bce", [](at::Tensor logit, at::Tensor label, c10::optional<at::Tensor> pred, c10::optional<at::Tensor> dlogit,
                  float grad_scale, at::Tensor sums) {
    c10::cuda::CUDAGuard guard(logit.device());
    TORCH_CHECK(label.numel() >= logit.numel() && label.scalar_type() == at::kFloat && label.is_contiguous(), "bce: a label per logit");
    tn::launch_bce(ptr_of<float>(logit), ptr_of<float>(label), (int)logit.numel(), pred ? ptr_of<float>(*pred) : nullptr,
                   dlogit ? ptr_of<float>(*dlogit) : nullptr, grad_scale, ptr_of<float>(sums), hist_bins(sums), cur_stream());
  });
  m.attr("EMBED_INPUT_COLUMNS") = tn::kEmbedInputColumns;
  m.def("embed_input_bwd", [](at::Tensor inverse, c10::optional<at::Tensor> offsets, int B, int S, int D, int dim, int combiner, at::Tensor dX0,
                              c10::optional<at::Tensor> E, c10::optional<at::Tensor> fsum, c10::optional<at::Tensor> gfm,
                              c10::optional<at::Tensor> gE, c10::optional<at::Tensor> dL, int lin_col, at::Tensor gU, int gstride) {
    c10::cuda::CUDAGuard guard(dX0.device());
    auto f32 = [](const c10::optional<at::Tensor>& t, int64_t n) { return !t || (t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() >= n); };
    auto cols = [&](const c10::optional<at::Tensor>& t) { return !t || (f32(t, 0) && t->dim() == 2 && t->size(0) == B && t->size(1) >= (int64_t)S * D); };
    TORCH_CHECK(dX0.scalar_type() == at::kBFloat16 && dX0.dim() == 2 && dX0.stride(1) == 1 && dX0.size(0) == B && dX0.size(1) >= (int64_t)S * D &&
                    cols(E) && cols(gE) && (!E || !gE || E->size(1) == gE->size(1)) && f32(fsum, (int64_t)B * ((D + 3) / 4 * 4)) && f32(gfm, B) &&
                    f32(dL, (int64_t)B * S) && (!gfm || (E && fsum)), "embed_input_bwd: gradients");
    tn::EmbedGrad a = {};
    a.inverse = ptr_of<int>(inverse); a.offsets = offsets ? ptr_of<int>(*offsets) : nullptr;
    a.B = B; a.S = S; a.D = D; a.dim = dim; a.combiner = combiner;
    a.dX0 = dX0.data_ptr(); a.ld = (int)dX0.stride(0);
    a.E = E ? ptr_of<float>(*E) : nullptr; a.fsum = fsum ? ptr_of<float>(*fsum) : nullptr; a.gfm = gfm ? ptr_of<float>(*gfm) : nullptr;
    a.gE = gE ? ptr_of<float>(*gE) : nullptr; a.ldE = E ? (int)E->size(1) : gE ? (int)gE->size(1) : 0; a.dL = dL ? ptr_of<float>(*dL) : nullptr; a.lin_col = lin_col;
    a.gU = ptr_of<float>(gU); a.gstride = gstride;
    if (const char* err = tn::launch_embed_input_bwd(a, cur_stream())) throw std::runtime_error(err);
  });
  {
    auto pieces_of = [](const std::vector<at::Tensor>& pieces, const std::vector<int>& widths, at::Tensor w) {
      TORCH_CHECK(!pieces.empty() && pieces.size() <= tn::kMaxHeadPieces && widths.size() == pieces.size(), "head: number of pieces");
      TORCH_CHECK(w.scalar_type() == at::kFloat && w.is_contiguous(), "head: weight must be contiguous fp32");
      tn::HeadArgs a = {};
      a.B = (int)pieces[0].size(0); a.n = (int)pieces.size(); a.K = (int)w.numel() - 1;
      a.w = ptr_of<float>(w);
      for (int p = 0; p < a.n; ++p) {
        const at::Tensor& t = pieces[p];
        TORCH_CHECK(t.is_cuda() && t.dim() == 2 && t.size(0) == a.B && (t.stride(1) == 1 || t.size(1) == 1) && widths[p] <= t.size(1) &&
                        (t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat), "head: piece ", p);
        a.src[p] = t.data_ptr();
        a.width[p] = widths[p];
        a.ld[p] = a.gld[p] = (int)t.stride(0);
        a.kind[p] = t.scalar_type() == at::kBFloat16 ? tn::kHeadBf16 : tn::kHeadF32;
      }
      return a;
    };
    m.attr("HEAD_MAX_SPAN") = tn::kMaxHeadSpan;
    m.attr("HEAD_COPIES") = tn::kHeadCopies;
    m.def("head_loss", [pieces_of](std::vector<at::Tensor> pieces, std::vector<int> widths, at::Tensor w, at::Tensor label,
                                   std::vector<c10::optional<at::Tensor>> grads, bool relu_first, at::Tensor gw, at::Tensor sums,
                                   at::Tensor loss_out, at::Tensor scratch, c10::optional<at::Tensor> pred) {
      c10::cuda::CUDAGuard guard(w.device());
      tn::HeadArgs a = pieces_of(pieces, widths, w);
      TORCH_CHECK(grads.size() == pieces.size() && gw.is_contiguous() && gw.numel() == w.numel() && gw.scalar_type() == at::kFloat &&
                      label.is_contiguous() && label.scalar_type() == at::kFloat && label.numel() == a.B, "head_loss: gradients or labels");
      int64_t span = 0;
      for (int p = 0; p < a.n; ++p) {
        span += (widths[p] + 7) / 8 * 8;
        if (!grads[p]) continue;
        const at::Tensor& g = *grads[p];
        TORCH_CHECK(g.dim() == 2 && g.size(0) == a.B && g.size(1) >= widths[p] && (g.stride(1) == 1 || g.size(1) == 1) &&
                        g.scalar_type() == pieces[p].scalar_type(), "head_loss: gradient of piece ", p);
        a.grad[p] = g.data_ptr();
        a.gld[p] = (int)g.stride(0);
      }
      TORCH_CHECK(scratch.scalar_type() == at::kFloat && scratch.numel() >= 4 + tn::kHeadCopies * (span + 8) &&
                      (reinterpret_cast<uintptr_t>(scratch.data_ptr()) & 15) == 0, "head_loss: scratch too small");
      a.relu_first = relu_first;
      a.label = ptr_of<float>(label); a.gw = ptr_of<float>(gw); a.sums = ptr_of<float>(sums); a.nbins = hist_bins(sums);
      TORCH_CHECK(!pred || (pred->is_contiguous() && pred->numel() == a.B && pred->scalar_type() == at::kFloat), "head_loss: pred");
      a.pred = pred ? ptr_of<float>(*pred) : nullptr;
      a.loss_out = ptr_of<float>(loss_out); a.scratch = ptr_of<float>(scratch);
      if (const char* err = tn::launch_head_loss(a, cur_stream())) throw std::runtime_error(err);
    });
    m.def("head_score", [pieces_of](std::vector<at::Tensor> pieces, std::vector<int> widths, at::Tensor w, at::Tensor logits) {
      c10::cuda::CUDAGuard guard(w.device());
      tn::HeadArgs a = pieces_of(pieces, widths, w);
      TORCH_CHECK(logits.is_contiguous() && logits.numel() == a.B && logits.scalar_type() == at::kFloat, "head_score: logits");
      a.pred = ptr_of<float>(logits);
      if (const char* err = tn::launch_head_score(a, cur_stream())) throw std::runtime_error(err);
    });
  }
  m.def("unique_assign", [](at::Tensor ids, c10::optional<at::Tensor> labels, at::Tensor dd_keys, at::Tensor dd_vals, at::Tensor uniq,
                            at::Tensor inverse, c10::optional<at::Tensor> show, c10::optional<at::Tensor> click, at::Tensor count,
                            at::Tensor status) {
    c10::cuda::CUDAGuard guard(ids.device());
    const int64_t cap2 = dd_keys.numel();
    TORCH_CHECK(cap2 >= 2 && (cap2 & (cap2 - 1)) == 0 && dd_vals.numel() >= cap2, "unique_assign: scratch must be a power of two");
    TORCH_CHECK(ids.scalar_type() == at::kLong && ids.is_contiguous() && inverse.numel() >= ids.numel(), "unique_assign: bad ids / inverse");
    g_launches.fetch_add(2, std::memory_order_relaxed);
    tn::launch_unique_assign(ptr_of<long long>(ids), (int)ids.numel(), labels ? ptr_of<float>(*labels) : nullptr,
                             ptr_of<unsigned long long>(dd_keys), ptr_of<int>(dd_vals), (unsigned)cap2,
                             ptr_of<unsigned long long>(uniq), (int)uniq.numel(), ptr_of<int>(inverse),
                             show ? ptr_of<float>(*show) : nullptr, click ? ptr_of<float>(*click) : nullptr, ptr_of<int>(count),
                             ptr_of<int>(status), cur_stream());
  });
  m.def("dict_lookup_pool", [](py::dict table, at::Tensor ids, c10::optional<at::Tensor> offsets, int B, int S, int combiner,
                               at::Tensor out, int ld_out, int ones_col) {
    c10::cuda::CUDAGuard guard(ids.device());
    tn::TableView t = table_from_dict(table);
    TORCH_CHECK(t.dim % 4 == 0, "dict_lookup_pool: dim must be a multiple of 4");
    tn::launch_dict_lookup_pool(t, ptr_of<long long>(ids), offsets ? ptr_of<int>(*offsets) : nullptr, B, S, combiner, out.data_ptr(),
                                ld_out, ones_col, cur_stream());
  });
  m.def("sigmoid", [](at::Tensor x, at::Tensor y) {
    c10::cuda::CUDAGuard guard(x.device());
    tn::launch_sigmoid(ptr_of<float>(x), ptr_of<float>(y), (int)x.numel(), cur_stream());
  });
  m.def("cross_v2_bwd_elem", [](at::Tensor g, at::Tensor u, at::Tensor x0, at::Tensor gx0, at::Tensor du, bool first) {
    TORCH_CHECK(g.is_contiguous() && u.is_contiguous() && x0.is_contiguous() && gx0.is_contiguous() && du.is_contiguous(), "contiguous operands");
    TORCH_CHECK(g.numel() % 8 == 0 && u.numel() == g.numel() && x0.numel() == g.numel() && gx0.numel() == g.numel() && du.numel() == g.numel(), "sizes");
    TORCH_CHECK(g.scalar_type() == at::kBFloat16 && gx0.scalar_type() == at::kFloat, "g / u / x0 / du are bf16, gx0 is fp32");
    c10::cuda::CUDAGuard guard(g.device());
    tn::launch_cross_v2_bwd_elem(g.data_ptr(), u.data_ptr(), x0.data_ptr(), ptr_of<float>(gx0), du.data_ptr(), g.numel(), first ? 1 : 0, cur_stream());
  });
  m.def("cross_v2_du", [](at::Tensor g, at::Tensor x0, at::Tensor du) {
    TORCH_CHECK(g.is_contiguous() && x0.is_contiguous() && du.is_contiguous(), "contiguous operands");
    TORCH_CHECK(g.numel() % 8 == 0 && x0.numel() == g.numel() && du.numel() == g.numel(), "sizes");
    TORCH_CHECK(g.scalar_type() == at::kBFloat16 && x0.scalar_type() == at::kBFloat16 && du.scalar_type() == at::kBFloat16, "g / x0 / du are bf16");
    c10::cuda::CUDAGuard guard(g.device());
    tn::launch_cross_v2_du(g.data_ptr(), x0.data_ptr(), du.data_ptr(), g.numel(), cur_stream());
  });
  m.attr("MAX_CROSS_LAYERS") = (int)tn::kMaxCrossLayers;
  m.def("cross_v2_bwd_sum", [](std::vector<at::Tensor> g, std::vector<at::Tensor> u, at::Tensor g0, at::Tensor out) {
    TORCH_CHECK(g.size() == u.size() && g.size() <= (size_t)tn::kMaxCrossLayers, "cross_v2_bwd_sum: one u per g, at most 8 layers");
    TORCH_CHECK(g0.is_contiguous() && out.is_contiguous() && g0.numel() % 8 == 0 && out.numel() == g0.numel(), "operands");
    TORCH_CHECK(g0.scalar_type() == at::kBFloat16 && out.scalar_type() == at::kBFloat16, "bf16 operands");
    tn::CrossTerms t{};
    t.n = (int)g.size();
    for (size_t l = 0; l < g.size(); ++l) {
      for (const at::Tensor* x : {&g[l], &u[l]})
        TORCH_CHECK(x->is_contiguous() && x->numel() == g0.numel() && x->scalar_type() == at::kBFloat16, "cross_v2_bwd_sum: contiguous bf16 terms");
      t.g[l] = g[l].data_ptr();
      t.u[l] = u[l].data_ptr();
    }
    c10::cuda::CUDAGuard guard(g0.device());
    tn::launch_cross_v2_bwd_sum(t, g0.data_ptr(), out.data_ptr(), g0.numel(), cur_stream());
  });
  m.def("cross_v2_bwd_final", [](at::Tensor gx0, at::Tensor g, at::Tensor out) {
    TORCH_CHECK(gx0.is_contiguous() && g.is_contiguous() && out.is_contiguous() && g.numel() % 8 == 0 && gx0.numel() == g.numel() && out.numel() == g.numel(), "operands");
    c10::cuda::CUDAGuard guard(g.device());
    tn::launch_cross_v2_bwd_final(ptr_of<float>(gx0), g.data_ptr(), out.data_ptr(), g.numel(), cur_stream());
  });
  m.def("relu_mask", [](at::Tensor g, at::Tensor y, at::Tensor out) {
    c10::cuda::CUDAGuard guard(g.device());
    TORCH_CHECK(g.numel() % 8 == 0 && g.numel() == y.numel() && g.numel() == out.numel(), "relu_mask: numel must be a multiple of 8");
    for (const at::Tensor& v : {g, y, out})
      TORCH_CHECK(v.is_contiguous() && v.scalar_type() == at::kBFloat16 && reinterpret_cast<uintptr_t>(v.data_ptr()) % 16 == 0,
                  "relu_mask: contiguous bf16 tensors on 16 bytes");
    tn::launch_relu_mask(g.data_ptr(), y.data_ptr(), out.data_ptr(), g.numel(), cur_stream());
  });
  {
    // ws, bs (and their gradients): fp32 vectors of the input's width, one per layer
    auto net = [](const at::Tensor& x0, const std::vector<at::Tensor>& ws, const std::vector<at::Tensor>& bs) {
      TORCH_CHECK(x0.is_cuda() && x0.scalar_type() == at::kFloat && x0.is_contiguous() && x0.dim() == 2 && x0.size(0) >= 1 &&
                      x0.size(1) <= tn::kCrossNetColumns, "cross_v1_net: input must be fp32 [B, D], D at most 1024");
      TORCH_CHECK(!ws.empty() && ws.size() <= (size_t)tn::kMaxCrossLayers && bs.size() == ws.size(), "cross_v1_net: one to eight layers");
      tn::CrossNet n{};
      n.layers = (int)ws.size();
      for (size_t l = 0; l < ws.size(); ++l) {
        for (const at::Tensor& v : {ws[l], bs[l]})
          TORCH_CHECK(v.is_cuda() && v.scalar_type() == at::kFloat && v.is_contiguous() && v.numel() == x0.size(1), "cross_v1_net: layer vectors");
        n.w[l] = ptr_of<float>(ws[l]);
        n.b[l] = ptr_of<float>(bs[l]);
      }
      return n;
    };
    m.def("cross_v1_net_fwd", [net](at::Tensor x0, std::vector<at::Tensor> ws, std::vector<at::Tensor> bs, at::Tensor y, at::Tensor dots) {
      c10::cuda::CUDAGuard guard(x0.device());
      tn::launch_cross_v1_net_fwd(net(x0, ws, bs), ptr_of<float>(x0), (int)x0.size(0), (int)x0.size(1), ptr_of<float>(y), ptr_of<float>(dots),
                                  cur_stream());
    });
    m.def("cross_v1_net_bwd", [net](at::Tensor x0, std::vector<at::Tensor> ws, std::vector<at::Tensor> bs, at::Tensor dots, at::Tensor gy,
                                    at::Tensor gx0, std::vector<at::Tensor> gws, std::vector<at::Tensor> gbs, at::Tensor t_row) {
      c10::cuda::CUDAGuard guard(x0.device());
      tn::CrossNet n = net(x0, ws, bs);
      TORCH_CHECK(gy.is_contiguous() && gy.scalar_type() == at::kFloat && (int)gws.size() == n.layers && (int)gbs.size() == n.layers, "cross_v1_net: gradients");
      for (int l = 0; l < n.layers; ++l) {
        for (const at::Tensor& g : {gws[l], gbs[l]})
          TORCH_CHECK(g.is_cuda() && g.is_contiguous() && g.scalar_type() == at::kFloat && g.numel() == x0.size(1), "cross_v1_net: gradients");
        n.gw[l] = ptr_of<float>(gws[l]);
        n.gb[l] = ptr_of<float>(gbs[l]);
      }
      tn::launch_cross_v1_net_bwd(n, ptr_of<float>(x0), (int)x0.size(0), (int)x0.size(1), ptr_of<float>(dots), ptr_of<float>(gy),
                                  ptr_of<float>(gx0), ptr_of<float>(t_row), cur_stream());
      g_launches.fetch_add(1, std::memory_order_relaxed);
    });
  }
  m.def("cross_v1_fwd", [](at::Tensor x0, at::Tensor xl, at::Tensor w, at::Tensor bias, at::Tensor y, at::Tensor dot) {
    c10::cuda::CUDAGuard guard(x0.device());
    tn::launch_cross_v1_fwd(ptr_of<float>(x0), ptr_of<float>(xl), ptr_of<float>(w), ptr_of<float>(bias), (int)x0.size(0),
                            (int)x0.size(1), ptr_of<float>(y), ptr_of<float>(dot), cur_stream());
  });
  m.def("cross_v1_bwd", [](at::Tensor x0, at::Tensor xl, at::Tensor w, at::Tensor dot, at::Tensor gy, at::Tensor gx0,
                           at::Tensor gxl, at::Tensor gw, at::Tensor gb) {
    c10::cuda::CUDAGuard guard(x0.device());
    at::Tensor scratch;
    if (x0.size(1) > tn::kCrossV1OneTile) scratch = at::empty({x0.size(0)}, x0.options());
    tn::launch_cross_v1_bwd(ptr_of<float>(x0), ptr_of<float>(xl), ptr_of<float>(w), ptr_of<float>(dot), ptr_of<float>(gy),
                            (int)x0.size(0), (int)x0.size(1), ptr_of<float>(gx0), ptr_of<float>(gxl), ptr_of<float>(gw),
                            ptr_of<float>(gb), scratch.defined() ? ptr_of<float>(scratch) : nullptr, cur_stream());
  });
}
