// Batches of independent operators: one persistent launch per (dimension, order) class.
//
// Operators on the any-dimension Kronecker kernel are grouped by (D, N, kernel variant); each group's
// parameter table (the operators' forward parameters, x and y patched per apply) and the prefix sums
// of their element batches live on the device, and one launch of the group's batch kernel walks every
// element batch of every operator of the group.  Operators on another kernel are applied one
// launch each.  The launches are independent, so they are spread over the caller's stream and a
// few more that fork from it and join it again (largest operators first): a launch's tail, and the
// small operators, run beside the others (24 systems of 2D to 4D, p = 1..5: 216 us, 332 us in one
// stream).  Members that repeat an operator whose applies share device memory keep one stream.  Results equal those of the operators' own applies bit for bit (same arithmetic).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <new>
#include <vector>

#include "dgop_internal.h"

using namespace dgop;

namespace {
struct BatchGroup {
  const KronNDEntry<double>* entry = nullptr;
  int variant = 0;
  std::vector<int> members;                 // indices into the batch
  std::vector<KronNDParams<double>> table;  // host copy (x, y patched per apply)
  std::vector<int64_t> first;
  KronNDParams<double>* d_table = nullptr;  // part of the batch's table
  int64_t* d_first = nullptr;
  KronNDParams<double>* h_pinned = nullptr;  // part of the staging of the table's upload
  int eb = 1;
  size_t smem = 0;
  dim3 grid, block;
};
// Small 3D register-kernel operators of one order in one launch (kron3d_pack_kernel).
struct BatchPack {
  const KronVariant<double>* variant = nullptr;
  std::vector<int> members;
  bool sep = false;                 // with a separate mass term
  std::vector<double> parameters;   // of the launch (KronVariant::fill_pack); x and y set per apply
  dim3 grid, block;
  size_t smem = 0;
  KronHead<double>& head(size_t k) {
    return *reinterpret_cast<KronHead<double>*>(reinterpret_cast<unsigned char*>(parameters.data()) + k * variant->pack_stride);
  }
};
}  // namespace

struct dgop_batch {
  std::vector<dgop_operator*> ops;
  std::vector<int> versions;  // of the operators' launch configurations, when the batch was made
  std::vector<BatchGroup> groups;
  std::vector<BatchPack> packs;
  std::vector<int> singles;  // operators applied one launch each
  std::vector<size_t> lane;  // stream of every launch: the singles', the groups', the packs' (0: the caller's)
  cudaEvent_t uploaded = nullptr;  // the staging buffer has been read
  cudaEvent_t applied = nullptr;   // the last apply's launches are done with the device tables
  std::mutex mutex;                // an apply's events and staging are one thread's at a time
  // every group's parameter table, uploaded by one copy
  KronNDParams<double>* d_tables = nullptr;
  KronNDParams<double>* h_tables = nullptr;
  size_t table_bytes = 0;
  // side streams of an apply, their fork and join events
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> joined;
  cudaEvent_t forked = nullptr;
};

namespace {

#define DGOP_CUDA_B(call)                               \
  do {                                                  \
    cudaError_t _e = (call);                            \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)

void release(dgop_batch* b) {
  for (auto& g : b->groups) {
    if (g.d_first) cudaFree(g.d_first);
  }
  if (b->d_tables) cudaFree(b->d_tables);
  if (b->h_tables) cudaFreeHost(b->h_tables);
  for (cudaStream_t s : b->side) cudaStreamDestroy(s);
  for (cudaEvent_t e : b->joined) cudaEventDestroy(e);
  if (b->forked) cudaEventDestroy(b->forked);
  if (b->uploaded) cudaEventDestroy(b->uploaded);
  if (b->applied) cudaEventDestroy(b->applied);
}

// The split variant's own launch prefetches its elements and reads its parameters from constant memory, the
// batch kernel does neither, so a group pays where the launches it saves (5 to 7 us of the host each) outweigh
// that: members up to about 3 us of kernel, four of them at least, in a batch that keeps the host busier
// than the GPU (below about 300,000 dofs per launch, 5 us at 60 GDoF/s; 24 systems of 671,000 dofs on
// average 218 one launch each, 228 with its two small groups).  Us per batched apply, one launch
// each / grouped: 32 systems of 2D p = 3, 128,000 dofs 158 / 99, 320,000 dofs 171 / 208; of 2D p = 5,
// 144,000 dofs 167 / 158, 288,000 dofs 194 / 287; 4D p = 2, 81,000 dofs (64 systems) 326 / 205, 324,000
// dofs 268 / 289; 512 of 2D p = 2, 9,000 dofs 2514 / 1119.  (2D p = 1: grouped from two members on, up to the
// limit of the other variants.)
constexpr int64_t kSplitGroupDofs = 200000;
constexpr size_t kSplitGroupMembers = 4;
constexpr int64_t kSplitMeanDofs = 300000;

int setup(dgop_batch* b) {
  int sms = 0, dev = 0;
  DGOP_CUDA_B(cudaGetDevice(&dev));
  DGOP_CUDA_B(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int max_smem = 0;
  DGOP_CUDA_B(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  int64_t mean = 0;  // dofs per operator
  for (const dgop_operator* op : b->ops) mean += op->sp.ndofs;
  mean /= (int64_t)b->ops.size();
  std::map<const void*, int> per_sm_of;  // resident CTAs per SM of each batch kernel used
  std::map<std::tuple<int, int, int>, int> index;
  for (int i = 0; i < (int)b->ops.size(); ++i) {
    dgop_operator* op = b->ops[i];
    const int v = op->n64.variant;
    if (op->kernel != DGOP_KERNEL_KRONND || !op->n64.ready || !op->n64.entry->launch_batch[v]) {
      b->singles.push_back(i);
      continue;
    }
    const void* fn = op->n64.entry->func_batch[v];
    auto pit = per_sm_of.find(fn);
    if (pit == per_sm_of.end()) {
      cudaFuncAttributes fa{};
      DGOP_CUDA_B(cudaFuncGetAttributes(&fa, fn));
      DGOP_CUDA_B(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       max_smem - (int)fa.sharedSizeBytes));
      int per_sm = 0;
      DGOP_CUDA_B(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, op->n64.var[v].threads,
                                                                op->n64.var[v].smem));
      pit = per_sm_of.emplace(fn, per_sm < 1 ? 1 : per_sm).first;
    }
    // an instance whose element batches fill every CTA slot twice over keeps its own launch (its
    // parameters in constant memory, no per-batch instance lookup): the persistent kernel gains
    // nothing there and measured a few per cent slower
    const int64_t eb = op->n64.var[v].eb;
    const bool split = v == 5 && !(op->sp.D == 2 && op->sp.n == 2);
    if ((op->sp.nelem + eb - 1) / eb >= 2 * (int64_t)sms * pit->second || (split && (op->sp.ndofs > kSplitGroupDofs || mean > kSplitMeanDofs))) {
      b->singles.push_back(i);
      continue;
    }
    const auto key = std::make_tuple(op->sp.D, op->sp.n, v);
    auto it = index.find(key);
    if (it == index.end()) {
      it = index.emplace(key, (int)b->groups.size()).first;
      b->groups.emplace_back();
      b->groups.back().entry = op->n64.entry;
      b->groups.back().variant = v;
      b->groups.back().eb = op->n64.var[v].eb;
      b->groups.back().smem = op->n64.var[v].smem;
      b->groups.back().block = dim3(op->n64.var[v].threads);
    }
    BatchGroup& group = b->groups[it->second];
    group.members.push_back(i);
  }
  // few operators of the split variant keep their own launches
  for (size_t k = 0; k < b->groups.size();) {
    const auto& m = b->groups[k].members;
    const dgop_space& sp = b->ops[m[0]]->sp;
    if (b->groups[k].variant == 5 && m.size() < (sp.D == 2 && sp.n == 2 ? 2 : kSplitGroupMembers)) {
      b->singles.insert(b->singles.end(), m.begin(), m.end());
      b->groups.erase(b->groups.begin() + (long)k);
    } else {
      ++k;
    }
  }
  // Small 3D register-kernel operators above p = 3: several in one launch, under the split variant's rules.
  // A launch of 30 KB of parameters costs the host 7 to 17 us, seven or ten launches of one operator 5 us each (us,
  // one launch each / together: 64 systems of p = 4, 14,000 dofs 347 / 247, 129,000 dofs 345 / 190; of p = 5, 25,000
  // dofs 336 / 196; 512 of p = 4, 135,000 dofs 2621 / 1502).
  std::map<std::pair<int, bool>, std::vector<int>> small;
  for (size_t k = 0; k < b->singles.size();) {
    const int i = b->singles[k];
    const dgop_operator* op = b->ops[i];
    const auto& K = op->k64;
    if (op->kernel == DGOP_KERNEL_KRON && K.ready && K.entry->v[K.variant].launch_pack && !K.params.general &&
        !K.factors && op->sp.ndofs <= kSplitGroupDofs && mean <= kSplitMeanDofs) {
      const auto& p = K.params;
      small[{op->sp.n, p.has_adv && p.has_mass && !p.mass_merged}].push_back(i);
      b->singles.erase(b->singles.begin() + (long)k);
    } else {
      ++k;
    }
  }
  for (const auto& [key, members] : small) {
    if (members.size() < kSplitGroupMembers) {
      b->singles.insert(b->singles.end(), members.begin(), members.end());
      continue;
    }
    for (size_t m = 0; m < members.size();) {
      BatchPack pack;
      const auto& K0 = b->ops[members[m]]->k64;
      pack.variant = &K0.entry->v[K0.variant];
      const auto& L = K0.launch[K0.variant];
      pack.block = L.block;
      pack.smem = L.smem;
      const void* fn = pack.variant->func_pack[key.second ? 1 : 0];
      cudaFuncAttributes fa{};
      DGOP_CUDA_B(cudaFuncGetAttributes(&fa, fn));
      DGOP_CUDA_B(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes));
      unsigned blocks = 1;
      for (; m < members.size() && (int)pack.members.size() < pack.variant->pack; ++m) {
        pack.members.push_back(members[m]);
        blocks = std::max(blocks, b->ops[members[m]]->k64.launch[K0.variant].grid.x);
      }
      pack.grid = dim3(blocks, (unsigned)pack.members.size());
      pack.sep = key.second;
      pack.parameters.resize((pack.variant->pack_bytes + sizeof(double) - 1) / sizeof(double));
      std::vector<KronParams<double>> params;
      for (int i : pack.members) {
        params.push_back(b->ops[i]->k64.params);
        params.back().alpha = 1.0;
        params.back().beta_y = 0.0;
        params.back().flags = b->ops[i]->flags;
        params.back().e_begin = 0;
        params.back().nelem = b->ops[i]->sp.nelem;
      }
      std::vector<const KronParams<double>*> at;
      for (const auto& p : params) at.push_back(&p);
      pack.variant->fill_pack(at.data(), (int)at.size(), pack.parameters.data());
      b->packs.push_back(std::move(pack));
    }
  }
  for (auto& g : b->groups) {
    g.first.push_back(0);
    for (int i : g.members) {
      dgop_operator* op = b->ops[i];
      KronNDParams<double> p = op->n64.params;
      p.eb = g.eb;
      p.e_begin = 0;
      p.nelem = op->sp.nelem;
      p.alpha = 1.0;
      p.beta_y = 0.0;
      p.flags = op->flags;
      p.skip = nullptr;
      g.table.push_back(p);
      g.first.push_back(g.first.back() + (op->sp.nelem + g.eb - 1) / g.eb);
    }
    b->table_bytes += sizeof(KronNDParams<double>) * g.table.size();
    DGOP_CUDA_B(cudaMalloc(&g.d_first, sizeof(int64_t) * g.first.size()));
    DGOP_CUDA_B(cudaMemcpy(g.d_first, g.first.data(), sizeof(int64_t) * g.first.size(), cudaMemcpyHostToDevice));
    const int per_sm = per_sm_of[g.entry->func_batch[g.variant]];
    g.grid = dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(g.first.back(), (int64_t)sms * per_sm)));
  }
  if (b->table_bytes) {
    DGOP_CUDA_B(cudaMalloc(&b->d_tables, b->table_bytes));
    DGOP_CUDA_B(cudaMallocHost(&b->h_tables, b->table_bytes));
    size_t at = 0;
    for (auto& g : b->groups) {
      g.d_table = b->d_tables + at;
      g.h_pinned = b->h_tables + at;
      at += g.table.size();
    }
  }
  DGOP_CUDA_B(cudaEventCreateWithFlags(&b->uploaded, cudaEventDisableTiming));
  DGOP_CUDA_B(cudaEventCreateWithFlags(&b->applied, cudaEventDisableTiming));
  // one launch per group and single operator: as many streams as launches, at most kStreams
  constexpr size_t kStreams = 6;
  std::stable_sort(b->singles.begin(), b->singles.end(),
                   [&](int i, int j) { return b->ops[i]->sp.ndofs > b->ops[j]->sp.ndofs; });
  const size_t launches = b->groups.size() + b->singles.size() + b->packs.size();
  for (size_t k = 1; k < std::min(launches, kStreams); ++k) {
    cudaStream_t s = nullptr;
    DGOP_CUDA_B(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    b->side.push_back(s);
    cudaEvent_t e = nullptr;
    DGOP_CUDA_B(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    b->joined.push_back(e);
  }
  DGOP_CUDA_B(cudaEventCreateWithFlags(&b->forked, cudaEventDisableTiming));
  // launches in turn over the streams; an operator whose applies write memory of its own keeps one
  // stream for all its members, which run in the order of the list there
  std::map<const dgop_operator*, size_t> kept;
  for (size_t k = 0, next = 0; k < launches; ++k) {
    size_t lane = next % (b->side.size() + 1);
    if (k < b->singles.size() && applies_share_memory(b->ops[b->singles[k]])) {
      const auto it = kept.emplace(b->ops[b->singles[k]], lane);
      if (!it.second) {
        b->lane.push_back(it.first->second);
        continue;
      }
    }
    b->lane.push_back(lane);
    ++next;
  }
  return DGOP_OK;
}

}  // namespace

extern "C" {

int dgop_batch_create(dgop_operator* const* ops, int count, dgop_batch** out) {
  if (!ops || !out || count < 1) {
    set_error("dgop_batch_create: bad arguments");
    return DGOP_ERR_ARG;
  }
  *out = nullptr;
  auto* b = new (std::nothrow) dgop_batch();
  if (!b) {
    set_error("host allocation failed");
    return DGOP_ERR_ALLOC;
  }
  for (int i = 0; i < count; ++i) {
    if (!ops[i]) {
      delete b;
      set_error("dgop_batch_create: null operator");
      return DGOP_ERR_ARG;
    }
    b->ops.push_back(ops[i]);
    b->versions.push_back(ops[i]->version);
  }
  const int rc = setup(b);
  if (rc != DGOP_OK) {
    release(b);
    delete b;
    return rc;
  }
  *out = b;
  return DGOP_OK;
}

int dgop_batch_groups(const dgop_batch* b) { return b ? (int)(b->groups.size() + b->packs.size()) : -1; }

int dgop_batch_apply(dgop_batch* b, const double* const* x, double* const* y, void* stream) {
  if (!b || !x || !y) {
    set_error("dgop_batch_apply: null argument");
    return DGOP_ERR_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lock(b->mutex);
  for (auto& g : b->groups)
    for (int i : g.members)
      if (!x[i] || !y[i] || x[i] == y[i]) {
        set_error("dgop_batch_apply: null or aliasing vectors");
        return DGOP_ERR_ARG;
      }
  // Under stream capture the groups' members are launched one by one (the same results): a table upload in the
  // graph would read whatever the staging buffer holds when the graph runs.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
  const bool grouped = capture == cudaStreamCaptureStatusNone && !b->groups.empty();
  if (grouped) {
    // the staging buffer of the previous apply may still be in flight
    DGOP_CUDA_B(cudaEventSynchronize(b->uploaded));
    for (auto& g : b->groups)
      for (size_t k = 0; k < g.members.size(); ++k) {
        const int i = g.members[k];
        g.h_pinned[k] = g.table[k];
        g.h_pinned[k].x = x[i];
        g.h_pinned[k].y = y[i];
      }
    // and its kernels, on whatever stream it ran, may still read the device tables
    DGOP_CUDA_B(cudaStreamWaitEvent(st, b->applied, 0));
    DGOP_CUDA_B(cudaMemcpyAsync(b->d_tables, b->h_tables, b->table_bytes, cudaMemcpyHostToDevice, st));
    DGOP_CUDA_B(cudaEventRecord(b->uploaded, st));
  }
  // fork the side streams, launch, and join them
  const size_t ns = b->side.size();
  int rc = DGOP_OK;
  auto keep = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && rc == DGOP_OK) rc = cuda_fail(e, what);
    return e == cudaSuccess;
  };
  size_t forked = 0;
  if (ns && keep(cudaEventRecord(b->forked, st), "batch fork"))
    while (forked < ns && keep(cudaStreamWaitEvent(b->side[forked], b->forked, 0), "batch fork")) ++forked;
  size_t next = 0;
  auto stream_of = [&]() {
    const size_t k = b->lane[next++];
    return k == 0 ? st : b->side[k - 1];
  };
  // single operators first: the largest are among them
  for (int i : b->singles) {
    if (rc != DGOP_OK) break;
    rc = dgop_apply(b->ops[i], x[i], y[i], stream_of());
  }
  // members whose kernel or variant was chosen anew since the batch was made apply on their own
  auto as_made = [&](const std::vector<int>& members) {
    for (int i : members)
      if (b->ops[i]->version != b->versions[i]) return false;
    return true;
  };
  for (auto& g : b->groups) {
    const bool one_launch = grouped && as_made(g.members);
    if (!one_launch)
      for (size_t k = 0; rc == DGOP_OK && k < g.members.size(); ++k) {
        dgop_operator* op = b->ops[g.members[k]];
        const size_t lane = applies_share_memory(op) ? 0 : k % (ns + 1);
        rc = dgop_apply(op, x[g.members[k]], y[g.members[k]], lane ? b->side[lane - 1] : st);
      }
    if (!one_launch) {
      ++next;
      continue;
    }
    if (rc != DGOP_OK) break;
    g.entry->launch_batch[g.variant](g.d_table, g.d_first, (int)g.members.size(), g.eb, g.grid, g.block, g.smem,
                                     stream_of());
    keep(cudaGetLastError(), "batch kernel launch");
  }
  for (auto& g : b->packs) {
    if (rc != DGOP_OK) break;
    const cudaStream_t q = stream_of();
    bool together = as_made(g.members);
    for (size_t k = 0; k < g.members.size(); ++k) {
      const int i = g.members[k];
      const uintptr_t ax = reinterpret_cast<uintptr_t>(x[i]), ay = reinterpret_cast<uintptr_t>(y[i]);
      together = together && ax && ay && ax != ay && ax % 16 == 0 && ay % 16 == 0;
      g.head(k).x = x[i];
      g.head(k).y = y[i];
    }
    if (together) {
      g.variant->launch_pack(g.parameters.data(), g.sep, g.grid, g.block, g.smem, q);
      keep(cudaGetLastError(), "batch kernel launch");
    } else {  // vectors off 16 bytes take another kernel, others are errors: each by its own apply
      for (size_t k = 0; rc == DGOP_OK && k < g.members.size(); ++k)
        rc = dgop_apply(b->ops[g.members[k]], x[g.members[k]], y[g.members[k]], q);
    }
  }
  // join every forked stream, also after an error: the caller's stream waits for what was queued
  for (size_t k = 0; k < forked; ++k)
    if (keep(cudaEventRecord(b->joined[k], b->side[k]), "batch join"))
      keep(cudaStreamWaitEvent(st, b->joined[k], 0), "batch join");
  if (grouped) keep(cudaEventRecord(b->applied, st), "batch event");
  return rc;
}

int dgop_batch_destroy(dgop_batch* b) {
  if (!b) return DGOP_OK;
  if (b->applied) cudaEventSynchronize(b->applied);
  release(b);
  delete b;
  return DGOP_OK;
}

}  // extern "C"
