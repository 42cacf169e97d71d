// Batched execution (see batch.hpp).
#include "batch.hpp"

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <tuple>
#include <utility>

namespace dfft {

namespace {

// A stage the batched kernels run: a register-resident C2C, R2C or C2R stage
// whose line length has a batched tile body.
bool batchable(const Op& op) {
  if (op.type != Op::Stage || !op.fast) return false;
  if (op.kind != dev::kC2C && op.kind != dev::kR2C && op.kind != dev::kC2R) return false;
  return dev::batch_stage_supported(op.sa.n);
}

// kind, inverse, a-fast rows, line length, two-line tiles: one batched launch
// per group
using GroupKey = std::tuple<int, bool, bool, int, bool>;

// complex64 C2C stages the one-tile launches would run two lines per thread
// (separable sides, pair-aligned: op.single_B is set) take the batched
// two-line tiles (which address positions by stride only)
bool pair_batchable(const Op& op, bool dbl) {
  return !dbl && op.kind == dev::kC2C && op.single_B != 0 && !op.sa.src_atab && !op.sa.dst_atab && dev::batch_pair_lines(op.sa.n, op.sa.load_afast != 0) > 0;
}

void ck(cudaError_t e) {
  if (e != cudaSuccess) fail(kErrCuda, std::string("batch stream fork / join: ") + cudaGetErrorString(e));
}

}  // namespace

Batch::Batch(std::vector<const Plan*> plans) : plans_(std::move(plans)) {
  if (plans_.empty()) fail(kErrInvalidArgument, "a batch needs at least one plan");
  std::set<const Plan*> seen;
  for (const Plan* p : plans_) {
    if (!p) fail(kErrInvalidArgument, "null plan in batch");
    if (!p->on_device()) fail(kErrInvalidArgument, "plan was created by dfft_plan_analyze and cannot execute");
    if (!seen.insert(p).second)
      fail(kErrInvalidArgument, "a plan appears twice in the batch (its scratch arrays would be shared)");
    if (p->desc().exec_mode != 0) fail(kErrInvalidArgument, "batched execution needs fused plans");
    if (p->is_rank_plan()) fail(kErrInvalidArgument, "batched execution needs plans over all ranks, not per-rank plans");
    for (bool fwd : {true, false})
      for (const Op& op : p->program(fwd))
        if (op.type != Op::Stage || op.chirp)
          fail(kErrInvalidArgument, "batched execution needs fused plans whose stages are all FFT stage kernels");
  }
  dbl_ = plans_[0]->desc().dbl;
  for (const Plan* p : plans_)
    if (p->desc().dbl != dbl_) fail(kErrInvalidArgument, "all plans of a batch must have the same precision");
  bool ok = cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming) == cudaSuccess;
  for (int i = 0; ok && i < kAux; ++i)
    ok = cudaStreamCreateWithFlags(&aux_[i], cudaStreamNonBlocking) == cudaSuccess &&
         cudaEventCreateWithFlags(&join_[i], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    release();
    fail(kErrCuda, "batch stream / event creation failed");
  }
}

Batch::~Batch() { release(); }

void Batch::release() {
  for (int i = 0; i < kAux; ++i) {
    if (aux_[i]) cudaStreamDestroy(aux_[i]);
    if (join_[i]) cudaEventDestroy(join_[i]);
    aux_[i] = nullptr;
    join_[i] = nullptr;
  }
  if (fork_) cudaEventDestroy(fork_);
  fork_ = nullptr;
}

std::size_t Batch::launches(bool forward) const {
  std::size_t nst = 0, n = 0;
  for (const Plan* p : plans_) nst = std::max(nst, p->program(forward).size());
  for (std::size_t s = 0; s < nst; ++s) {
    std::map<GroupKey, std::size_t> groups;
    for (const Plan* p : plans_) {
      const auto& prog = p->program(forward);
      if (s >= prog.size() || prog[s].tiles == 0) continue;
      const Op& op = prog[s];
      if (batchable(op))
        ++groups[GroupKey(op.kind, op.inverse, op.sa.load_afast != 0, op.sa.n, pair_batchable(op, dbl_))];
      else
        ++n;
    }
    for (auto& g : groups) n += (g.second + dev::kMaxBatchFields - 1) / dev::kMaxBatchFields;
  }
  return n;
}

// One group's launches of one stage, kMaxBatchFields fields each; the largest
// fields come first, so that a launch ends with small tiles.
void Batch::launch_group(const Group& g, cudaStream_t st) const {
  auto tiles_of = [](const dev::StageArgs& A) { return static_cast<long long>(A.tiles_b) * A.Eo0 * A.Eo1; };
  auto list = g.args;
  std::stable_sort(list.begin(), list.end(),
                   [&](const dev::StageArgs& x, const dev::StageArgs& y) { return tiles_of(x) > tiles_of(y); });
  for (std::size_t c = 0; c < list.size(); c += dev::kMaxBatchFields) {
    dev::BatchParams P;
    std::memset(&P, 0, sizeof(P));
    P.nfields = static_cast<int>(std::min<std::size_t>(dev::kMaxBatchFields, list.size() - c));
    P.prefix[0] = 0;
    for (int i = 0; i < P.nfields; ++i) {
      P.f[i] = list[c + i];
      const long long tiles = tiles_of(P.f[i]);
      if (tiles >= (1ll << 31)) fail(kErrUnsupported, "too many tiles in one field of a batch");
      P.prefix[i + 1] = P.prefix[i] + tiles;
    }
    const cudaError_t e = g.pair ? dev::launch_fft_batch_pair(P, g.inverse, g.afast, st)
                                 : dev::launch_fft_batch(P, dbl_, g.kind, g.inverse, g.afast, st);
    if (e != cudaSuccess) fail(kErrCuda, std::string("batched stage launch failed: ") + cudaGetErrorString(e));
  }
}

// whether the output of a field overlaps the input or output of a field of
// another group
bool Batch::shares_memory(const void* const* ins, void* const* outs, bool forward,
                          const std::vector<int>& group) const {
  struct Range {
    std::uintptr_t begin, end;
    int group;
    bool written;
  };
  std::vector<Range> r;
  for (std::size_t f = 0; f < plans_.size(); ++f) {
    const PlanDesc& d = plans_[f]->desc();
    const std::size_t real = dbl_ ? 8 : 4;
    const std::size_t in = total_size(d.gin) * real * (d.r2c ? 1 : 2), out = total_size(d.gout) * real * 2;
    const auto a = reinterpret_cast<std::uintptr_t>(ins[f]), b = reinterpret_cast<std::uintptr_t>(outs[f]);
    r.push_back(Range{a, a + (forward ? in : out), group[f], false});
    r.push_back(Range{b, b + (forward ? out : in), group[f], true});
  }
  std::sort(r.begin(), r.end(), [](const Range& x, const Range& y) { return x.begin < y.begin; });
  for (std::size_t i = 0; i < r.size(); ++i)
    for (std::size_t j = i + 1; j < r.size() && r[j].begin < r[i].end; ++j)
      if (r[i].group != r[j].group && (r[i].written || r[j].written)) return true;
  return false;
}

void Batch::execute(const void* const* ins, void* const* outs, bool forward, cudaStream_t st) const {
  if (!ins || !outs) fail(kErrInvalidArgument, "null buffer arrays");
  for (std::size_t f = 0; f < plans_.size(); ++f) plans_[f]->check_buffers(ins[f], outs[f], forward);
  std::size_t nst = 0;
  for (const Plan* p : plans_) nst = std::max(nst, p->program(forward).size());
  // the groups of every stage index, the stages that launch per field, and the
  // group each field is in (numbered by their first field)
  std::vector<std::vector<Group>> groups(nst);
  std::vector<std::vector<std::pair<std::size_t, dev::StageArgs>>> single(nst);  // (field, args)
  std::vector<std::vector<int>> member(nst);
  for (std::size_t s = 0; s < nst; ++s) {
    std::map<GroupKey, int> index;
    member[s].assign(plans_.size(), -1);
    for (std::size_t f = 0; f < plans_.size(); ++f) {
      const Plan* p = plans_[f];
      const auto& prog = p->program(forward);
      if (s >= prog.size()) continue;
      const Op& op = prog[s];
      if (op.tiles == 0) continue;
      dev::StageArgs A = op.sa;
      A.in = op.src == kBufIn ? const_cast<void*>(ins[f]) : op.src == kBufOut ? outs[f] : p->device_buffer(op.src);
      A.out = op.dst == kBufIn ? const_cast<void*>(ins[f]) : op.dst == kBufOut ? outs[f] : p->device_buffer(op.dst);
      if (!batchable(op)) {
        single[s].emplace_back(f, A);
        continue;
      }
      // the batched tile bodies: two lines per thread where the one-tile
      // launch could run them, else one line per thread group; lines per
      // tile fixed by the line length
      // (b-fast pairs move 16 bytes at a time: both buffers on 16-byte boundaries)
      const bool aligned = ((reinterpret_cast<std::uintptr_t>(A.in) | reinterpret_cast<std::uintptr_t>(A.out)) & 15) == 0;
      const bool pair = pair_batchable(op, dbl_) && (A.load_afast || aligned);
      A.pairs = 0;
      A.comp = 0;
      A.B = pair ? dev::batch_pair_lines(A.n, A.load_afast != 0) : dev::batch_stage_lines(dbl_, A.n);
      const int per = (op.kind == dev::kC2C) ? A.B : 2 * A.B;
      A.tiles_b = (A.Eb + per - 1) / per;
      const GroupKey key(op.kind, op.inverse, A.load_afast != 0, A.n, pair);
      auto it = index.find(key);
      if (it == index.end()) {
        it = index.emplace(key, static_cast<int>(groups[s].size())).first;
        groups[s].push_back(Group{op.kind, op.inverse, A.load_afast != 0, pair, {}});
      }
      groups[s][it->second].args.push_back(A);
      member[s][f] = it->second;
    }
  }
  // Fields that share a launch at one stage share it at every stage (cubic
  // fields), and none writes to memory that a field of another group uses: each
  // group's stages follow one another on a lane of their own, without waiting
  // for the other groups between stages.  Else the groups of one stage run
  // concurrently and join before the next, so that every input has been read
  // before the last stages write.
  bool chains = true;
  for (std::size_t s = 0; s < nst; ++s)
    chains = chains && single[s].empty() && member[s] == member[0];
  chains = chains && nst > 0 && !shares_memory(ins, outs, forward, member[0]);
  if (chains) {
    const int nl = static_cast<int>(groups[0].size());
    fork(st, nl);
    for (std::size_t s = 0; s < nst; ++s)
      for (int g = 0; g < nl; ++g) launch_group(groups[s][g], lane(st, g));
    join(st, nl);
    return;
  }
  for (std::size_t s = 0; s < nst; ++s) {
    for (auto& fa : single[s]) {
      const Plan* p = plans_[fa.first];
      const cudaError_t e = p->launch_op(p->program(forward)[s], fa.second, st);
      if (e != cudaSuccess) fail(kErrCuda, std::string("kernel launch failed: ") + cudaGetErrorString(e));
    }
    const int nl = static_cast<int>(groups[s].size());
    fork(st, nl);
    for (int g = 0; g < nl; ++g) launch_group(groups[s][g], lane(st, g));
    join(st, nl);
  }
}

void Batch::fork(cudaStream_t st, int lanes) const {
  if (lanes <= 1) return;
  ck(cudaEventRecord(fork_, st));
  for (int i = 0; i < std::min(lanes - 1, kAux); ++i) ck(cudaStreamWaitEvent(aux_[i], fork_, 0));
}

void Batch::join(cudaStream_t st, int lanes) const {
  if (lanes <= 1) return;
  for (int i = 0; i < std::min(lanes - 1, kAux); ++i) {
    ck(cudaEventRecord(join_[i], aux_[i]));
    ck(cudaStreamWaitEvent(st, join_[i], 0));
  }
}

}  // namespace dfft
