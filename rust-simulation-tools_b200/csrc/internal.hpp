// Internal host-side structures of librstg.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "rstg.h"

namespace rstg {

// Error carrying an rstg_status; converted to the C status at the ABI edge.
struct Error : std::runtime_error {
  rstg_status code;
  Error(rstg_status c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void set_last_error(const std::string& m);

#define RSTG_CUDA(expr)                                                                              \
  do {                                                                                               \
    cudaError_t e_ = (expr);                                                                         \
    if (e_ != cudaSuccess)                                                                           \
      throw ::rstg::Error(RSTG_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_));      \
  } while (0)

// AmberTopology (core/src/amber/prmtop.rs:34-105), host copy.
struct Topology {
  int64_t n_atoms = 0, n_residues = 0, n_types = 0;
  std::vector<std::string> atom_names, residue_labels;
  std::vector<int64_t> type_idx, residue_pointers;
  std::vector<double> charges, charges_amber, masses, radii, screen;
  std::vector<int64_t> bond_i, bond_j, bond_t;
  std::vector<double> bond_k, bond_req, angle_k, angle_teq, dih_pk, dih_pn, dih_phase;
  std::vector<int64_t> ang_i, ang_j, ang_k, ang_t;
  std::vector<int64_t> dih_i, dih_j, dih_k, dih_l, dih_t;
  std::vector<uint8_t> dih_ignore14;
  std::vector<int64_t> num_excluded, excluded_list;  // -1 = placeholder
  double scee = 1.2, scnb = 2.0;
  std::vector<double> lj_a, lj_b;
  std::vector<int64_t> nb_index;

  std::vector<int64_t> atom_residue_indices() const;
  std::vector<int64_t> select(const std::vector<int64_t>& residues) const;  // throws on range
};

Topology parse_prmtop(const std::string& path);
Topology extract_subtopology(const Topology& t, const std::vector<int64_t>& atoms);

// Non-bonded pair classes of one topology: the reference checks 1-4 first
// (scaled), then exclusion (skipped), else full (mm_energy.rs:230-252).
// Stored as sorted (i < j) key lists for O(log) host lookups.
struct PairClasses {
  std::vector<uint64_t> excl_keys, p14_keys;  // (i << 32) | j, sorted, unique
  static PairClasses build(const Topology& t);
  int cls(int64_t i, int64_t j) const;  // 0 skip, 1 full, 2 scaled 1-4
};

// The same classes as the plain kernels read them (mm_energy.rs:8-39): per atom
// i two words with a bit for each of the 64 atoms after it (excluded, 1-4),
// and per atom the pairs farther along, far_ptr[i] .. far_ptr[i + 1] into
// far, (j, class) each.
struct PairWindows {
  std::vector<uint64_t> win;  // [n][2]
  std::vector<int32_t> far_ptr, far;
  static PairWindows build(const Topology& t);
};

// The receptor/ligand split of binding.rs:142-211 / decomposition.rs:125-208.
struct Split {
  Topology complex, rec, lig;
  std::vector<int64_t> complex_atoms;  // topology atom of each complex atom
  std::vector<int64_t> rec_atoms, lig_atoms;  // complex numbering
  std::vector<int64_t> rec_res, lig_res;  // complex residue numbering
  static Split make(const Topology& t, const std::vector<int64_t>& rres, const std::vector<int64_t>& lres);
};

// Stream-ordered device buffer.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaStream_t s = nullptr;
  int device = 0;
  DevBuf() = default;
  DevBuf(size_t n, cudaStream_t st);
  ~DevBuf();
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes), s(o.s), device(o.device) { o.p = nullptr; }
  DevBuf& operator=(DevBuf&& o) noexcept;
  void give_back();
  template <class T>
  T* as() const {
    return (T*)p;
  }
};

// Two streams beside a context's own one and the events that order them.
struct SideStreams {
  cudaStream_t s[2] = {};
  cudaEvent_t fork = nullptr, join[2] = {};
  SideStreams();
  ~SideStreams() { release(); }
  void release();
  SideStreams(const SideStreams&) = delete;
  SideStreams& operator=(const SideStreams&) = delete;
};

struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::recursive_mutex mu;
  std::atomic<int64_t> launches{0};
  cudaDeviceProp prop{};
  std::mutex side_mu;
  std::vector<std::unique_ptr<SideStreams>> side_free;  // sets that no call holds (under side_mu)
  void bind() const { cudaSetDevice(device); }
};

// Side streams for independent parts of one call, held by that call alone:
// calls of one context run at the same time from several threads (systems in
// plain mode, a server's workers), and an event recorded anew by another call
// would unorder this one's kernels.  Where the caller owns the stream every part
// runs on it.  A call that throws between fork and join leaves no kernel running
// on memory that its buffers give back to the pool: declare the lease after them.
class SideLease {
 public:
  explicit SideLease(Ctx* c);
  ~SideLease();
  SideLease(const SideLease&) = delete;
  SideLease& operator=(const SideLease&) = delete;
  void fork();  // both streams after what the context's stream holds
  void join();  // the context's stream after both
  cudaStream_t operator[](int k) const { return set_ ? set_->s[k] : c_->stream; }

 private:
  Ctx* c_;
  int unwinding_;
  std::unique_ptr<SideStreams> set_;
};

// Records a kernel launch for the context's counter and checks the launch.
void launched(Ctx* c, int n = 1);

}  // namespace rstg

struct rstg_ctx : rstg::Ctx {};
struct rstg_topology : rstg::Topology {};
