// C ABI and host orchestration of the B200 descriptor / GAP path.
//
// Host objects mirror the reference's: a calculator owns its hypers and the
// radial spline (calculator_spherical_expansion.hh:1019-1156), a structure set
// owns the structures, their neighbour list and the computed features
// (ManagerCollection + Properties, structure_manager_collection.hh), a GAP
// model owns the sparse points and weights (models/krr.py, sparse_points.hh).
// Every device buffer is owned by one of these handles and reused across
// calls; kernels run on the structure set's stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <map>
#include <memory>
#include <set>
#include <string>
#include <vector>

#include "common.cuh"
#include "json_lite.h"

namespace rgpu {
int64_t launches(bool reset);
}  // namespace rgpu

using namespace rgpu;

namespace {

thread_local std::string t_err;
thread_local int t_kind = RGPU_EXC_NONE;

int fail(const Error & e) {
  t_err = e.what();
  t_kind = e.kind;
  return e.code;
}

template <class F>
int guard(F && f) {
  try {
    t_err.clear();
    t_kind = RGPU_EXC_NONE;
    f();
    return RGPU_OK;
  } catch (const Error & e) {
    return fail(e);
  } catch (const std::bad_alloc &) {
    return fail(Error(RGPU_ERR_CUDA, "host allocation failed"));
  } catch (const std::exception & e) {
    return fail(Error(RGPU_ERR_INVALID_ARGUMENT, e.what()));
  }
}

const double kPi = 3.14159265358979323846264338327950288;

}  // namespace

// ------------------------------------------------------------------- hypers
namespace rgpu {
void parse_hypers(const std::string & kind, const std::string & text, Hypers & h) {
  Json j = Json::parse(text);
  if (j.type != Json::Object) throw Error(RGPU_ERR_INVALID_ARGUMENT, "hypers must be a JSON object");
  h.kind = kind;
  if (kind != "sphericalinvariants" && kind != "sphericalexpansion")
    throw Error(RGPU_ERR_INVALID_ARGUMENT,
                "The representations factory " + kind +
                    " has not been registered. The available combinations are: "
                    "['sphericalexpansion', 'sphericalinvariants']");
  h.max_radial = j.at("max_radial").as_int();
  h.max_angular = j.at("max_angular").as_int();
  if (h.max_radial < 1) throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_radial must be >= 1");
  if (h.max_angular < 0 || h.max_angular > kMaxL)
    throw Error(RGPU_ERR_INVALID_ARGUMENT, "max_angular must be in [0, 12] on the GPU path");
  h.compute_gradients = j.has("compute_gradients") ? j.at("compute_gradients").as_bool() : false;
  if (kind == "sphericalinvariants") {
    h.normalize = j.at("normalize").as_bool();
    h.soap_type = j.at("soap_type").as_string();
    if (h.soap_type != "PowerSpectrum") {
      if (h.soap_type == "RadialSpectrum" || h.soap_type == "BiSpectrum")
        throw Error(RGPU_ERR_INVALID_ARGUMENT,
                    "Requested SphericalInvariants type '" + h.soap_type +
                        "' is not on the B200 path. Supported: 'PowerSpectrum'.");
      throw Error(RGPU_ERR_INVALID_ARGUMENT,
                  "Requested SphericalInvariants type '" + h.soap_type +
                      "' has not been implemented.  Must be one of: 'PowerSpectrum', "
                      "'RadialSpectrum', or 'BiSpectrum'.");
    }
    if (j.has("coefficient_subselection"))
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "coefficient_subselection is not on the B200 path");
  }
  if (j.has("expansion_by_species_method")) {
    std::string m = j.at("expansion_by_species_method").as_string();
    if (m != "environment wise" && m != "user defined" && m != "structure wise")
      throw Error(RGPU_ERR_INVALID_ARGUMENT,
                  "expansion_by_species_method provided:'" + m +
                      "' is not part of the implemented methods: 'environment wise', "
                      "'structure wise', 'user defined', ");
  }
  const Json & fc = j.at("cutoff_function");
  std::string fct = fc.at("type").as_string();
  if (fct != "ShiftedCosine" && fct != "RadialScaling")
    throw Error(RGPU_ERR_INVALID_ARGUMENT,
                "Requested cutoff function type '" + fct + "' is not on the B200 path. Supported: "
                                                          "'ShiftedCosine', 'RadialScaling'.");
  h.cutoff = fc.at("cutoff").at("value").as_number();
  h.smooth_width = fc.at("smooth_width").at("value").as_number();
  h.radial_scaling = fct == "RadialScaling";
  if (h.radial_scaling) {
    // representations/cutoff_functions.hh:243-253
    h.rs_rate = fc.at("rate").at("value").as_number();
    if (h.rs_rate < 0) throw Error(RGPU_ERR_INVALID_ARGUMENT, "RadialScaling's rate should be positive");
    h.rs_exponent = fc.at("exponent").at("value").as_number();
    h.rs_scale = fc.at("scale").at("value").as_number();
  }
  const Json & gd = j.at("gaussian_density");
  std::string gt = gd.at("type").as_string();
  if (gt != "Constant")
    throw Error(RGPU_ERR_INVALID_ARGUMENT,
                "Requested Smearing type '" + gt + "' has not been implemented.  Must be one of: 'Constant'.");
  h.sigma = gd.at("gaussian_sigma").at("value").as_number();
  const Json & rc = j.at("radial_contribution");
  std::string rt = rc.at("type").as_string();
  if (rt != "GTO")
    throw Error(RGPU_ERR_INVALID_ARGUMENT,
                "Requested Radial contribution type '" + rt + "' is not on the B200 path. Supported: 'GTO'.");
  h.spline = false;
  h.spline_accuracy = 1e-13;  // direct 1F1 evaluation is served by a spline this fine
  if (rc.has("optimization")) {
    const Json & o = rc.at("optimization");
    if (o.has("RadialDimReduction"))
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "RadialDimReduction is not on the B200 path");
    if (o.has("Spline")) {
      h.spline = true;
      const Json & sp = o.at("Spline");
      if (!sp.has("accuracy")) throw Error(RGPU_ERR_INVALID_ARGUMENT, "No Spline accuracy was given.");
      h.spline_accuracy = sp.at("accuracy").as_number();
      if (!(h.spline_accuracy > 0)) throw Error(RGPU_ERR_INVALID_ARGUMENT, "Error bound must be > 0");
    }
  }
  if (!(h.cutoff > 0)) throw Error(RGPU_ERR_INVALID_ARGUMENT, "cutoff must be > 0");
  h.name = kind + "_" + j.dump();
}
}  // namespace rgpu

// ------------------------------------------------------------------ handles
// What a structure set keeps of a calculator or model (features, recorded
// calls) is tied to its serial number: an address may be that of a later
// object, whose buffers may lie where the former's did.
static uint64_t next_serial() {
  static std::atomic<uint64_t> n{0};
  return ++n;
}
template <class Handle>
static uint64_t serial_of(const Handle * h) {
  return h ? h->serial : 0;
}

struct rgpu_calculator {
  const uint64_t serial{next_serial()};
  int device{-1};  // device of the uploaded tables (-1: not uploaded yet)
  Hypers hy;
  RadialSpline spline;
  DevBuf grid, y, y2h, q4f, center;
  SplineDev dev{};
};

// A part of a device buffer.
struct DevView {
  void * p{nullptr};
  size_t bytes{0};
  template <class T>
  T * as() const {
    return static_cast<T *>(p);
  }
};

// Status words of a handle's kernels, copied to the host together.
struct HandleStatus {
  DevStatus nl;  // neighbour list
  int tc[2];     // bounded waits of the tcgen05 kernels: gave up, stage
  int pad[2];
};

struct GapLayout;

// One FP32 prediction (rgpu_gap_predict / rgpu_gap_predict_stress) recorded
// as a CUDA graph: the device buffers it was recorded with, and a neighbour
// list built to capacities 12.5 % above the counts of the recording call.
struct PredictGraph {
  cudaGraph_t graph{nullptr};
  cudaGraphExec_t exec{nullptr};
  NlCaps caps{};
  std::vector<const void *> buffers;
  double * out_h{nullptr};  // pinned: energies, forces, stress sums of a replay
  int64_t kernels{0};
};

// The recordings of one size: the same model, output kind, numbers of
// structures and atoms, species layout and centres per species. Energies
// alone skip the force half and have a recording of their own beside the full
// one, so that calls of both kinds in turn over a few sizes find their
// recordings: with a place for each they pushed one another out from three
// sizes on (energies, then forces, of about 3 000 clusters: 14.3 ms instead of
// 4.1).
struct PredictBucket {
  uint64_t model{0};  // serial
  bool stress{false}, outputs{false};
  int n_struct{0};
  int64_t n_atoms{0};
  std::vector<int> species;
  std::vector<int64_t> species_count;
  PredictGraph full, alone;
  int energies_alone{0};  // calls for energies alone that had no recording of their own
  uint64_t used{0};
};
constexpr size_t kMaxBuckets = 4;

struct rgpu_structures {
  int device{-1};  // device current at creation: owns the stream and every buffer
  cudaStream_t st{nullptr};
  int n_struct{0};
  int64_t n_atoms{0};
  std::vector<int64_t> atom_off;
  std::vector<int32_t> types;
  std::vector<double> cells_h;  // [n_struct][9], lattice vectors as rows
  std::vector<uint8_t> mask;
  bool has_mask{false};
  std::vector<int64_t> center_off_h;
  DevBuf in_d;  // every input array, one after the other
  DevView atom_off_d, pos_d, types_d, cells_d, pbc_d, tag2idx_d, ncent_d, center_off_d, atom_struct_d;
  // staging (pinned) for host inputs
  void * pinned{nullptr};
  size_t pinned_cap{0};
  // neighbour list
  bool nl_valid{false};
  double nl_cutoff{-1};
  NlWork nlw;
  NlOutputs nl;
  int64_t exact_pairs{0};  // pairs of the last list built with synchronisation (nl.n_pairs may be a capacity)
  std::vector<int64_t> pair_off_h;  // host copy of nl.pair_off, made on demand
  bool pair_off_h_valid{false};
  std::vector<int> batch_species;   // sorted atom types present in the batch
  int64_t centres_of_type[130]{};   // centres per atom type (the mask applied)
  // layout and features
  std::vector<int> species;  // dense layout (sorted)
  DevBuf lut;
  FeatureDims fd{};
  std::vector<int64_t> species_count;
  DevBuf row_of_center, center_of_row, sort_tmp, present, tile_mask;
  DevBuf C64, X64, invn64, dC64, C32, X32, xscale32;  // xscale32[row] = 1/|p| (FP32 path)
  int feat_precision{-1};
  uint64_t feat_calc{0};  // serial
  bool feat_gradients{false};
  bool feat_valid{false};
  // GAP work
  DevBuf out_d;  // energies, forces, stress sums, one after the other
  DevBuf K64, t64, erow64, Wh, Wl, dX32, dC32, epart, Xh, Xl, chunk_map;
  int chunk_map_of[3]{0, 0, 0};  // the (S, n, L) that chunk_map holds
  bool feat_x32{false};  // FP32 features also kept unsplit (for export)
  DevBuf dCp, dCs, dXp;
  DevBuf export_d;               // rows of rgpu_get_features on their way out
  DevBuf knm, plist, Tq;  // sparse kernel matrices for training
  // MD step recorded as a CUDA graph (rgpu_md_step)
  cudaGraph_t md_graph{nullptr};
  cudaGraphExec_t md_exec{nullptr};
  uint64_t md_model{0};  // serial
  bool md_stress{false};
  NlCaps md_caps{};
  std::vector<const void *> md_buffers;  // device buffer addresses at recording
  std::vector<int> md_species;
  int64_t md_replays{0};       // replays since the graph was recorded
  int64_t md_kernels{0};       // kernel nodes of the recorded graph
  int64_t md_reason{0};        // why the last step did not replay: 0 none (first step or no
                               // recording), 1 a buffer moved, 3 model or layout, 100 + status
  bool md_no_graph{false};     // recording failed once: ordinary path only
  double * md_pos_h{nullptr};  // pinned: positions in, outputs out
  double * md_out_h{nullptr};
  size_t md_pos_cap{0}, md_out_cap{0};
  // FP32 predictions recorded as CUDA graphs, a few size buckets per handle
  std::vector<PredictBucket> pbuckets;
  bool use_graphs{true};
  uint64_t pgraph_clock{0};
  int64_t pgraph_replays{0}, pgraph_records{0}, pgraph_last_kernels{0};
  // autograd: the serial of the model whose forward (rgpu_gap_forward_dev)
  // left W, the features and the list in place for rgpu_gap_backward_dev (0:
  // none)
  uint64_t fwd_model{0};
  DevBuf y0_d;  // per-structure energy baseline of fwd_model
  // status and timing
  HandleStatus * status_d{nullptr};
  HandleStatus * status_h{nullptr};
  double * E() const { return out_d.as<double>(); }
  double * F() const { return E() + n_struct; }
  double * S() const { return F() + 3 * n_atoms; }
  cudaEvent_t ev[10]{};
  double stage_ms[10]{};
  bool timed{false};
};

struct rgpu_gap_model {
  const uint64_t serial{next_serial()};
  int device{-1};  // device of the model's buffers (-1: none allocated yet)
  rgpu_calculator * calc{nullptr};
  std::vector<int> species;  // model layout species (sorted)
  int M{0};
  std::vector<int32_t> sp_species;
  std::vector<double> T;  // M x D_model
  std::vector<double> alpha;
  int zeta{2};
  std::vector<double> self_contrib;  // per model species
  // device copies for a batch layout
  std::vector<int> layout_species;
  int layout_D{0};
  std::vector<GapSpecies> segs;  // per batch species
  DevBuf T64, alpha64, Th, Tl, Tth, Ttl, alpha32;
  std::vector<int64_t> tt_off;  // per batch species offset into Tt32
  DevBuf ucol;                  // caller's index of each sparse point in layout order
  std::vector<double> T_layout, alpha_layout;  // host copies in the batch layout
  int64_t tt_total{0};
  bool layout_bf16{false};
};

namespace {

// Runs the rest of a call on a structure set's device and gives the caller
// back the device that was current before. A structure set belongs to the
// device that was current when it was created (its stream and buffers live
// there), so a call made while another device is current still works on its
// own device's memory.
struct OnDevice {
  int prev{-1};
  explicit OnDevice(const rgpu_structures * s) {
    if (!s || s->device < 0) return;
    int cur = 0;
    RGPU_CUDA(cudaGetDevice(&cur));
    if (cur != s->device) {
      RGPU_CUDA(cudaSetDevice(s->device));
      prev = cur;
    }
  }
  ~OnDevice() {
    if (prev >= 0) cudaSetDevice(prev);
  }
  OnDevice(const OnDevice &) = delete;
  OnDevice & operator=(const OnDevice &) = delete;
};

// Ties a calculator or model to the current device on its first device
// allocation, and rejects later use with a structure set of another device
// (its buffers would be another GPU's memory).
void bind_device(int & owner, const char * what) {
  const int dev = current_device();
  if (owner < 0) {
    owner = dev;
  } else if (owner != dev) {
    throw Error(RGPU_ERR_INVALID_ARGUMENT, std::string(what) + " lives on device " + std::to_string(owner) +
                                               " and cannot be used with a structure set of device " +
                                               std::to_string(dev));
  }
}

void ensure_stream(rgpu_structures * s) {
  if (!s->st) {
    s->device = current_device();
    RGPU_CUDA(cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking));
    RGPU_CUDA(cudaMalloc(&s->status_d, sizeof(HandleStatus)));
    RGPU_CUDA(cudaMemset(s->status_d, 0, sizeof(HandleStatus)));
    RGPU_CUDA(cudaMallocHost(&s->status_h, sizeof(HandleStatus)));
    *s->status_h = HandleStatus{};
    for (auto & e : s->ev) RGPU_CUDA(cudaEventCreate(&e));
  }
}

void * staging(rgpu_structures * s, size_t bytes) {
  if (bytes > s->pinned_cap) {
    if (s->pinned) {
      RGPU_CUDA(cudaStreamSynchronize(s->st));  // no copy in flight may still use it
      cudaFreeHost(s->pinned);
    }
    s->pinned = nullptr;
    RGPU_CUDA(cudaMallocHost(&s->pinned, bytes));
    s->pinned_cap = bytes;
  }
  return s->pinned;
}

// Host -> device through the pinned staging buffer, in order on the stream.
void upload(rgpu_structures * s, DevBuf & dst, const void * src, size_t bytes) {
  dst.ensure(bytes);
  if (bytes == 0) return;
  RGPU_CUDA(cudaStreamSynchronize(s->st));  // staging buffer reuse
  void * p = staging(s, bytes);
  std::memcpy(p, src, bytes);
  RGPU_CUDA(cudaMemcpyAsync(dst.p, p, bytes, cudaMemcpyHostToDevice, s->st));
}

// The input arrays of a structure set through the staging buffer in one copy
// into one device buffer, each view on a 256-byte boundary.
struct Upload {
  DevView * dst;
  const void * src;
  size_t bytes;
};
void upload_inputs(rgpu_structures * s, const std::vector<Upload> & ups) {
  size_t total = 0;
  for (const Upload & u : ups) total += (u.bytes + 255) & ~size_t(255);
  s->in_d.ensure(std::max<size_t>(total, 256));
  RGPU_CUDA(cudaStreamSynchronize(s->st));  // staging buffer reuse
  unsigned char * base = static_cast<unsigned char *>(staging(s, std::max<size_t>(total, 256)));
  size_t off = 0;
  for (const Upload & u : ups) {
    u.dst->p = s->in_d.as<unsigned char>() + off;
    u.dst->bytes = u.bytes;
    if (u.bytes) std::memcpy(base + off, u.src, u.bytes);
    off += (u.bytes + 255) & ~size_t(255);
  }
  if (total) RGPU_CUDA(cudaMemcpyAsync(s->in_d.p, base, total, cudaMemcpyHostToDevice, s->st));
}

// New positions into their place.
void upload_positions(rgpu_structures * s, const double * positions) {
  const size_t bytes = sizeof(double) * 3 * size_t(s->n_atoms);
  if (bytes == 0) return;
  if (bytes > s->pos_d.bytes) throw Error(RGPU_ERR_INVALID_ARGUMENT, "the structures have not been uploaded");
  RGPU_CUDA(cudaStreamSynchronize(s->st));  // staging buffer reuse
  void * p = staging(s, bytes);
  std::memcpy(p, positions, bytes);
  RGPU_CUDA(cudaMemcpyAsync(s->pos_d.p, p, bytes, cudaMemcpyHostToDevice, s->st));
}

// The outputs' buffer, and zeros in the energies and what else is asked for.
void zero_outputs(rgpu_structures * s, bool forces, bool stress) {
  s->out_d.ensure(sizeof(double) * (7 * size_t(s->n_struct) + 3 * size_t(s->n_atoms) + 1));
  const size_t n = stress ? size_t(s->S() - s->E()) + 6 * size_t(s->n_struct)
                          : size_t(s->n_struct) + (forces ? 3 * size_t(s->n_atoms) : 0);
  if (n) RGPU_CUDA(cudaMemsetAsync(s->E(), 0, sizeof(double) * n, s->st));
}

// The handle's status words to the host, in order on the stream, and what a
// call that has waited for them makes of a tcgen05 wait that gave up.
void fetch_status(rgpu_structures * s) {
  RGPU_CUDA(cudaMemcpyAsync(s->status_h, s->status_d, sizeof(HandleStatus), cudaMemcpyDeviceToHost, s->st));
}
bool timed_out(rgpu_structures * s, int * where = nullptr) {
  if (!s->status_h->tc[0]) return false;
  if (where) *where = s->status_h->tc[1];
  RGPU_CUDA(cudaMemsetAsync(s->status_d->tc, 0, sizeof(s->status_d->tc), s->st));
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  s->status_h->tc[0] = s->status_h->tc[1] = 0;
  return true;
}
void check_timeout(rgpu_structures * s) {
  int where = 0;
  if (timed_out(s, &where))
    throw Error(RGPU_ERR_TIMEOUT, "tensor-core GEMM: a bounded pipeline wait gave up (stage " +
                                      std::to_string(where) + ")");
}
// Clears the status words after a replay whose results were dropped.
void reset_status(rgpu_structures * s) {
  RGPU_CUDA(cudaMemsetAsync(s->status_d, 0, sizeof(HandleStatus), s->st));
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  *s->status_h = HandleStatus{};
}

// Nothing computed so far is reused by a later call: the list, the features
// and what a forward left for its backward.
void drop_results(rgpu_structures * s) {
  s->nl_valid = false;
  s->feat_valid = false;
  s->fwd_model = 0;
}

void mark(rgpu_structures * s, int i) {
  if (s->timed) RGPU_CUDA(cudaEventRecord(s->ev[i], s->st));
}

FeatureDims make_dims(const Hypers & hy, int S) {
  FeatureDims f;
  f.S = S;
  f.n = hy.max_radial;
  f.L = hy.max_angular;
  f.K = (f.L + 1) * (f.L + 1);
  f.W = f.n * (f.L + 1);
  f.nK = f.n * f.K;
  f.P = S * (S + 1) / 2;
  f.D = f.P * f.n * f.n * (f.L + 1);
  f.Dpad = (f.D + 31) / 32 * 32;
  f.Sn = S * f.n;
  if (f.n % 2 == 0) {  // row pairs never straddle two species
    f.G = S;
    f.npg = f.n / 2;
  } else {
    f.G = 1;
    f.npg = (f.Sn + 1) / 2;
  }
  f.TD = f.npg * (f.npg + 1) / 2;
  f.TO = f.npg * f.npg;
  f.lenD = (4 * (f.L + 1) * f.TD + 31) / 32 * 32;
  f.lenO = (4 * (f.L + 1) * f.TO + 31) / 32 * 32;
  f.Dg = f.G * f.lenD + f.G * (f.G - 1) / 2 * f.lenO;
  return f;
}

// Choose the dense species layout: batch species plus `extra`.
void set_layout(rgpu_structures * s, const Hypers & hy, const std::vector<int> & extra) {
  std::set<int> sp(s->batch_species.begin(), s->batch_species.end());
  sp.insert(extra.begin(), extra.end());
  std::vector<int> species(sp.begin(), sp.end());
  if (int(species.size()) > kMaxSpecies)
    throw Error(RGPU_ERR_INVALID_ARGUMENT, "more than 16 species in one batch is not supported on the GPU");
  FeatureDims fd = make_dims(hy, int(species.size()));
  bool same = species == s->species && fd.n == s->fd.n && fd.L == s->fd.L;
  s->fd = fd;
  if (same) return;
  s->species = species;
  std::vector<int8_t> lut(130, -1);
  for (size_t i = 0; i < species.size(); ++i) lut[species[i]] = int8_t(i);
  upload(s, s->lut, lut.data(), lut.size());
  s->feat_valid = false;
}

void build_nl(rgpu_structures * s, double cutoff) {
  if (s->nl_valid && s->nl_cutoff == cutoff) return;
  s->fwd_model = 0;
  NlInputs in;
  in.n_struct = s->n_struct;
  in.n_atoms = s->n_atoms;
  in.atom_off = s->atom_off_d.as<int64_t>();
  in.pos = s->pos_d.as<double>();
  in.types = s->types_d.as<int32_t>();
  in.cells = s->cells_d.as<double>();
  in.pbc = s->pbc_d.as<int32_t>();
  in.tag2idx = s->has_mask ? s->tag2idx_d.as<int32_t>() : nullptr;
  in.n_centers = s->ncent_d.as<int32_t>();
  in.center_off = s->center_off_d.as<int64_t>();
  in.atom_struct = s->atom_struct_d.as<int32_t>();
  in.n_centers_total = s->center_off_h[s->n_struct];
  build_neighbour_list(in, cutoff, s->nlw, s->nl, &s->status_d->nl, &s->status_h->nl, s->st);
  s->exact_pairs = s->nl.n_pairs;
  s->pair_off_h_valid = false;
  s->nl_valid = true;
  s->nl_cutoff = cutoff;
  s->feat_valid = false;
}

// Host copy of the neighbour list's centre offsets (for chunking the plain
// path's gradient passes).
const std::vector<int64_t> & pair_offsets_host(rgpu_structures * s) {
  if (!s->pair_off_h_valid) {
    s->pair_off_h.resize(s->nl.n_centers + 1);
    RGPU_CUDA(cudaMemcpyAsync(s->pair_off_h.data(), s->nl.pair_off, sizeof(int64_t) * (s->nl.n_centers + 1),
                              cudaMemcpyDeviceToHost, s->st));
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    s->pair_off_h_valid = true;
  }
  return s->pair_off_h;
}

ExpansionArgs exp_args(const rgpu_calculator * c, const rgpu_structures * s) {
  ExpansionArgs a;
  a.fd = s->fd;
  a.sp = c->dev;
  a.center_contrib = c->center.as<double>();
  a.species_lut = s->lut.as<int8_t>();
  a.rc = c->hy.cutoff;
  a.sw = c->hy.smooth_width;
  a.rs.on = c->hy.radial_scaling ? 1 : 0;
  a.rs.rate = c->hy.rs_rate;
  a.rs.exponent = c->hy.rs_exponent;
  a.rs.scale = c->hy.rs_scale;
  a.n_centers = s->nl.n_centers;
  a.n_pairs = s->exact_pairs;
  a.center_atom = s->nl.center_atom;
  a.pair_off = s->nl.pair_off;
  a.pair_j = s->nl.pair_j;
  a.pair_dist = s->nl.pair_dist;
  a.pair_dir = s->nl.pair_dir;
  a.types = s->types_d.as<int32_t>();
  return a;
}

// Rows and 128-row tiles of each central species (rows in species order).
TileMaskArgs tile_mask_args(const rgpu_structures * s) {
  TileMaskArgs a{};
  a.S = s->fd.S;
  int64_t r = 0, t = 0;
  for (int sI = 0; sI < s->fd.S; ++sI) {
    a.row0[sI] = r;
    a.rows[sI] = s->species_count[sI];
    a.tile_off[sI] = t;
    r += s->species_count[sI];
    t += (s->species_count[sI] + 127) / 128;
  }
  a.tile_off[s->fd.S] = t;
  return a;
}

// Row order of X: grouped by central species. The FP32 path's layouts of more
// than one segment group are sorted by the presence masks as well, after the
// expansion that writes them (sort_rows_by_mask), so they skip this.
void sort_rows(rgpu_structures * s, bool by_mask) {
  const int64_t nc = s->nl.n_centers;
  s->row_of_center.ensure(sizeof(int32_t) * (nc + 1));
  s->center_of_row.ensure(sizeof(int32_t) * (nc + 1));
  if (!by_mask)
    launch_species_sort(nc, s->types_d.as<int32_t>(), s->nl.center_atom, s->lut.as<int8_t>(), s->fd.S,
                        s->row_of_center.as<int32_t>(), s->center_of_row.as<int32_t>(), s->sort_tmp, s->st);
  // the counts per central species are known on the host since the upload
  s->species_count.assign(s->fd.S, 0);
  for (int sI = 0; sI < s->fd.S; ++sI) s->species_count[sI] = s->centres_of_type[s->species[sI]];
}

bool sorts_by_mask(const rgpu_calculator * c, const rgpu_structures * s) {
  return c->hy.kind == "sphericalinvariants" && s->fd.G > 1;
}

// Rows of one species ordered by their neighbour species, so that the GEMM
// tiles of the packed layout's species segments can skip what none of their
// rows holds; and the species present in each 128-row tile.
void sort_rows_by_mask(rgpu_structures * s) {
  const TileMaskArgs tm = tile_mask_args(s);
  s->tile_mask.ensure(sizeof(uint32_t) * size_t(std::max<int64_t>(tm.tile_off[s->fd.S], 1)) + 64);
  launch_mask_sort(s->nl.n_centers, s->types_d.as<int32_t>(), s->nl.center_atom, s->lut.as<int8_t>(),
                   s->present.as<uint32_t>(), s->fd.S, tm, s->row_of_center.as<int32_t>(),
                   s->center_of_row.as<int32_t>(), s->tile_mask.as<uint32_t>(), s->sort_tmp, s->st);
}

void compute_features(rgpu_calculator * c, rgpu_structures * s, int precision, bool grads,
                      const std::vector<int> & extra_species, bool need_x32 = true) {
  build_nl(s, c->hy.cutoff);
  set_layout(s, c->hy, extra_species);
  if (s->feat_valid && s->feat_calc == c->serial && s->feat_precision == precision &&
      (precision == RGPU_PRECISION_FP64 || s->feat_x32 || !need_x32)) {
    s->feat_gradients = s->feat_gradients || grads;
    return;
  }
  s->fwd_model = 0;
  mark(s, 2);
  const bool by_mask = precision == RGPU_PRECISION_FP32 && sorts_by_mask(c, s);
  sort_rows(s, by_mask);
  const int64_t nc = s->nl.n_centers;
  const FeatureDims & fd = s->fd;
  ExpansionArgs ea = exp_args(c, s);
  s->present.ensure(sizeof(uint32_t) * (nc + 1));
  PsArgs pa;
  pa.fd = fd;
  pa.n_centers = nc;
  pa.normalize = c->hy.normalize;
  pa.row_of_center = s->row_of_center.as<int32_t>();
  if (precision == RGPU_PRECISION_FP64) {
    s->C64.ensure(sizeof(double) * size_t(nc) * fd.S * fd.nK + 64);
    launch_expansion_fp64(ea, s->C64.as<double>(), s->present.as<uint32_t>(), s->st);
    mark(s, 3);
    if (c->hy.kind == "sphericalinvariants") {
      s->X64.ensure(sizeof(double) * size_t(nc) * fd.Dpad + 64);
      s->invn64.ensure(sizeof(double) * (nc + 1));
      launch_ps_fwd_fp64(pa, s->C64.as<double>(), s->X64.as<double>(), s->invn64.as<double>(), s->st);
    }
  } else {
    s->C32.ensure(sizeof(float) * size_t(nc) * fd.S * fd.n * row_stride(fd.L) + 64);
    launch_expansion_fp32(ea, s->C32.as<float>(), s->present.as<uint32_t>(), s->st);
    if (by_mask) sort_rows_by_mask(s);
    mark(s, 3);
    if (c->hy.kind == "sphericalinvariants") {
      if (need_x32) s->X32.ensure(sizeof(float) * size_t(nc) * fd.Dg + 64);
      s->Xh.ensure(sizeof(uint16_t) * size_t(nc) * fd.Dg + 64);
      s->Xl.ensure(sizeof(uint16_t) * size_t(nc) * fd.Dg + 64);
      s->xscale32.ensure(sizeof(float) * (nc + 1));
      pa.present = s->present.as<uint32_t>();
      pa.tc_status = s->status_d->tc;
      launch_ps_fwd_fast(pa, s->C32.as<float>(), need_x32 ? s->X32.as<float>() : nullptr,
                         s->Xh.as<__nv_bfloat16>(), s->Xl.as<__nv_bfloat16>(), s->xscale32.as<float>(), s->st);
    }
    s->feat_x32 = need_x32;
  }
  s->feat_valid = true;
  s->feat_calc = c->serial;
  s->feat_precision = precision;
  s->feat_gradients = grads;
}

// Keys present in the batch, as the reference's union of per-centre keys.
std::vector<std::pair<int, int>> present_keys(const rgpu_calculator * c, const rgpu_structures * s) {
  const int64_t nc = s->nl.n_centers;
  std::vector<uint32_t> pres(nc);
  RGPU_CUDA(cudaMemcpyAsync(pres.data(), s->present.p, sizeof(uint32_t) * nc, cudaMemcpyDeviceToHost, s->st));
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  std::set<uint32_t> masks(pres.begin(), pres.end());
  std::set<std::pair<int, int>> keys;
  for (uint32_t m : masks) {
    for (int a = 0; a < s->fd.S; ++a) {
      if (!(m >> a & 1)) continue;
      if (c->hy.kind == "sphericalexpansion") {
        keys.insert({s->species[a], s->species[a]});
        continue;
      }
      for (int b = a; b < s->fd.S; ++b)
        if (m >> b & 1) keys.insert({s->species[a], s->species[b]});
    }
  }
  return std::vector<std::pair<int, int>>(keys.begin(), keys.end());
}

// Column blocks of the dense layout for the requested keys (-1 = absent).
std::vector<int> key_blocks(const rgpu_calculator * c, const rgpu_structures * s, int n_keys,
                            const int32_t * keys) {
  std::vector<int> blocks(n_keys, -1);
  std::map<int, int> sidx;
  for (int i = 0; i < s->fd.S; ++i) sidx[s->species[i]] = i;
  std::map<std::pair<int, int>, int> kid;
  int k = 0;
  for (int a = 0; a < s->fd.S; ++a)
    for (int b = a; b < s->fd.S; ++b) kid[{a, b}] = k++;
  for (int i = 0; i < n_keys; ++i) {
    int ka = keys[2 * i], kb = keys[2 * i + 1];
    if (!sidx.count(ka)) continue;
    if (c->hy.kind == "sphericalexpansion") {
      blocks[i] = sidx[ka];
      continue;
    }
    if (!sidx.count(kb)) continue;
    int a = sidx[ka], b = sidx[kb];
    if (a > b) std::swap(a, b);
    blocks[i] = kid[{a, b}];
  }
  return blocks;
}

// Dense expansion gradients (property_block_sparse.hh:961-987): 3 rows per
// pair (x, y, z), key blocks of n*K. A pair's gradient has the key of its
// neighbour's species only; the self pair's has every species
// (calculator_spherical_expansion.hh:2327-2366).
void export_expansion_gradient(const rgpu_calculator * calc, rgpu_structures * s, int n_keys,
                               const std::vector<int> & blocks, double * out) {
  const FeatureDims & fd = s->fd;
  const int64_t nc = s->nl.n_centers;
  const int inner = fd.nK;
  ExpansionArgs ea = exp_args(calc, s);
  const std::vector<int64_t> & poff = pair_offsets_host(s);
  const size_t per_pair = sizeof(double) * 3 * size_t(fd.nK);
  const size_t per_center = sizeof(double) * size_t(fd.S) * 3 * fd.nK;
  const size_t budget = size_t(4) << 30;
  std::map<int, int> sidx;
  for (int i = 0; i < fd.S; ++i) sidx[s->species[i]] = i;
  std::vector<double> hp, hs;
  std::vector<int32_t> pj;
  int64_t c0 = 0;
  while (c0 < nc) {
    int64_t c1 = c0;
    size_t bytes = 0;
    while (c1 < nc) {
      size_t add = per_pair * size_t(poff[c1 + 1] - poff[c1]) + per_center;
      if (c1 > c0 && bytes + add > budget) break;
      bytes += add;
      ++c1;
    }
    const int64_t p_base = poff[c0];
    const int64_t np = poff[c1] - p_base;
    s->dCp.ensure(per_pair * size_t(np) + 64);
    s->dCs.ensure(per_center * size_t(c1 - c0) + 64);
    launch_expansion_grad_fp64(ea, c0, c1, p_base, s->dCp.as<double>(), s->st);
    launch_expansion_selfgrad_fp64(ea, c0, c1, p_base, s->dCp.as<double>(), s->dCs.as<double>(), s->st);
    hp.resize(size_t(np) * 3 * fd.nK);
    hs.resize(size_t(c1 - c0) * fd.S * 3 * fd.nK);
    pj.resize(size_t(np));
    RGPU_CUDA(cudaMemcpyAsync(hp.data(), s->dCp.p, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, s->st));
    RGPU_CUDA(cudaMemcpyAsync(hs.data(), s->dCs.p, sizeof(double) * hs.size(), cudaMemcpyDeviceToHost, s->st));
    RGPU_CUDA(cudaMemcpyAsync(pj.data(), s->nl.pair_j + p_base, sizeof(int32_t) * np, cudaMemcpyDeviceToHost,
                              s->st));
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    for (int64_t ci = c0; ci < c1; ++ci)
      for (int64_t p = poff[ci]; p < poff[ci + 1]; ++p) {
        const bool self = (p == poff[ci]);
        const int sj = self ? -1 : sidx.at(s->types[pj[size_t(p - p_base)]]);
        for (int c = 0; c < 3; ++c) {
          double * dst = out + (size_t(p) * 3 + c) * size_t(n_keys) * inner;
          for (int k = 0; k < n_keys; ++k) {
            const int b = blocks[k];
            const double * src = nullptr;
            if (b >= 0 && self)
              src = &hs[((size_t(ci - c0) * fd.S + b) * 3 + c) * fd.nK];
            else if (b >= 0 && b == sj)
              src = &hp[(size_t(p - p_base) * 3 + c) * fd.nK];
            if (src)
              std::memcpy(dst + size_t(k) * inner, src, sizeof(double) * inner);
            else
              std::memset(dst + size_t(k) * inner, 0, sizeof(double) * inner);
          }
        }
      }
    c0 = c1;
  }
}

void model_layout_bf16(rgpu_gap_model * m, rgpu_structures * s);

// Device copies of a model's sparse points in the batch's layout: FP64
// always, the BF16 splits of the tensor-core path only when `bf16` asks.
void model_layout(rgpu_gap_model * m, rgpu_structures * s, bool bf16) {
  bind_device(m->device, "the GAP model");
  const FeatureDims & fd = s->fd;
  if (m->layout_species == s->species && m->layout_D == fd.D) {
    if (bf16 && !m->layout_bf16) model_layout_bf16(m, s);
    return;
  }
  const int Sm = int(m->species.size());
  FeatureDims fm = make_dims(m->calc->hy, Sm);
  std::map<int, int> bidx;
  for (int i = 0; i < fd.S; ++i) bidx[s->species[i]] = i;
  std::vector<std::vector<int>> kb(fd.S, std::vector<int>(fd.S, -1));
  int k = 0;
  for (int a = 0; a < fd.S; ++a)
    for (int b = a; b < fd.S; ++b) kb[a][b] = k++;
  const int blk = fd.n * fd.n * (fd.L + 1);
  // group sparse points by batch species, keep their order inside a species
  std::vector<std::vector<int>> rows(fd.S);
  for (int i = 0; i < m->M; ++i) rows[bidx.at(m->sp_species[i])].push_back(i);
  m->segs.assign(fd.S, GapSpecies{});
  std::vector<double> T(size_t(m->M) * fd.Dpad, 0.), al(m->M);
  int pos = 0;
  int64_t tt_total = 0;
  std::vector<int32_t> user(size_t(std::max(m->M, 1)), 0);
  m->tt_off.assign(fd.S, 0);
  for (int sI = 0; sI < fd.S; ++sI) {
    GapSpecies & g = m->segs[sI];
    g.m0 = pos;
    g.M = int(rows[sI].size());
    g.Mpad = (g.M + 31) / 32 * 32;
    m->tt_off[sI] = tt_total;
    tt_total += int64_t(g.Mpad) * fd.Dg;
    for (int r : rows[sI]) {
      user[pos] = r;
      al[pos] = m->alpha[r];
      const double * src = &m->T[size_t(r) * fm.D];
      double * dst = &T[size_t(pos) * fd.Dpad];
      int km = 0;
      for (int a = 0; a < Sm; ++a)
        for (int b = a; b < Sm; ++b, ++km) {
          int A = bidx.at(m->species[a]), B = bidx.at(m->species[b]);
          int kk = kb[std::min(A, B)][std::max(A, B)];
          std::memcpy(dst + size_t(kk) * blk, src + size_t(km) * blk, sizeof(double) * blk);
        }
      ++pos;
    }
  }
  upload(s, m->T64, T.data(), sizeof(double) * T.size());
  upload(s, m->alpha64, al.data(), sizeof(double) * al.size());
  upload(s, m->ucol, user.data(), sizeof(int32_t) * user.size());
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  m->T_layout.swap(T);
  m->alpha_layout.swap(al);
  m->tt_total = tt_total;
  m->layout_species = s->species;
  m->layout_D = fd.D;
  m->layout_bf16 = false;
  if (bf16) model_layout_bf16(m, s);
}

// BF16 hi/lo splits of T (rows = sparse points) and of T^T per species
// (rows = feature index, padded to Mpad columns) for the tensor-core GEMMs.
void model_layout_bf16(rgpu_gap_model * m, rgpu_structures * s) {
  const FeatureDims & fd = s->fd;
  const std::vector<double> & T = m->T_layout;
  const std::vector<double> & al = m->alpha_layout;
  const int64_t tt_total = m->tt_total;
  auto f2bf = [](float f) -> uint16_t {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) return 0x7fc0;
    return uint16_t((u + 0x7fffu + ((u >> 16) & 1u)) >> 16);
  };
  auto bf2f = [](uint16_t h) -> float {
    uint32_t u = uint32_t(h) << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
  };
  // the BF16 copies use the packed layout of the FP32 path (padding stays 0)
  std::vector<uint16_t> Th(size_t(std::max(m->M, 1)) * fd.Dg, 0), Tl(Th.size(), 0);
  std::vector<double> packed(fd.Dg);
  for (int r = 0; r < m->M; ++r) {
    pack_reference_row(fd, &T[size_t(r) * fd.Dpad], packed.data());
    for (int d = 0; d < fd.Dg; ++d) {
      const float v = float(packed[d]);
      const size_t o = size_t(r) * fd.Dg + d;
      Th[o] = f2bf(v);
      Tl[o] = f2bf(v - bf2f(Th[o]));
    }
  }
  std::vector<float> al32(al.size());
  for (size_t i = 0; i < al.size(); ++i) al32[i] = float(al[i]);
  std::vector<uint16_t> Tth(size_t(std::max<int64_t>(tt_total, 1)), 0), Ttl(Tth.size(), 0);
  for (int sI = 0; sI < fd.S; ++sI) {
    const GapSpecies & g = m->segs[sI];
    for (int mm = 0; mm < g.M; ++mm)
      for (int d = 0; d < fd.Dg; ++d) {
        const size_t src = size_t(g.m0 + mm) * fd.Dg + d;
        const size_t dst = size_t(m->tt_off[sI]) + size_t(d) * g.Mpad + mm;
        Tth[dst] = Th[src];
        Ttl[dst] = Tl[src];
      }
  }
  upload(s, m->Th, Th.data(), sizeof(uint16_t) * Th.size());
  upload(s, m->Tl, Tl.data(), sizeof(uint16_t) * Tl.size());
  upload(s, m->alpha32, al32.data(), sizeof(float) * al32.size());
  upload(s, m->Tth, Tth.data(), sizeof(uint16_t) * Tth.size());
  upload(s, m->Ttl, Ttl.data(), sizeof(uint16_t) * Ttl.size());
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  m->layout_bf16 = true;
}

size_t plain_budget_bytes() { return size_t(24) << 30; }

// The dots K = X_s T_s^T of every central species, as planes in s->K64.
GapGroup species_dots(rgpu_gap_model * m, rgpu_structures * s) {
  const FeatureDims & fd = s->fd;
  GapGroup g;
  g.S = fd.S;
  for (int sI = 0; sI < fd.S; ++sI) {
    g.rows[sI] = s->species_count[sI];
    g.row0[sI + 1] = g.row0[sI] + g.rows[sI];
    g.M[sI] = m->segs[sI].M;
    g.m0[sI] = m->segs[sI].m0;
    g.ldk[sI] = (g.M[sI] + 1) & ~1;
    g.koff[sI] = g.plane;
    g.plane += g.rows[sI] * g.ldk[sI];
  }
  gap_dots_split(g, fd.D);
  s->K64.ensure(sizeof(double) * size_t(g.plane) * g.splits + 64);
  launch_gap_dots_fp64(g, fd.D, s->X64.as<double>(), fd.Dpad, m->T64.as<double>(), fd.Dpad, s->K64.as<double>(),
                       s->st);
  return g;
}

// FP64 prediction: energies, forces (F_d, = -dE/dr) and stress sums.
void gap_plain(rgpu_gap_model * m, rgpu_structures * s, double * E_d, double * F_d, bool forces, double * stress_d) {
  rgpu_calculator * c = m->calc;
  const FeatureDims & fd = s->fd;
  const int64_t nc = s->nl.n_centers;
  cudaStream_t st = s->st;
  mark(s, 4);
  // k = X T^T, pointwise, t = W T, all species in one launch each
  s->erow64.ensure(sizeof(double) * (nc + 1));
  s->t64.ensure(sizeof(double) * size_t(nc) * fd.Dpad + 64);
  const GapGroup g = species_dots(m, s);
  launch_gap_pointwise_fp64(g, s->K64.as<double>(), m->alpha64.as<double>(), m->zeta, s->erow64.as<double>(), st);
  if (forces) {
    launch_gap_scaled_fp64(g, fd.D, s->K64.as<double>(), m->T64.as<double>(), fd.Dpad, s->t64.as<double>(), fd.Dpad,
                           st);
    for (int sI = 0; sI < fd.S; ++sI)
      if (g.rows[sI] > 0 && g.M[sI] == 0)
        launch_fill_f64(s->t64.as<double>() + size_t(g.row0[sI]) * fd.Dpad, g.rows[sI] * fd.Dpad, 0., st);
  }
  // struct of each sorted row
  launch_energy_reduce(nc, EnergyParts{}, nullptr, s->erow64.as<double>(), s->center_of_row.as<int32_t>(),
                       s->nl.center_struct, E_d, st);
  mark(s, 5);
  mark(s, 6);
  if (!forces) {
    mark(s, 7);
    return;
  }
  PsArgs pa;
  pa.fd = fd;
  pa.n_centers = nc;
  pa.normalize = c->hy.normalize;
  pa.row_of_center = s->row_of_center.as<int32_t>();
  pa.present = s->present.as<uint32_t>();
  s->dC64.ensure(sizeof(double) * size_t(nc) * fd.S * fd.nK + 64);
  launch_ps_bwd_fp64(pa, s->C64.as<double>(), s->X64.as<double>(), s->invn64.as<double>(), s->t64.as<double>(),
                     s->dC64.as<double>(), st);
  mark(s, 7);
  launch_pair_adjoint_fp64(exp_args(c, s), s->dC64.as<double>(), s->nl.pair_center, s->nl.n_pairs, F_d,
                           s->nl.center_struct, stress_d, st);
}

// W offsets of the species segments (rows x Mpad BF16 each) in s->Wh/Wl.
std::vector<int64_t> w_offsets(const rgpu_gap_model * m, const rgpu_structures * s) {
  std::vector<int64_t> wofs(s->fd.S);
  int64_t woff = 0;
  for (int sI = 0; sI < s->fd.S; ++sI) {
    wofs[sI] = woff;
    woff += s->species_count[sI] * m->segs[sI].Mpad;
  }
  return wofs;
}

// Species skipping of a grouped GEMM over the packed columns (mode 1: K, the
// forward; 2: N, the backward), for layouts of more than one species group.
void set_segments(Bf16x3Gemm & a, const rgpu_structures * s, const TileMaskArgs & tm, int sI, int mode) {
  const FeatureDims & fd = s->fd;
  if (fd.G < 2) return;
  a.seg_mode = mode;
  a.seg_G = fd.G;
  a.seg_LD = fd.lenD / 32;
  a.seg_LO = fd.lenO / 32;
  a.tile_mask = s->tile_mask.as<uint32_t>() + tm.tile_off[sI];
}

// Fast path, forward half: the grouped tcgen05 GEMM with the GAP epilogue
// (energy partials and, for the backward half, W = alpha zeta k^(zeta-1) as
// a BF16 pair), then the per-structure energies (baseline not included).
void gap_fast_forward(rgpu_gap_model * m, rgpu_structures * s, double * E_d, bool need_w = true) {
  const FeatureDims & fd = s->fd;
  const int64_t nc = s->nl.n_centers;
  cudaStream_t st = s->st;
  s->fwd_model = 0;
  mark(s, 4);
  // per-species W (BF16 hi/lo) and energy partials ([tiles along M][rows])
  int points[kMaxSpecies];
  for (int sI = 0; sI < fd.S; ++sI) points[sI] = m->segs[sI].M;
  const int tile_n = gemm_forward_tile(s->species_count.data(), points, fd.S, fd.Dg);
  int64_t wtot = 0, eparts = 0, eofs[kMaxSpecies];
  for (int sI = 0; sI < fd.S; ++sI) {
    if (need_w) wtot += s->species_count[sI] * m->segs[sI].Mpad;
    eofs[sI] = eparts;
    eparts += s->species_count[sI] * ((points[sI] + tile_n - 1) / tile_n);
  }
  s->Wh.ensure(sizeof(uint16_t) * size_t(std::max<int64_t>(wtot, 1)) + 64);
  s->Wl.ensure(sizeof(uint16_t) * size_t(std::max<int64_t>(wtot, 1)) + 64);
  s->epart.ensure(sizeof(float) * size_t(std::max<int64_t>(eparts, 1)) + 64);
  if (need_w) s->dX32.ensure(sizeof(float) * size_t(nc) * fd.Dg + 64);
  const TileMaskArgs tm = tile_mask_args(s);
  const __nv_bfloat16 * Xh = s->Xh.as<__nv_bfloat16>();
  const __nv_bfloat16 * Xl = s->Xl.as<__nv_bfloat16>();
  __nv_bfloat16 * Wh = s->Wh.as<__nv_bfloat16>();
  __nv_bfloat16 * Wl = s->Wl.as<__nv_bfloat16>();
  const std::vector<int64_t> wofs = w_offsets(m, s);
  int64_t row0 = 0;
  std::vector<Bf16x3Gemm> fwd;
  for (int sI = 0; sI < fd.S; ++sI) {
    const int64_t rows = s->species_count[sI];
    const GapSpecies & g = m->segs[sI];
    if (rows > 0 && g.M > 0) {
      Bf16x3Gemm a{};
      a.M = rows;
      a.N = g.M;
      a.K = fd.Dg;
      a.A_hi = Xh + size_t(row0) * fd.Dg;
      a.A_lo = Xl + size_t(row0) * fd.Dg;
      a.lda = fd.Dg;
      a.B_hi = m->Th.as<__nv_bfloat16>() + size_t(g.m0) * fd.Dg;
      a.B_lo = m->Tl.as<__nv_bfloat16>() + size_t(g.m0) * fd.Dg;
      a.ldb = fd.Dg;
      a.epilogue = 1;
      a.W_hi = need_w ? Wh + wofs[sI] : nullptr;
      a.W_lo = need_w ? Wl + wofs[sI] : nullptr;
      a.ldw = g.Mpad;
      a.alpha = m->alpha32.as<float>() + g.m0;
      a.zeta = m->zeta;
      a.e_part = s->epart.as<float>() + eofs[sI];
      a.row_scale = s->xscale32.as<float>() + row0;  // k = (p . t) / |p|
      a.status = s->status_d->tc;
      set_segments(a, s, tm, sI, 1);  // K blocks of species pairs absent from a tile are skipped
      fwd.push_back(a);
    }
    row0 += rows;
  }
  gemm_bf16x3_grouped(fwd.data(), int(fwd.size()), st, tile_config(fd.S, fd.n, fd.L).gemm_variant, tile_n);
  EnergyParts ep;
  ep.S = fd.S;
  for (int sI = 0; sI < fd.S; ++sI) {
    ep.row0[sI + 1] = ep.row0[sI] + s->species_count[sI];
    ep.ofs[sI] = eofs[sI];
    ep.parts[sI] = (points[sI] + tile_n - 1) / tile_n;
  }
  launch_energy_reduce(nc, ep, s->epart.as<float>(), nullptr, s->center_of_row.as<int32_t>(), s->nl.center_struct,
                       E_d, st);
  mark(s, 5);
}

// The power-spectrum backward's chunk map depends on the layout alone: written
// when the layout changes, also before the replay of a graph recorded with
// another one than the last call's.
void ensure_chunk_map(rgpu_structures * s, const FeatureDims & fd) {
  if (s->chunk_map_of[0] == fd.S && s->chunk_map_of[1] == fd.n && s->chunk_map_of[2] == fd.L) return;
  s->chunk_map.ensure(sizeof(uint32_t) * size_t(fd.Dg / 4) + 64);
  launch_chunk_map(fd, s->chunk_map.as<uint32_t>(), s->st);
  s->chunk_map_of[0] = fd.S;
  s->chunk_map_of[1] = fd.n;
  s->chunk_map_of[2] = fd.L;
}

// Fast path, backward half: dE/dx = W T (grouped GEMM), the power-spectrum
// backward to dE/dc, then the pair adjoint into F_d (= -dE/dr) and the
// optional stress sums. With struct_scale, the contributions of every
// structure are multiplied by struct_scale[structure] (an upstream gradient
// per structure energy).
void gap_fast_backward(rgpu_gap_model * m, rgpu_structures * s, double * F_d, double * stress_d,
                       const double * struct_scale = nullptr) {
  rgpu_calculator * c = m->calc;
  const FeatureDims & fd = s->fd;
  const int64_t nc = s->nl.n_centers;
  cudaStream_t st = s->st;
  const __nv_bfloat16 * Xh = s->Xh.as<__nv_bfloat16>();
  const __nv_bfloat16 * Xl = s->Xl.as<__nv_bfloat16>();
  __nv_bfloat16 * Wh = s->Wh.as<__nv_bfloat16>();
  __nv_bfloat16 * Wl = s->Wl.as<__nv_bfloat16>();
  const std::vector<int64_t> wofs = w_offsets(m, s);
  int64_t row0 = 0;
  std::vector<Bf16x3Gemm> bwd;
  for (int sI = 0; sI < fd.S; ++sI) {
    const int64_t rows = s->species_count[sI];
    const GapSpecies & g = m->segs[sI];
    if (rows > 0 && g.M > 0) {
      Bf16x3Gemm a{};
      a.M = rows;
      a.N = fd.Dg;
      a.K = g.Mpad;
      a.A_hi = Wh + wofs[sI];
      a.A_lo = Wl + wofs[sI];
      a.lda = g.Mpad;
      a.B_hi = m->Tth.as<__nv_bfloat16>() + m->tt_off[sI];
      a.B_lo = m->Ttl.as<__nv_bfloat16>() + m->tt_off[sI];
      a.ldb = g.Mpad;
      a.epilogue = 0;
      a.C = s->dX32.as<float>() + size_t(row0) * fd.Dg;
      a.ldc = fd.Dg;
      // N tiles of species pairs absent from a tile are not computed; the
      // power-spectrum backward reads zeros for them (chunk map)
      a.status = s->status_d->tc;
      set_segments(a, s, tile_mask_args(s), sI, 2);
      bwd.push_back(a);
    } else if (rows > 0) {
      launch_fill_f32(s->dX32.as<float>() + size_t(row0) * fd.Dg, rows * fd.Dg, 0.f, st);
    }
    row0 += rows;
  }
  gemm_bf16x3_grouped(bwd.data(), int(bwd.size()), st, tile_config(fd.S, fd.n, fd.L).gemm_variant);
  mark(s, 6);
  PsArgs pa;
  pa.fd = fd;
  pa.n_centers = nc;
  pa.normalize = c->hy.normalize;
  pa.row_of_center = s->row_of_center.as<int32_t>();
  s->dC32.ensure(sizeof(float) * size_t(nc) * fd.S * fd.nK + 64);
  ensure_chunk_map(s, fd);
  launch_ps_bwd_fp32(pa, s->C32.as<float>(), Xh, Xl, s->xscale32.as<float>(), s->dX32.as<float>(),
                     s->chunk_map.as<uint32_t>(), s->present.as<uint32_t>(), s->dC32.as<float>(), st);
  mark(s, 7);
  ExpansionArgs ea = exp_args(c, s);
  launch_pair_adjoint_fp32(ea, s->nl.pair_center, s->nl.n_pairs, s->dC32.as<float>(), F_d, st,
                           s->nl.center_struct, stress_d, struct_scale);
}

void gap_fast(rgpu_gap_model * m, rgpu_structures * s, double * E_d, double * F_d, bool forces,
              double * stress_d) {
  gap_fast_forward(m, s, E_d, forces);
  if (forces) {
    gap_fast_backward(m, s, F_d, stress_d);
  } else {
    mark(s, 6);
    mark(s, 7);
  }
}

}  // namespace

// Cell volume as the reference computes it, from the lattice vector lengths
// and the cosines of the angles between them
// (structure_managers/atomic_structure.hh:137-155); rows of `cell` are the
// lattice vectors.
static double cell_volume(const double * cell) {
  double len[3], v[3][3];
  for (int i = 0; i < 3; ++i) {
    for (int k = 0; k < 3; ++k) v[i][k] = cell[3 * i + k];
    len[i] = std::sqrt(v[i][0] * v[i][0] + v[i][1] * v[i][1] + v[i][2] * v[i][2]);
  }
  auto dot = [&](int a, int b) { return v[a][0] * v[b][0] + v[a][1] * v[b][1] + v[a][2] * v[b][2]; };
  const double al = std::acos(dot(1, 2) / len[1] / len[2]);
  const double be = std::acos(dot(0, 2) / len[0] / len[2]);
  const double ga = std::acos(dot(1, 0) / len[1] / len[0]);
  const double c0 = std::cos(al), c1 = std::cos(be), c2 = std::cos(ga);
  return len[0] * len[1] * len[2] * std::sqrt(1 - c0 * c0 - c1 * c1 - c2 * c2 + 2 * c0 * c1 * c2);
}

extern "C" {
static void calculator_to_device(rgpu_calculator * c);
}

// Energy baseline of each structure (models/krr.py:68-90), FP64 on the host:
// a table over the atom types (validated to [0, 130) by rgpu_structures_set).
static std::vector<double> structure_baselines(const rgpu_gap_model * m, const rgpu_structures * s) {
  double sc[130] = {0.};
  for (size_t i = 0; i < m->species.size(); ++i)
    if (m->species[i] >= 0 && m->species[i] < 130) sc[m->species[i]] = m->self_contrib[i];
  std::vector<double> y0(s->n_struct, 0.);
  for (int k = 0; k < s->n_struct; ++k)
    for (int64_t a = s->atom_off[k]; a < s->atom_off[k + 1]; ++a) y0[k] += sc[s->types[a]];
  return y0;
}

// Energies, forces and (optionally) the negative stress of a GAP model: the
// reference's KRR.predict / predict_forces / predict_stress
// (bindings/rascal/models/krr.py:92-210) on the GPU.
static void gap_predict_impl(rgpu_gap_model * m, rgpu_structures * s, int precision, double * energies,
                             double * forces, double * neg_stress) {
  {
    if (!m || !s) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    if (s->has_mask)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "Can't compute spherical expansion gradients with masked center atoms",
                  RGPU_EXC_LOGIC_ERROR);
    calculator_to_device(m->calc);
    s->timed = true;
    mark(s, 0);
    // energies alone need neither the second GEMM nor the adjoint; a call
    // that asks for no output leaves both on the device
    const bool want_forces = forces || neg_stress || !energies;
    // neighbour list, layout, features
    build_nl(s, m->calc->hy.cutoff);
    mark(s, 1);
    // the gradients of what a prediction computed may be exported, forces or not
    compute_features(m->calc, s, precision, /*grads=*/true, m->species, /*need_x32=*/false);
    model_layout(m, s, precision == RGPU_PRECISION_FP32);
    const int64_t na = s->n_atoms;
    zero_outputs(s, want_forces, neg_stress != nullptr);
    double * stress_d = neg_stress ? s->S() : nullptr;
    if (precision == RGPU_PRECISION_FP64)
      gap_plain(m, s, s->E(), s->F(), want_forces, stress_d);
    else
      gap_fast(m, s, s->E(), s->F(), want_forces, stress_d);
    mark(s, 8);
    // outputs in one copy through the pinned staging buffer: a device-to-host
    // copy into the caller's pageable memory is staged by the driver at a
    // fraction of the bandwidth
    const size_t ns = size_t(s->n_struct), lo = energies ? 0 : (forces ? ns : ns + 3 * size_t(na)),
                 hi = neg_stress ? 7 * ns + 3 * size_t(na) : (forces ? ns + 3 * size_t(na) : (energies ? ns : lo));
    const size_t need = sizeof(double) * (hi - lo) + 64;
    if (need > s->pinned_cap) RGPU_CUDA(cudaStreamSynchronize(s->st));  // no copy may use the old buffer
    double * pin = static_cast<double *>(staging(s, need)) - lo;
    if (hi > lo)
      RGPU_CUDA(cudaMemcpyAsync(pin + lo, s->E() + lo, sizeof(double) * (hi - lo), cudaMemcpyDeviceToHost, s->st));
    if (precision == RGPU_PRECISION_FP32) fetch_status(s);
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    if (energies) std::memcpy(energies, pin, sizeof(double) * ns);
    if (forces) std::memcpy(forces, pin + ns, sizeof(double) * 3 * size_t(na));
    if (neg_stress) std::memcpy(neg_stress, pin + ns + 3 * size_t(na), sizeof(double) * 6 * ns);
    if (precision == RGPU_PRECISION_FP32) check_timeout(s);
    if (energies) {
      const std::vector<double> y0 = structure_baselines(m, s);
      for (int st = 0; st < s->n_struct; ++st) energies[st] += y0[st];
    }
    if (neg_stress)
      for (int st = 0; st < s->n_struct; ++st) {
        const double v = cell_volume(&s->cells_h[9 * size_t(st)]);
        for (int k = 0; k < 6; ++k) neg_stress[6 * st + k] /= v;
      }
  }
}

// Forward half of the adjoint path for automatic differentiation: energies
// of the FP32 path into device memory, with everything the backward needs
// (neighbour list, features, W) left on the device. The reference computes
// energies and forces in separate calls, KRR.predict and
// KRR.predict_forces (bindings/rascal/models/krr.py:92-166).
static void gap_forward_dev_impl(rgpu_gap_model * m, rgpu_structures * s, const double * positions_dev,
                                 double * energies_dev) {
  if (!m || !s || !energies_dev) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  if (s->has_mask)
    throw Error(RGPU_ERR_INVALID_ARGUMENT, "Can't compute spherical expansion gradients with masked center atoms",
                RGPU_EXC_LOGIC_ERROR);
  calculator_to_device(m->calc);
  s->timed = false;
  // the baselines go up before the stream has work: the upload waits for it
  const std::vector<double> y0 = structure_baselines(m, s);
  upload(s, s->y0_d, y0.data(), sizeof(double) * y0.size());
  if (positions_dev) {
    RGPU_CUDA(cudaMemcpyAsync(s->pos_d.p, positions_dev, sizeof(double) * 3 * s->n_atoms,
                              cudaMemcpyDeviceToDevice, s->st));
    s->nl_valid = false;
    s->feat_valid = false;
  }
  build_nl(s, m->calc->hy.cutoff);
  compute_features(m->calc, s, RGPU_PRECISION_FP32, true, m->species, /*need_x32=*/false);
  model_layout(m, s, true);
  zero_outputs(s, false, false);
  gap_fast_forward(m, s, s->E());
  launch_add_f64(s->E(), s->y0_d.as<double>(), energies_dev, s->n_struct, s->st);
  fetch_status(s);
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  check_timeout(s);
  s->fwd_model = m->serial;
}

// Backward half: grad_dev[a][c] = sum_A energies_grad_dev[A] dE_A/dr_a[c]
// from the state the forward left: dE/dx = W T, the power-spectrum
// backward, the per-structure scaling, the pair adjoint.
static void gap_backward_dev_impl(rgpu_gap_model * m, rgpu_structures * s, const double * energies_grad_dev,
                                  double * grad_dev) {
  if (!m || !s || !energies_grad_dev || !grad_dev) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  if (s->fwd_model != m->serial || !s->feat_valid || !s->nl_valid)
    throw Error(RGPU_ERR_NOT_COMPUTED, "the backward needs the forward of the same model and structures, with "
                                       "no other call on the structures in between");
  s->timed = false;
  const int64_t na = s->n_atoms;
  model_layout(m, s, true);  // another set may have used the model since
  zero_outputs(s, true, false);
  gap_fast_backward(m, s, s->F(), nullptr, energies_grad_dev);
  // the adjoint accumulates forces, -dE/dr
  launch_scale_f64(s->F(), -1.0, grad_dev, 3 * na, s->st);
  fetch_status(s);
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  check_timeout(s);
}

// ---------------------------------------------------------------- training
// Sparse kernel matrices of a GAP model (models/sparse_kernels.hh), FP64.
// Their columns follow the order in which the sparse points were given.
static void kernel_features(rgpu_gap_model * m, rgpu_structures * s, bool grads) {
  if (!m || !s) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  if (grads && s->has_mask)
    throw Error(RGPU_ERR_INVALID_ARGUMENT, "Can't compute spherical expansion gradients with masked center atoms",
                RGPU_EXC_LOGIC_ERROR);
  calculator_to_device(m->calc);
  s->timed = false;
  build_nl(s, m->calc->hy.cutoff);
  compute_features(m->calc, s, RGPU_PRECISION_FP64, grads, m->species, /*need_x32=*/false);
  model_layout(m, s, false);
}

// K_NM energy rows: SparseKernelImpl<GAP>::compute for target Structure
// (models/sparse_kernels.hh:104-131) or Atom (:165-191).
static void sparse_kernel_impl(rgpu_gap_model * m, rgpu_structures * s, bool atom_target, double * out) {
  kernel_features(m, s, false);
  const int64_t rows_out = atom_target ? s->nl.n_centers : s->n_struct;
  const size_t bytes = sizeof(double) * size_t(rows_out) * m->M;
  s->knm.ensure(bytes + 64);
  RGPU_CUDA(cudaMemsetAsync(s->knm.p, 0, bytes, s->st));
  const GapGroup g = species_dots(m, s);
  launch_knm_rows(g, s->K64.as<double>(), m->zeta, s->center_of_row.as<int32_t>(), s->nl.center_struct, atom_target,
                  m->ucol.as<int32_t>(), s->knm.as<double>(), m->M, s->st);
  if (bytes) RGPU_CUDA(cudaMemcpyAsync(out, s->knm.p, bytes, cudaMemcpyDeviceToHost, s->st));
  RGPU_CUDA(cudaStreamSynchronize(s->st));
}

// K_NM gradient rows: SparseKernelImpl<GAP>::compute_derivative
// (models/sparse_kernels.hh:258-499): the pairs' power-spectrum gradients are
// formed chunk by chunk and contracted with the sparse points (training.cu).
static void sparse_kernel_derivative_impl(rgpu_gap_model * m, rgpu_structures * s, bool neg_stress,
                                          double * out) {
  kernel_features(m, s, true);
  s->timed = true;
  for (int k = 0; k < 4; ++k) mark(s, k);
  rgpu_calculator * c = m->calc;
  const FeatureDims & fd = s->fd;
  const int64_t nc = s->nl.n_centers;
  const int M = m->M;
  cudaStream_t st = s->st;
  const int64_t rows_out = 3 * nc + (neg_stress ? 6 * int64_t(s->n_struct) : 0);
  const size_t bytes = sizeof(double) * size_t(rows_out) * M;
  s->knm.ensure(bytes + 64);
  RGPU_CUDA(cudaMemsetAsync(s->knm.p, 0, bytes, st));
  if (M == 0 || nc == 0) {
    RGPU_CUDA(cudaStreamSynchronize(st));
    return;
  }
  // x_i . T_m of every row
  mark(s, 4);
  const GapGroup gg = species_dots(m, s);
  launch_dots_sum(gg, s->K64.as<double>(), st);
  mark(s, 5);
  mark(s, 6);
  // The reference returns from its loop over structures at the first one
  // whose centre species have no sparse points (models/sparse_kernels.hh:
  // 347-349): that structure and all later ones keep zero rows.
  std::vector<int> sp_index(130, -1);
  for (int sI = 0; sI < fd.S; ++sI) sp_index[s->species[sI]] = sI;
  int64_t c_stop = nc;
  for (int st_i = 0; st_i < s->n_struct; ++st_i) {
    bool shared = false;
    for (int64_t a = s->atom_off[st_i]; a < s->atom_off[st_i + 1] && !shared; ++a)
      shared = m->segs[sp_index[s->types[a]]].M > 0;
    if (!shared) {
      c_stop = s->atom_off[st_i];  // centres are the atoms (no centre mask with gradients)
      break;
    }
  }
  const std::vector<int64_t> & poff = pair_offsets_host(s);
  KnmGradArgs a{};
  a.fd = fd;
  a.ea = exp_args(c, s);
  a.normalize = c->hy.normalize;
  a.pair_center = s->nl.pair_center;
  a.row_of_center = s->row_of_center.as<int32_t>();
  a.center_struct = s->nl.center_struct;
  a.C = s->C64.as<double>();
  a.inv_norm = s->invn64.as<double>();
  if (a.normalize) {
    // d(x . p)/dc: the power-spectrum backward of t = x without its
    // projection (inv_norm is applied by the pair rows)
    PsArgs pa;
    pa.fd = fd;
    pa.n_centers = nc;
    pa.normalize = false;
    pa.row_of_center = s->row_of_center.as<int32_t>();
    pa.present = s->present.as<uint32_t>();
    s->dC64.ensure(sizeof(double) * size_t(nc) * fd.S * fd.nK + 64);
    launch_ps_bwd_fp64(pa, s->C64.as<double>(), s->X64.as<double>(), s->invn64.as<double>(), s->X64.as<double>(),
                       s->dC64.as<double>(), st);
  }
  a.U = s->dC64.as<double>();
  s->Tq.ensure(sizeof(double) * size_t(fd.S) * M * knm_row_len(fd) + 64);
  launch_knm_points(fd, M, m->T64.as<double>(), fd.Dpad, s->Tq.as<double>(), st);
  a.Tq = s->Tq.as<double>();
  a.M = M;
  a.dots = &gg;
  a.K = s->K64.as<double>();
  a.zeta = m->zeta;
  a.ucol = m->ucol.as<int32_t>();
  a.out = s->knm.as<double>();
  a.ldo = M;
  a.stress_row0 = neg_stress ? 3 * nc : -1;
  // pairs in chunks of a bounded scratch
  const int64_t chunk = std::max<int64_t>(1, int64_t(plain_budget_bytes() / knm_pair_bytes(fd)));
  int64_t c0 = 0;
  while (c0 < c_stop) {
    int64_t c1 = c0 + 1;
    while (c1 < c_stop && poff[c1 + 1] - poff[c0] <= chunk) ++c1;
    a.p0 = poff[c0];
    a.p1 = poff[c1];
    launch_knm_gradient(a, s->plist, s->dXp, st);
    c0 = c1;
  }
  mark(s, 7);
  mark(s, 8);
  RGPU_CUDA(cudaMemcpyAsync(out, s->knm.p, bytes, cudaMemcpyDeviceToHost, st));
  RGPU_CUDA(cudaStreamSynchronize(st));
  if (neg_stress)
    for (int st_i = 0; st_i < s->n_struct; ++st_i) {
      const double v = cell_volume(&s->cells_h[9 * size_t(st_i)]);
      double * r = out + size_t(3 * nc + 6 * int64_t(st_i)) * M;
      for (int k = 0; k < 6 * M; ++k) r[k] /= v;
    }
}

// K_MM: SparseKernel::compute(sparse_points) (models/sparse_kernels.hh:
// 141-156, models/sparse_points.hh:144-170), one FP64 T_s T_s^T per species.
static void sparse_kernel_mm_impl(rgpu_gap_model * m, double * out) {
  if (!m) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  const int M = m->M;
  if (M == 0) return;
  const int Sm = int(m->species.size());
  const FeatureDims fm = make_dims(m->calc->hy, Sm);
  std::vector<int32_t> order;
  std::vector<int> m0(Sm + 1, 0);
  for (int a = 0; a < Sm; ++a) {
    m0[a] = int(order.size());
    for (int r = 0; r < M; ++r)
      if (m->sp_species[r] == m->species[a]) order.push_back(r);
  }
  m0[Sm] = int(order.size());
  std::vector<double> T(size_t(M) * fm.D);
  for (int k = 0; k < M; ++k)
    std::memcpy(&T[size_t(k) * fm.D], &m->T[size_t(order[k]) * fm.D], sizeof(double) * fm.D);
  int Mmax = 0;
  for (int a = 0; a < Sm; ++a) Mmax = std::max(Mmax, m0[a + 1] - m0[a]);
  cudaStream_t st = nullptr;
  RGPU_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamSynchronize(s); cudaStreamDestroy(s); }
  } guard_st{st};
  DevBuf Td, Kd, Od, Ud;
  Td.ensure(sizeof(double) * T.size());
  Kd.ensure(sizeof(double) * size_t(Mmax) * Mmax + 64);
  Od.ensure(sizeof(double) * size_t(M) * M);
  Ud.ensure(sizeof(int32_t) * order.size());
  RGPU_CUDA(cudaMemcpyAsync(Td.p, T.data(), sizeof(double) * T.size(), cudaMemcpyHostToDevice, st));
  RGPU_CUDA(cudaMemcpyAsync(Ud.p, order.data(), sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice, st));
  RGPU_CUDA(cudaMemsetAsync(Od.p, 0, sizeof(double) * size_t(M) * M, st));
  for (int a = 0; a < Sm; ++a) {
    const int Ms = m0[a + 1] - m0[a];
    if (Ms == 0) continue;
    const double * Ts = Td.as<double>() + size_t(m0[a]) * fm.D;
    gemm_nt_fp64(Ms, Ms, fm.D, Ts, fm.D, Ts, fm.D, Kd.as<double>(), Ms, st);
    launch_kmm_scatter(Ms, Kd.as<double>(), m->zeta, Ud.as<int32_t>() + m0[a], Od.as<double>(), M, st);
  }
  RGPU_CUDA(cudaMemcpyAsync(out, Od.p, sizeof(double) * size_t(M) * M, cudaMemcpyDeviceToHost, st));
  RGPU_CUDA(cudaStreamSynchronize(st));
}

// ------------------------------------------------------------------ MD step
// A step of a molecular-dynamics loop on a fixed set of structures: the FP32
// path from new positions to energies, forces (and the negative stress),
// with no host synchronisation inside, so that it is recorded once as a
// CUDA graph and then replayed. The neighbour list is built to capacities
// 25 % above the counts of the step that recorded the graph; when a step
// outgrows them (status 104) it is recomputed by the ordinary path and the
// graph is recorded again.
// Addresses of every device buffer a recorded step can use: those of the
// structures handle (neighbour-list work included), of the model and of its
// calculator. The recording is replayed only while none of them moved.
static std::vector<const void *> md_buffers(const rgpu_gap_model * m, const rgpu_structures * s) {
  std::vector<const void *> v;
  for (const DevView * b : {&s->atom_off_d, &s->pos_d, &s->types_d, &s->cells_d, &s->pbc_d, &s->ncent_d,
                            &s->center_off_d, &s->atom_struct_d})
    v.push_back(b->p);
  for (const DevBuf * b : {&s->lut, &s->row_of_center,
                           &s->center_of_row, &s->sort_tmp, &s->present, &s->tile_mask,
                           &s->C64, &s->X64,
                           &s->invn64, &s->dC64, &s->C32, &s->X32, &s->xscale32, &s->out_d, &s->K64,
                           &s->t64, &s->erow64, &s->Wh, &s->Wl, &s->dX32, &s->dC32, &s->epart, &s->Xh, &s->Xl,
                           &s->chunk_map, &s->dCp, &s->dCs, &s->dXp, &s->knm, &s->plist, &s->Tq})
    v.push_back(b->p);
  const NlWork & w = s->nlw;
  for (const DevBuf * b : {&w.geom, &w.counts64, &w.scan_tmp, &w.ghost_off, &w.site_x, &w.site_type, &w.site_real,
                           &w.site_shift, &w.site_box, &w.box_base, &w.box_count, &w.box_ptr, &w.binned,
                           &w.sorted, &w.sorted_x, &w.pair_count, &w.center_atom,
                           &w.center_struct, &w.pair_off, &w.pair_j, &w.pair_shift, &w.pair_dist, &w.pair_dir,
                           &w.pair_center})
    v.push_back(b->p);
  for (const DevBuf * b : {&m->T64, &m->alpha64, &m->Th, &m->Tl, &m->Tth, &m->Ttl, &m->alpha32, &m->ucol})
    v.push_back(b->p);
  const rgpu_calculator * c = m->calc;
  for (const DevBuf * b : {&c->grid, &c->y, &c->y2h, &c->q4f, &c->center}) v.push_back(b->p);
  return v;
}

static void md_drop(rgpu_structures * s) {
  if (s->md_exec) cudaGraphExecDestroy(s->md_exec);
  if (s->md_graph) cudaGraphDestroy(s->md_graph);
  s->md_exec = nullptr;
  s->md_graph = nullptr;
  s->md_model = 0;
}

// The FP32 prediction on the structures' stream with no host
// synchronisation, so that it can be recorded: positions from pinned
// pos_h (null: those already on the device), the neighbour list to `caps`,
// outputs (energies, forces, stress sums) into pinned out_h (null: left on
// the device), and the status word copied to the host at the end.
static void graph_enqueue(rgpu_gap_model * m, rgpu_structures * s, bool stress, const double * pos_h,
                          double * out_h, const NlCaps & caps, bool forces = true) {
  rgpu_calculator * c = m->calc;
  cudaStream_t st = s->st;
  const int64_t na = s->n_atoms;
  if (pos_h) RGPU_CUDA(cudaMemcpyAsync(s->pos_d.p, pos_h, sizeof(double) * 3 * na, cudaMemcpyHostToDevice, st));
  NlInputs in;
  in.n_struct = s->n_struct;
  in.n_atoms = na;
  in.atom_off = s->atom_off_d.as<int64_t>();
  in.pos = s->pos_d.as<double>();
  in.types = s->types_d.as<int32_t>();
  in.cells = s->cells_d.as<double>();
  in.pbc = s->pbc_d.as<int32_t>();
  in.tag2idx = nullptr;
  in.n_centers = s->ncent_d.as<int32_t>();
  in.center_off = s->center_off_d.as<int64_t>();
  in.atom_struct = s->atom_struct_d.as<int32_t>();
  in.n_centers_total = s->center_off_h[s->n_struct];
  build_neighbour_list(in, c->hy.cutoff, s->nlw, s->nl, &s->status_d->nl, &s->status_h->nl, st, &caps);
  // features (the FP32 branch of compute_features, layout unchanged)
  const bool by_mask = sorts_by_mask(c, s);
  sort_rows(s, by_mask);
  const int64_t nc = s->nl.n_centers;
  const FeatureDims & fd = s->fd;
  ExpansionArgs ea = exp_args(c, s);
  PsArgs pa;
  pa.fd = fd;
  pa.n_centers = nc;
  pa.normalize = c->hy.normalize;
  pa.row_of_center = s->row_of_center.as<int32_t>();
  launch_expansion_fp32(ea, s->C32.as<float>(), s->present.as<uint32_t>(), st);
  if (by_mask) sort_rows_by_mask(s);
  pa.present = s->present.as<uint32_t>();
  pa.tc_status = s->status_d->tc;
  launch_ps_fwd_fast(pa, s->C32.as<float>(), nullptr, s->Xh.as<__nv_bfloat16>(), s->Xl.as<__nv_bfloat16>(),
                     s->xscale32.as<float>(), st);
  zero_outputs(s, forces, stress);
  gap_fast(m, s, s->E(), s->F(), forces, stress ? s->S() : nullptr);
  if (out_h) {
    const size_t n = size_t(s->n_struct) * (stress ? 7 : 1) + (forces ? 3 * size_t(na) : 0);
    if (n) RGPU_CUDA(cudaMemcpyAsync(out_h, s->E(), sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  }
  fetch_status(s);
}

// The step's work on the structures' stream, positions from s->md_pos_h.
static void md_enqueue(rgpu_gap_model * m, rgpu_structures * s, bool stress) {
  graph_enqueue(m, s, stress, s->md_pos_h, s->md_out_h, s->md_caps);
}

// Kernel nodes of a recorded graph (the kernels one replay launches).
static int64_t graph_kernels(cudaGraph_t g) {
  size_t n = 0;
  int64_t k = 0;
  if (cudaGraphGetNodes(g, nullptr, &n) == cudaSuccess && n > 0) {
    std::vector<cudaGraphNode_t> nodes(n);
    if (cudaGraphGetNodes(g, nodes.data(), &n) == cudaSuccess)
      for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) ++k;
      }
  }
  return k;
}

// Energy baseline and cell volume, as in gap_predict_impl.
static void md_finish(const rgpu_gap_model * m, const rgpu_structures * s, double * energies, double * forces,
                      double * neg_stress) {
  const int64_t na = s->n_atoms;
  const double * out = s->md_out_h;
  if (energies) {
    double sc[130] = {0.};
    for (size_t i = 0; i < m->species.size(); ++i)
      if (m->species[i] >= 0 && m->species[i] < 130) sc[m->species[i]] = m->self_contrib[i];
    for (int st = 0; st < s->n_struct; ++st) {
      double y0 = 0.;
      for (int64_t a = s->atom_off[st]; a < s->atom_off[st + 1]; ++a) y0 += sc[s->types[a]];
      energies[st] = out[st] + y0;
    }
  }
  if (forces) std::memcpy(forces, out + s->n_struct, sizeof(double) * 3 * na);
  if (neg_stress)
    for (int st = 0; st < s->n_struct; ++st) {
      const double v = cell_volume(&s->cells_h[9 * size_t(st)]);
      for (int k = 0; k < 6; ++k) neg_stress[6 * st + k] = out[s->n_struct + 3 * na + 6 * st + k] / v;
    }
}

static void md_step_impl(rgpu_gap_model * m, rgpu_structures * s, const double * positions, double * energies,
                         double * forces, double * neg_stress) {
  if (!m || !s || !positions) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  const bool stress = neg_stress != nullptr;
  const int64_t na = s->n_atoms;
  ensure_stream(s);
  bool replay = false;
  if (s->md_exec) {
    if (s->md_model == m->serial) {
      // the model's device copies may be laid out for another set's species
      set_layout(s, m->calc->hy, m->species);
      model_layout(m, s, true);
    }
    if (s->md_model != m->serial || s->md_stress != stress || s->md_species != s->species)
      s->md_reason = 3;
    else if (md_buffers(m, s) != s->md_buffers)
      s->md_reason = 1;
    else
      replay = true;
  }
  if (replay) {
    std::memcpy(s->md_pos_h, positions, sizeof(double) * 3 * na);
    ensure_chunk_map(s, s->fd);
    drop_results(s);  // the replay overwrites positions, list and features
    RGPU_CUDA(cudaGraphLaunch(s->md_exec, s->st));
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    ++s->md_replays;
    check_timeout(s);
    if (s->status_h->nl.code == 0) {
      md_finish(m, s, energies, forces, neg_stress);
      return;
    }
    // outgrown capacities or an input error: the ordinary path below
    // rebuilds, or reports the error with its message
    s->md_reason = 100 + s->status_h->nl.code;
    reset_status(s);
  }
  md_drop(s);
  // the ordinary path: checks the input, sizes every buffer, gives this step's results
  drop_results(s);
  upload_positions(s, positions);
  gap_predict_impl(m, s, RGPU_PRECISION_FP32, energies, forces, neg_stress);
  if (s->md_no_graph) return;
  // capacities 25 % above this step's counts
  int64_t sites = 0, boxes = 0;
  neighbour_list_counts(s->nlw, sites, boxes);
  s->md_caps.sites = sites + sites / 4 + 64;
  s->md_caps.boxes = boxes + boxes / 4 + 64;
  s->md_caps.pairs = s->nl.n_pairs + s->nl.n_pairs / 4 + 256;
  if (s->md_pos_cap < size_t(3 * na)) {
    if (s->md_pos_h) cudaFreeHost(s->md_pos_h);
    RGPU_CUDA(cudaMallocHost(&s->md_pos_h, sizeof(double) * 3 * std::max<int64_t>(na, 1)));
    s->md_pos_cap = size_t(3 * na);
  }
  const size_t nout = size_t(s->n_struct) * 7 + 3 * size_t(na);
  if (s->md_out_cap < nout) {
    if (s->md_out_h) cudaFreeHost(s->md_out_h);
    RGPU_CUDA(cudaMallocHost(&s->md_out_h, sizeof(double) * std::max<size_t>(nout, 1)));
    s->md_out_cap = nout;
  }
  std::memcpy(s->md_pos_h, positions, sizeof(double) * 3 * na);
  // one run without recording sizes the capacity buffers (no allocation may
  // happen while recording) and checks that the step fits them
  s->timed = false;
  drop_results(s);  // the list becomes the capacity-bound one
  md_enqueue(m, s, stress);
  RGPU_CUDA(cudaStreamSynchronize(s->st));
  if (s->status_h->nl.code != 0 || timed_out(s)) {
    // cannot happen with fresh capacities unless something is off: leave
    // the step to the ordinary path next time
    reset_status(s);
    return;
  }
  // record; a step that cannot be recorded keeps the ordinary path
  bool ok = cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
  if (ok) {
    try {
      md_enqueue(m, s, stress);
    } catch (...) {
      ok = false;
    }
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(s->st, &g);
    ok = ok && e == cudaSuccess && g != nullptr;
    if (ok) {
      s->md_graph = g;
      ok = cudaGraphInstantiate(&s->md_exec, s->md_graph, 0) == cudaSuccess;
    } else if (g) {
      cudaGraphDestroy(g);
    }
  }
  if (!ok) {
    (void)cudaGetLastError();
    md_drop(s);
    s->md_no_graph = true;
    return;
  }
  s->md_model = m->serial;
  s->md_stress = stress;
  s->md_buffers = md_buffers(m, s);
  s->md_species = s->species;
  s->md_kernels = graph_kernels(s->md_graph);
  s->md_replays = 0;
  // the ordinary step above already produced this call's results; the
  // positions of the next step arrive in md_pos_h
}

// ------------------------------------------------- predictions as CUDA graphs
static void pgraph_release(PredictGraph & g) {
  if (g.exec) cudaGraphExecDestroy(g.exec);
  if (g.graph) cudaGraphDestroy(g.graph);
  if (g.out_h) cudaFreeHost(g.out_h);
  g = PredictGraph{};
}

static std::vector<int64_t> centres_per_species(const rgpu_structures * s) {
  std::vector<int64_t> c(s->species.size());
  for (size_t i = 0; i < s->species.size(); ++i) c[i] = s->centres_of_type[s->species[i]];
  return c;
}

// Outputs of a replay, from its pinned copy: baseline added to the
// energies, stress sums divided by the cell volumes (as gap_predict_impl).
static void pgraph_outputs(const rgpu_gap_model * m, const rgpu_structures * s, const PredictGraph & g,
                           double * energies, double * forces, double * neg_stress) {
  const int64_t na = s->n_atoms;
  const double * out = g.out_h;
  if (energies) {
    const std::vector<double> y0 = structure_baselines(m, s);
    for (int k = 0; k < s->n_struct; ++k) energies[k] = out[k] + y0[k];
  }
  if (forces) std::memcpy(forces, out + s->n_struct, sizeof(double) * 3 * na);
  if (neg_stress)
    for (int k = 0; k < s->n_struct; ++k) {
      const double v = cell_volume(&s->cells_h[9 * size_t(k)]);
      for (int j = 0; j < 6; ++j) neg_stress[6 * k + j] = out[s->n_struct + 3 * na + 6 * k + j] / v;
    }
}

static bool pbucket_matches(const PredictBucket & b, const rgpu_gap_model * m, const rgpu_structures * s, bool stress,
                            bool outputs, const std::vector<int64_t> & species_count) {
  return b.model == m->serial && b.stress == stress && b.outputs == outputs && b.n_struct == s->n_struct &&
         b.n_atoms == s->n_atoms && b.species == s->species && b.species_count == species_count;
}

static void pbucket_release(PredictBucket & b) {
  pgraph_release(b.full);
  pgraph_release(b.alone);
}

// The bucket of a call that the ordinary path has answered (its layout is
// set); a new one takes the place of the one unused for longest.
static PredictBucket & pbucket_of(const rgpu_gap_model * m, rgpu_structures * s, bool stress, bool outputs) {
  const std::vector<int64_t> cnt = centres_per_species(s);
  for (PredictBucket & b : s->pbuckets)
    if (pbucket_matches(b, m, s, stress, outputs, cnt)) return b;
  if (s->pbuckets.size() >= kMaxBuckets) {
    auto lru = std::min_element(s->pbuckets.begin(), s->pbuckets.end(),
                                [](const PredictBucket & a, const PredictBucket & b) { return a.used < b.used; });
    pbucket_release(*lru);
    s->pbuckets.erase(lru);
  }
  PredictBucket b;
  b.model = m->serial;
  b.stress = stress;
  b.outputs = outputs;
  b.n_struct = s->n_struct;
  b.n_atoms = s->n_atoms;
  b.species = s->species;
  b.species_count = cnt;
  s->pbuckets.push_back(b);
  return s->pbuckets.back();
}

// Replays the recorded graph of this call's size bucket, if there is one:
// true when it produced the call's results. A replay whose neighbour list
// outgrew its capacities, or whose input is invalid, drops the recording and
// leaves the call to the ordinary path (which reports input errors with the
// reference's messages).
static bool pgraph_replay(rgpu_gap_model * m, rgpu_structures * s, bool stress, double * energies,
                          double * forces, double * neg_stress) {
  if (s->pbuckets.empty()) return false;
  calculator_to_device(m->calc);
  set_layout(s, m->calc->hy, m->species);
  model_layout(m, s, true);
  const bool outputs = energies || forces || neg_stress, alone = energies && !forces && !neg_stress;
  const std::vector<int64_t> cnt = centres_per_species(s);
  for (PredictBucket & b : s->pbuckets) {
    if (!pbucket_matches(b, m, s, stress, outputs, cnt)) continue;
    const std::vector<const void *> bufs = md_buffers(m, s);
    auto good = [&](const PredictGraph & g) { return g.exec && g.buffers == bufs; };
    // The first two calls for energies alone take the full recording where
    // there is one: a caller that asks for the energies once or twice beside
    // the forces does not pay for a second recording.
    PredictGraph * g = alone && good(b.alone) ? &b.alone : nullptr;
    if (!g && good(b.full) && (!alone || b.energies_alone < 2)) {
      g = &b.full;
      if (alone) ++b.energies_alone;
    }
    if (!g) return false;
    s->timed = false;
    if (g == &b.full) ensure_chunk_map(s, s->fd);
    drop_results(s);  // the list becomes the capacity-bound one
    RGPU_CUDA(cudaGraphLaunch(g->exec, s->st));
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    check_timeout(s);
    if (s->status_h->nl.code != 0) {
      reset_status(s);
      pgraph_release(*g);
      return false;
    }
    b.used = ++s->pgraph_clock;
    ++s->pgraph_replays;
    s->pgraph_last_kernels = g->kernels;
    pgraph_outputs(m, s, *g, energies, forces, neg_stress);
    return true;
  }
  return false;
}

// Records a call's kind in its bucket after an ordinary FP32 prediction: one
// run to the new capacities without recording (it sizes every buffer, since
// nothing may be allocated while recording, and checks that the call fits
// them), then the recording. A failure leaves the calls of this kind on the
// ordinary path.
static void pgraph_record(rgpu_gap_model * m, rgpu_structures * s, PredictBucket & b, bool alone) {
  PredictGraph & slot = alone ? b.alone : b.full;
  pgraph_release(slot);
  PredictGraph g;
  int64_t sites = 0, boxes = 0;
  neighbour_list_counts(s->nlw, sites, boxes);
  g.caps.sites = sites + sites / 8 + 64;
  g.caps.boxes = boxes + boxes / 8 + 64;
  g.caps.pairs = s->nl.n_pairs + s->nl.n_pairs / 8 + 256;
  if (b.outputs) {
    const size_t nout = size_t(s->n_struct) * 7 + 3 * size_t(s->n_atoms) + 1;
    RGPU_CUDA(cudaMallocHost(&g.out_h, sizeof(double) * nout));
  }
  s->timed = false;
  drop_results(s);  // the list becomes the capacity-bound one
  bool ok = true;
  try {
    graph_enqueue(m, s, b.stress, nullptr, g.out_h, g.caps, !alone);
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    ok = s->status_h->nl.code == 0 && !timed_out(s);
  } catch (...) {
    ok = false;
  }
  if (ok) {
    ok = cudaStreamBeginCapture(s->st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (ok) {
      try {
        graph_enqueue(m, s, b.stress, nullptr, g.out_h, g.caps, !alone);
      } catch (...) {
        ok = false;
      }
      cudaGraph_t gr = nullptr;
      const cudaError_t e = cudaStreamEndCapture(s->st, &gr);
      ok = ok && e == cudaSuccess && gr != nullptr;
      if (gr) g.graph = gr;
      ok = ok && cudaGraphInstantiate(&g.exec, g.graph, 0) == cudaSuccess;
    }
  }
  if (!ok) {
    (void)cudaGetLastError();
    reset_status(s);
    pgraph_release(g);
    return;
  }
  g.buffers = md_buffers(m, s);
  g.kernels = graph_kernels(g.graph);
  slot = g;
  ++s->pgraph_records;
}

// rgpu_gap_predict(_stress): FP32 calls go through the recorded graph of
// their size bucket when one exists, otherwise through the ordinary path,
// after which the call is recorded, energies alone from their second time on.
static void gap_predict_entry(rgpu_gap_model * m, rgpu_structures * s, int precision, double * energies,
                              double * forces, double * neg_stress) {
  if (!m || !s) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
  const bool graphs = precision == RGPU_PRECISION_FP32 && s->use_graphs && !s->has_mask;
  const bool stress = neg_stress != nullptr;
  if (graphs && pgraph_replay(m, s, stress, energies, forces, neg_stress)) return;
  gap_predict_impl(m, s, precision, energies, forces, neg_stress);
  if (!graphs) return;
  const bool alone = energies && !forces && !stress;
  PredictBucket & b = pbucket_of(m, s, stress, energies || forces || stress);
  b.used = ++s->pgraph_clock;
  if (!alone || ++b.energies_alone >= 2) pgraph_record(m, s, b, alone);
}

// ===================================================================== C ABI
extern "C" {

const char * rgpu_last_error(void) { return t_err.c_str(); }
int rgpu_error_kind(void) { return t_kind; }
int rgpu_version(void) { return 1; }

rgpu_status rgpu_calculator_create(const char * kind, const char * hypers_json, rgpu_calculator ** out) {
  return guard([&] {
    if (!kind || !hypers_json || !out) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    auto c = std::make_unique<rgpu_calculator>();
    parse_hypers(kind, hypers_json, c->hy);
    build_radial_spline(c->hy, c->spline);
    *out = c.release();
  });
}

rgpu_status rgpu_calculator_destroy(rgpu_calculator * calc) {
  return guard([&] { delete calc; });
}

// Device copies of the radial table, made on first use so that a calculator
// can be built (and its FP64 table inspected) on a host without a GPU.
static void calculator_to_device(rgpu_calculator * c) {
  bind_device(c->device, "the calculator");
  if (c->dev.y) return;
  {
    const RadialSpline & sp = c->spline;
    const size_t GW = size_t(sp.grid_size) * sp.width;
    std::vector<float> yf(GW), y2hf(GW);
    for (size_t i = 0; i < GW; ++i) {
      yf[i] = float(sp.y[i]);
      y2hf[i] = float(sp.y2h[i]);
    }
    // interval table of the FP32 path: one 16-byte load per channel, the
    // channels of one l side by side
    const size_t W = size_t(sp.width), L1 = size_t(c->hy.max_angular) + 1, n = W / L1;
    std::vector<float> q4(size_t(std::max(sp.grid_size - 1, 1)) * W * 4, 0.f);
    for (int k = 0; k + 1 < sp.grid_size; ++k)
      for (size_t ch = 0; ch < W; ++ch) {
        float * o = &q4[(size_t(k) * W + ch) * 4];
        const size_t c = ch % n * L1 + ch / n;
        o[0] = yf[size_t(k) * W + c];
        o[1] = y2hf[size_t(k) * W + c];
        o[2] = yf[size_t(k + 1) * W + c];
        o[3] = y2hf[size_t(k + 1) * W + c];
      }
    std::vector<double> center(sp.center.size());
    for (size_t i = 0; i < center.size(); ++i) center[i] = sp.center[i] / std::sqrt(4.0 * kPi);
    auto put = [](DevBuf & b, const void * src, size_t bytes) {
      b.ensure(bytes);
      RGPU_CUDA(cudaMemcpy(b.p, src, bytes, cudaMemcpyHostToDevice));
    };
    put(c->grid, sp.grid.data(), sizeof(double) * sp.grid.size());
    put(c->y, sp.y.data(), sizeof(double) * GW);
    put(c->y2h, sp.y2h.data(), sizeof(double) * GW);
    put(c->q4f, q4.data(), sizeof(float) * q4.size());
    put(c->center, center.data(), sizeof(double) * center.size());
    c->dev.grid = c->grid.as<double>();
    c->dev.y = c->y.as<double>();
    c->dev.y2h = c->y2h.as<double>();
    c->dev.q4f = c->q4f.as<float4>();
    c->dev.x1 = sp.x1;
    c->dev.h = sp.h;
    c->dev.inv_h = 1.0 / sp.h;
    c->dev.ppu = sp.points_per_unit;
    c->dev.search_size = sp.search_size;
    c->dev.W = sp.width;
  }
}

rgpu_status rgpu_calculator_name(const rgpu_calculator * calc, char * buf, size_t buflen) {
  return guard([&] {
    if (!calc || !buf) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    std::snprintf(buf, buflen, "%s", calc->hy.name.c_str());
  });
}

rgpu_status rgpu_calculator_spline_shape(const rgpu_calculator * calc, int32_t * grid_size, int32_t * width) {
  return guard([&] {
    *grid_size = calc->spline.grid_size;
    *width = calc->spline.width;
  });
}

rgpu_status rgpu_calculator_spline_table(const rgpu_calculator * calc, double * grid, double * y, double * y2h) {
  return guard([&] {
    const RadialSpline & s = calc->spline;
    if (grid) std::memcpy(grid, s.grid.data(), sizeof(double) * s.grid.size());
    if (y) std::memcpy(y, s.y.data(), sizeof(double) * s.y.size());
    if (y2h) std::memcpy(y2h, s.y2h.data(), sizeof(double) * s.y2h.size());
  });
}

rgpu_status rgpu_structures_create(rgpu_structures ** out) {
  return guard([&] {
    auto s = std::make_unique<rgpu_structures>();
    ensure_stream(s.get());
    *out = s.release();
  });
}

rgpu_status rgpu_structures_destroy(rgpu_structures * s) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s) return;
    if (s->st) cudaStreamSynchronize(s->st);
    if (s->md_exec) cudaGraphExecDestroy(s->md_exec);
    if (s->md_graph) cudaGraphDestroy(s->md_graph);
    for (PredictBucket & b : s->pbuckets) pbucket_release(b);
    if (s->md_pos_h) cudaFreeHost(s->md_pos_h);
    if (s->md_out_h) cudaFreeHost(s->md_out_h);
    if (s->pinned) cudaFreeHost(s->pinned);
    if (s->status_h) cudaFreeHost(s->status_h);
    if (s->status_d) cudaFree(s->status_d);
    for (auto & e : s->ev)
      if (e) cudaEventDestroy(e);
    if (s->st) cudaStreamDestroy(s->st);
    delete s;
  });
}

rgpu_status rgpu_structures_set(rgpu_structures * s, int32_t n_structures, const int64_t * atom_offsets,
                                const double * positions, const int32_t * numbers, const double * cells,
                                const int32_t * pbc, const uint8_t * center_mask) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s || n_structures < 0 || !atom_offsets) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    // everything is checked before the handle changes: a batch that is refused
    // leaves the former one in place
    if (atom_offsets[0] != 0) throw Error(RGPU_ERR_INVALID_ARGUMENT, "atom_offsets must start at 0");
    for (int i = 0; i < n_structures; ++i)
      if (atom_offsets[i + 1] < atom_offsets[i])
        throw Error(RGPU_ERR_INVALID_ARGUMENT, "atom_offsets must be non-decreasing");
    const int64_t n_atoms = atom_offsets[n_structures];
    if (n_atoms > (int64_t(1) << 31) - 1) throw Error(RGPU_ERR_INVALID_ARGUMENT, "too many atoms");
    // The mesh of a cell that is not finite has no boxes, and every site falls
    // outside. One pass without branches, then the search.
    const int64_t n_cell = 9 * int64_t(n_structures);
    unsigned bad = 0;
    for (int64_t k = 0; k < n_cell; ++k) bad |= unsigned(!(std::fabs(cells[k]) <= std::numeric_limits<double>::max()));
    for (int64_t k = 0; bad && k < n_cell; ++k)
      if (!std::isfinite(cells[k]))
        throw Error(RGPU_ERR_STRUCTURE,
                    "the unit cell holds a value that is not finite (structure " + std::to_string(k / 9) + ")");
    bool seen[130] = {false};
    for (int64_t a = 0; a < n_atoms; ++a) {
      if (numbers[a] < 0 || numbers[a] >= 130)
        throw Error(RGPU_ERR_STRUCTURE, "atom types (or atomic numbers) should be in the range [0, 130].");
      seen[numbers[a]] = true;
    }
    ensure_stream(s);
    md_drop(s);
    s->md_no_graph = false;
    drop_results(s);
    try {
      s->n_struct = n_structures;
      s->atom_off.assign(atom_offsets, atom_offsets + n_structures + 1);
      s->n_atoms = n_atoms;
      s->types.assign(numbers, numbers + s->n_atoms);
      s->cells_h.assign(cells, cells + 9 * size_t(n_structures));
      s->batch_species.clear();
      for (int z = 0; z < 130; ++z)
        if (seen[z]) s->batch_species.push_back(z);
      s->has_mask = false;
      if (center_mask)
        for (int64_t a = 0; a < s->n_atoms; ++a)
          if (!center_mask[a]) s->has_mask = true;
      std::fill(s->centres_of_type, s->centres_of_type + 130, int64_t(0));
      for (int64_t a = 0; a < s->n_atoms; ++a)
        if (!center_mask || center_mask[a]) ++s->centres_of_type[s->types[a]];
      std::vector<int32_t> ncent(n_structures), astruct(s->n_atoms);
      s->center_off_h.assign(n_structures + 1, 0);
      std::vector<int32_t> tag2idx;
      if (s->has_mask) tag2idx.resize(s->n_atoms);
      for (int i = 0; i < n_structures; ++i) {
        int64_t a0 = s->atom_off[i], a1 = s->atom_off[i + 1];
        int nc = 0;
        for (int64_t a = a0; a < a1; ++a) {
          astruct[a] = i;
          if (!center_mask || center_mask[a]) ++nc;
        }
        ncent[i] = nc;
        s->center_off_h[i + 1] = s->center_off_h[i] + nc;
        if (s->has_mask) {
          int64_t t = a0;
          for (int64_t a = a0; a < a1; ++a)
            if (center_mask[a]) tag2idx[t++] = int32_t(a);
          for (int64_t a = a0; a < a1; ++a)
            if (!center_mask[a]) tag2idx[t++] = int32_t(a);
        }
      }
      std::vector<Upload> ups = {
          {&s->atom_off_d, s->atom_off.data(), sizeof(int64_t) * (n_structures + 1)},
          {&s->pos_d, positions, sizeof(double) * 3 * s->n_atoms},
          {&s->types_d, numbers, sizeof(int32_t) * s->n_atoms},
          {&s->cells_d, cells, sizeof(double) * 9 * n_structures},
          {&s->pbc_d, pbc, sizeof(int32_t) * 3 * n_structures},
          {&s->ncent_d, ncent.data(), sizeof(int32_t) * n_structures},
          {&s->center_off_d, s->center_off_h.data(), sizeof(int64_t) * (n_structures + 1)},
          {&s->atom_struct_d, astruct.data(), sizeof(int32_t) * s->n_atoms}};
      if (s->has_mask) ups.push_back({&s->tag2idx_d, tag2idx.data(), sizeof(int32_t) * s->n_atoms});
      upload_inputs(s, ups);
    } catch (...) {
      // the former inputs may be gone and the new ones are not there: the
      // handle is left without structures
      s->n_struct = 0;
      s->n_atoms = 0;
      s->atom_off.assign(1, 0);
      s->center_off_h.assign(1, 0);
      s->batch_species.clear();
      std::fill(s->centres_of_type, s->centres_of_type + 130, int64_t(0));
      throw;
    }
  });
}

rgpu_status rgpu_structures_update_positions(rgpu_structures * s, const double * positions) {
  return guard([&] {
    OnDevice on_dev(s);
    drop_results(s);
    upload_positions(s, positions);
  });
}

rgpu_status rgpu_structures_invalidate(rgpu_structures * s) {
  return guard([&] {
    OnDevice on_dev(s);
    drop_results(s);
  });
}

rgpu_status rgpu_structures_stream(const rgpu_structures * s, void ** stream) {
  return guard([&] {
    OnDevice on_dev(s);
    *stream = static_cast<void *>(s->st);
  });
}

rgpu_status rgpu_neighbour_list_build(rgpu_structures * s, double cutoff) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!(cutoff > 0)) throw Error(RGPU_ERR_INVALID_ARGUMENT, "cutoff must be > 0");
    build_nl(s, cutoff);
  });
}

rgpu_status rgpu_neighbour_list_size(const rgpu_structures * s, int64_t * n_centers, int64_t * n_pairs) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s->nl_valid) throw Error(RGPU_ERR_NOT_COMPUTED, "the neighbour list has not been built");
    *n_centers = s->nl.n_centers;
    *n_pairs = s->nl.n_pairs;
  });
}

rgpu_status rgpu_neighbour_list_get(const rgpu_structures * s, int32_t * center_atom, int64_t * pair_offsets,
                                    int32_t * j_atom, int32_t * shift, double * distance, double * direction) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s->nl_valid) throw Error(RGPU_ERR_NOT_COMPUTED, "the neighbour list has not been built");
    const int64_t nc = s->nl.n_centers, np = s->nl.n_pairs;
    auto get = [&](void * dst, const void * src, size_t bytes) {
      if (dst && bytes) RGPU_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s->st));
    };
    get(center_atom, s->nl.center_atom, sizeof(int32_t) * nc);
    get(pair_offsets, s->nl.pair_off, sizeof(int64_t) * (nc + 1));
    get(j_atom, s->nl.pair_j, sizeof(int32_t) * np);
    get(shift, s->nl.pair_shift, sizeof(int32_t) * 3 * np);
    get(distance, s->nl.pair_dist, sizeof(double) * np);
    get(direction, s->nl.pair_dir, sizeof(double) * 3 * np);
    RGPU_CUDA(cudaStreamSynchronize(s->st));
  });
}

rgpu_status rgpu_compute(rgpu_calculator * calc, rgpu_structures * s, int precision, int gradients) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!calc || !s) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    if (precision != RGPU_PRECISION_FP64 && precision != RGPU_PRECISION_FP32)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "unknown precision");
    bool g = gradients || calc->hy.compute_gradients;
    if (g && s->has_mask)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "Can't compute spherical expansion gradients with masked center atoms",
                  RGPU_EXC_LOGIC_ERROR);
    calculator_to_device(calc);
    s->timed = false;
    compute_features(calc, s, precision, g, {});
    RGPU_CUDA(cudaStreamSynchronize(s->st));
  });
}

rgpu_status rgpu_get_species(const rgpu_structures * s, int32_t * n_species, int32_t * species) {
  return guard([&] {
    OnDevice on_dev(s);
    *n_species = int32_t(s->species.size());
    for (size_t i = 0; i < s->species.size(); ++i) species[i] = s->species[i];
  });
}

rgpu_status rgpu_get_feature_keys(const rgpu_calculator * calc, const rgpu_structures * s, int32_t * n_keys,
                                  int32_t * keys) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s->feat_valid || s->feat_calc != serial_of(calc)) throw Error(RGPU_ERR_NOT_COMPUTED, "features have not been computed");
    auto k = present_keys(calc, s);
    *n_keys = int32_t(k.size());
    if (keys)
      for (size_t i = 0; i < k.size(); ++i) {
        keys[2 * i] = k[i].first;
        keys[2 * i + 1] = k[i].second;
      }
  });
}

rgpu_status rgpu_get_features(const rgpu_calculator * calc, const rgpu_structures * s, int32_t n_keys,
                              const int32_t * keys, double * out) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s->feat_valid || s->feat_calc != serial_of(calc)) throw Error(RGPU_ERR_NOT_COMPUTED, "features have not been computed");
    const FeatureDims & fd = s->fd;
    const int64_t nc = s->nl.n_centers;
    const bool ps = calc->hy.kind == "sphericalinvariants";
    const int64_t row = int64_t(n_keys) * (ps ? fd.n * fd.n * (fd.L + 1) : fd.nK);
    if (nc == 0 || row == 0) return;
    if (ps && s->feat_precision != RGPU_PRECISION_FP64 && !s->feat_x32)
      throw Error(RGPU_ERR_NOT_COMPUTED, "the last FP32 prediction kept no features to export");
    // selected and rearranged on the device, then straight into the caller's
    // array, a bounded number of rows at a time
    const std::vector<int> blocks = key_blocks(calc, s, n_keys, keys);
    DevBuf & buf = const_cast<rgpu_structures *>(s)->export_d;
    const int64_t rows = std::min<int64_t>(nc, std::max<int64_t>(1, (int64_t(256) << 20) / int64_t(sizeof(double)) / row));
    const size_t head = (sizeof(int32_t) * size_t(n_keys) + 255) & ~size_t(255);
    buf.ensure(head + sizeof(double) * size_t(rows) * row);
    RGPU_CUDA(cudaMemcpyAsync(buf.p, blocks.data(), sizeof(int32_t) * n_keys, cudaMemcpyHostToDevice, s->st));
    FeatureExport a;
    a.fd = fd;
    a.power_spectrum = ps;
    a.fp64 = s->feat_precision == RGPU_PRECISION_FP64;
    a.src = a.fp64 ? (ps ? s->X64.p : s->C64.p) : (ps ? s->X32.p : s->C32.p);
    a.row_of_center = s->row_of_center.as<int32_t>();
    a.row_scale = s->xscale32.as<float>();
    a.blocks = buf.as<int32_t>();
    a.n_keys = n_keys;
    a.out = reinterpret_cast<double *>(buf.as<unsigned char>() + head);
    for (a.c0 = 0; a.c0 < nc; a.c0 = a.c1) {
      a.c1 = std::min(nc, a.c0 + rows);
      launch_feature_export(a, s->st);
      RGPU_CUDA(cudaMemcpyAsync(out + a.c0 * row, a.out, sizeof(double) * size_t(a.c1 - a.c0) * row,
                                cudaMemcpyDeviceToHost, s->st));
    }
    RGPU_CUDA(cudaStreamSynchronize(s->st));
  });
}

rgpu_status rgpu_get_features_gradient(const rgpu_calculator * calc, const rgpu_structures * s_in, int32_t n_keys,
                                       const int32_t * keys, double * out) {
  return guard([&] {
    OnDevice on_dev(s_in);
    rgpu_structures * s = const_cast<rgpu_structures *>(s_in);
    if (!s->feat_valid || s->feat_calc != serial_of(calc)) throw Error(RGPU_ERR_NOT_COMPUTED, "features have not been computed");
    if (!s->feat_gradients) throw Error(RGPU_ERR_NOT_COMPUTED, "gradients were not requested (compute_gradients)");
    if (s->feat_precision != RGPU_PRECISION_FP64)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "dense gradients are exported from the FP64 path");
    const FeatureDims & fd = s->fd;
    const int64_t nc = s->nl.n_centers;
    auto blocks = key_blocks(calc, s, n_keys, keys);
    if (calc->hy.kind == "sphericalexpansion") {
      export_expansion_gradient(calc, s, n_keys, blocks, out);
      return;
    }
    const int inner = fd.n * fd.n * (fd.L + 1);
    ExpansionArgs ea = exp_args(calc, s);
    PsArgs pa;
    pa.fd = fd;
    pa.n_centers = nc;
    pa.normalize = calc->hy.normalize;
    pa.row_of_center = s->row_of_center.as<int32_t>();
    const size_t per_pair = sizeof(double) * (3 * size_t(fd.D) + 3 * size_t(fd.nK));
    const size_t per_center = sizeof(double) * size_t(fd.S) * 3 * fd.nK;
    const size_t budget = size_t(4) << 30;
    std::vector<double> host;
    const std::vector<int64_t> & poff = pair_offsets_host(s);
    int64_t c0 = 0;
    while (c0 < nc) {
      int64_t c1 = c0;
      size_t bytes = 0;
      while (c1 < nc) {
        size_t add = per_pair * size_t(poff[c1 + 1] - poff[c1]) + per_center;
        if (c1 > c0 && bytes + add > budget) break;
        bytes += add;
        ++c1;
      }
      const int64_t p_base = poff[c0];
      const int64_t np = poff[c1] - p_base;
      s->dCp.ensure(sizeof(double) * size_t(np) * 3 * fd.nK + 64);
      s->dCs.ensure(per_center * size_t(c1 - c0) + 64);
      s->dXp.ensure(sizeof(double) * size_t(np) * 3 * fd.D + 64);
      launch_expansion_grad_fp64(ea, c0, c1, p_base, s->dCp.as<double>(), s->st);
      launch_expansion_selfgrad_fp64(ea, c0, c1, p_base, s->dCp.as<double>(), s->dCs.as<double>(), s->st);
      launch_ps_grad_fp64(pa, ea, c0, c1, p_base, s->C64.as<double>(), s->X64.as<double>(), s->invn64.as<double>(),
                          s->dCp.as<double>(), s->dCs.as<double>(), s->dXp.as<double>(), s->st);
      host.resize(size_t(np) * 3 * fd.D);
      RGPU_CUDA(cudaMemcpyAsync(host.data(), s->dXp.p, sizeof(double) * host.size(), cudaMemcpyDeviceToHost, s->st));
      RGPU_CUDA(cudaStreamSynchronize(s->st));
      for (int64_t p = 0; p < np; ++p)
        for (int c = 0; c < 3; ++c) {
          const double * src = &host[(size_t(p) * 3 + c) * fd.D];
          double * dst = out + (size_t(p_base + p) * 3 + c) * size_t(n_keys) * inner;
          for (int k = 0; k < n_keys; ++k) {
            if (blocks[k] < 0)
              std::memset(dst + size_t(k) * inner, 0, sizeof(double) * inner);
            else
              std::memcpy(dst + size_t(k) * inner, src + size_t(blocks[k]) * inner, sizeof(double) * inner);
          }
        }
      c0 = c1;
    }
  });
}

rgpu_status rgpu_gap_model_create(rgpu_calculator * calc, int32_t n_species, const int32_t * species,
                                  int32_t n_sparse, const int32_t * sparse_species, const double * T,
                                  const double * weights, int32_t zeta, const double * self_contributions,
                                  rgpu_gap_model ** out) {
  return guard([&] {
    if (!calc || !out || n_species <= 0 || n_sparse < 0) throw Error(RGPU_ERR_INVALID_ARGUMENT, "bad arguments");
    if (calc->hy.kind != "sphericalinvariants")
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "the GAP model needs a SphericalInvariants calculator");
    if (zeta < 1) throw Error(RGPU_ERR_INVALID_ARGUMENT, "zeta must be >= 1");
    auto m = std::make_unique<rgpu_gap_model>();
    m->calc = calc;
    m->species.assign(species, species + n_species);
    if (!std::is_sorted(m->species.begin(), m->species.end()))
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "model species must be sorted");
    m->M = n_sparse;
    m->sp_species.assign(sparse_species, sparse_species + n_sparse);
    for (int sp : m->sp_species)
      if (!std::binary_search(m->species.begin(), m->species.end(), sp))
        throw Error(RGPU_ERR_INVALID_ARGUMENT, "sparse point species missing from the model species");
    FeatureDims fm = make_dims(calc->hy, n_species);
    m->T.assign(T, T + size_t(n_sparse) * fm.D);
    if (weights)
      m->alpha.assign(weights, weights + n_sparse);
    else
      m->alpha.assign(size_t(n_sparse), 0.);  // kernel matrices only
    m->zeta = zeta;
    m->self_contrib.assign(n_species, 0.);
    if (self_contributions) m->self_contrib.assign(self_contributions, self_contributions + n_species);
    *out = m.release();
  });
}

rgpu_status rgpu_gap_model_destroy(rgpu_gap_model * m) {
  return guard([&] { delete m; });
}

rgpu_status rgpu_gap_predict(rgpu_gap_model * m, rgpu_structures * s, int precision, double * energies,
                             double * forces) {
  return guard([&] {
    OnDevice on_dev(s);
    gap_predict_entry(m, s, precision, energies, forces, nullptr);
  });
}

rgpu_status rgpu_gap_predict_stress(rgpu_gap_model * m, rgpu_structures * s, int precision, double * energies,
                                    double * forces, double * neg_stress) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!neg_stress) throw Error(RGPU_ERR_INVALID_ARGUMENT, "neg_stress output is required");
    gap_predict_entry(m, s, precision, energies, forces, neg_stress);
  });
}

rgpu_status rgpu_gap_forward_dev(rgpu_gap_model * m, rgpu_structures * s, const double * positions_dev,
                                 double * energies_dev) {
  return guard([&] {
    OnDevice on_dev(s);
    gap_forward_dev_impl(m, s, positions_dev, energies_dev);
  });
}

rgpu_status rgpu_gap_backward_dev(rgpu_gap_model * m, rgpu_structures * s, const double * energies_grad_dev,
                                  double * grad_dev) {
  return guard([&] {
    OnDevice on_dev(s);
    gap_backward_dev_impl(m, s, energies_grad_dev, grad_dev);
  });
}

rgpu_status rgpu_md_step(rgpu_gap_model * m, rgpu_structures * s, const double * positions, double * energies,
                         double * forces, double * neg_stress) {
  return guard([&] {
    OnDevice on_dev(s);
    md_step_impl(m, s, positions, energies, forces, neg_stress);
  });
}

rgpu_status rgpu_md_step_info(const rgpu_structures * s, int32_t * recorded, int64_t * info) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s || !recorded) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    *recorded = s->md_exec ? 1 : 0;
    if (info) {
      info[0] = s->md_caps.sites;
      info[1] = s->md_caps.boxes;
      info[2] = s->md_caps.pairs;
      info[3] = s->md_replays;
      info[4] = s->md_reason;
      info[5] = s->md_kernels;
    }
  });
}

rgpu_status rgpu_sparse_kernel(rgpu_gap_model * m, rgpu_structures * s, int32_t target_atom, double * out) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!out) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    sparse_kernel_impl(m, s, target_atom != 0, out);
  });
}

rgpu_status rgpu_sparse_kernel_derivative(rgpu_gap_model * m, rgpu_structures * s, int32_t neg_stress,
                                          double * out) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!out) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    sparse_kernel_derivative_impl(m, s, neg_stress != 0, out);
  });
}

rgpu_status rgpu_sparse_kernel_mm(rgpu_gap_model * m, double * out) {
  return guard([&] {
    if (!out) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    sparse_kernel_mm_impl(m, out);
  });
}

namespace {
__global__ void bf16_pair_to_f32_kernel(const __nv_bfloat16 * hi, const __nv_bfloat16 * lo, int64_t rows,
                                        int64_t cols, int64_t ld, float * out) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  int64_t r = i / cols, c = i - r * cols;
  out[i] = __bfloat162float(hi[r * ld + c]) + __bfloat162float(lo[r * ld + c]);
}
__global__ void sum_parts_kernel(const float * parts, int n_parts, int64_t M, float * e) {
  int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= M) return;
  float s = 0.f;
  for (int t = 0; t < n_parts; ++t) s += parts[int64_t(t) * M + r];
  e[r] = s;
}
}  // namespace

// Scratch of the GEMM test hook, one set per device (the hook is called
// from one host thread at a time).
struct DebugGemmBuffers {
  DevBuf ah, al, bh, bl, wh, wl, parts;
};
static PerDevice<DebugGemmBuffers> g_debug_gemm_buffers;

rgpu_status rgpu_debug_set_gemm_wait_limit(int64_t polls) {
  return guard([&] { set_gemm_wait_limit(polls); });
}

rgpu_status rgpu_debug_packed_layout(int32_t S, int32_t max_radial, int32_t max_angular, int64_t * D, int64_t * Dg,
                                     const double * ref, double * packed, double * unpacked) {
  return guard([&] {
    if (S < 1 || S > kMaxSpecies || max_radial < 1 || max_angular < 0 || max_angular > kMaxL)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "bad layout shape");
    Hypers hy;
    hy.max_radial = max_radial;
    hy.max_angular = max_angular;
    const FeatureDims fd = make_dims(hy, S);
    if (D) *D = fd.D;
    if (Dg) *Dg = fd.Dg;
    if (!ref) return;
    std::vector<double> pk(fd.Dg);
    pack_reference_row(fd, ref, pk.data());
    if (packed) std::copy(pk.begin(), pk.end(), packed);
    if (unpacked) {
      std::vector<float> pf(pk.begin(), pk.end());
      unpack_to_reference(fd, pf.data(), 1.f, unpacked);
    }
  });
}

rgpu_status rgpu_debug_gemm_bf16x3(int mode, int64_t M, int64_t N, int64_t K, const float * A, const float * B,
                                   const float * alpha, int32_t zeta, float * C, float * e, void * stream) {
  return guard([&] {
    if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C) throw Error(RGPU_ERR_INVALID_ARGUMENT, "bad GEMM arguments");
    if (mode == 0 && N % 4 != 0) throw Error(RGPU_ERR_INVALID_ARGUMENT, "N must be a multiple of 4");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    DebugGemmBuffers & B_ = g_debug_gemm_buffers.at(current_device());
    DevBuf &ah = B_.ah, &al = B_.al, &bh = B_.bh, &bl = B_.bl, &wh = B_.wh, &wl = B_.wl, &parts = B_.parts;
    const int64_t Kp = (K + 63) / 64 * 64, Np = (N + 31) / 32 * 32;
    ah.ensure(2 * size_t(M) * Kp);
    al.ensure(2 * size_t(M) * Kp);
    bh.ensure(2 * size_t(N) * Kp);
    bl.ensure(2 * size_t(N) * Kp);
    split_bf16(A, M, K, K, ah.as<__nv_bfloat16>(), al.as<__nv_bfloat16>(), Kp, st);
    split_bf16(B, N, K, K, bh.as<__nv_bfloat16>(), bl.as<__nv_bfloat16>(), Kp, st);
    Bf16x3Gemm g{};
    g.M = M;
    g.N = N;
    g.K = Kp;
    g.A_hi = ah.as<__nv_bfloat16>();
    g.A_lo = al.as<__nv_bfloat16>();
    g.lda = Kp;
    g.B_hi = bh.as<__nv_bfloat16>();
    g.B_lo = bl.as<__nv_bfloat16>();
    g.ldb = Kp;
    g.epilogue = mode;
    if (mode == 0) {
      g.C = C;
      g.ldc = N;
      gemm_bf16x3(g, st);
    } else {
      const int n_parts = int((N + kTcTileN - 1) / kTcTileN);
      wh.ensure(2 * size_t(M) * Np);
      wl.ensure(2 * size_t(M) * Np);
      parts.ensure(sizeof(float) * size_t(n_parts) * M);
      g.W_hi = wh.as<__nv_bfloat16>();
      g.W_lo = wl.as<__nv_bfloat16>();
      g.ldw = Np;
      g.alpha = alpha;
      g.zeta = zeta;
      g.e_part = parts.as<float>();
      gemm_bf16x3(g, st);
      bf16_pair_to_f32_kernel<<<div_up(M * N, 256), 256, 0, st>>>(g.W_hi, g.W_lo, M, N, Np, C);
      if (e) sum_parts_kernel<<<div_up(M, 256), 256, 0, st>>>(parts.as<float>(), n_parts, M, e);
    }
    RGPU_CUDA(cudaStreamSynchronize(st));
    const int where = gemm_tc_timeout(true);
    if (where) throw Error(RGPU_ERR_TIMEOUT, "tensor-core GEMM wait gave up at stage " + std::to_string(where));
  });
}

rgpu_status rgpu_gap_energies_noalloc(int64_t M, int64_t N, int64_t K, const float * A, const float * B,
                                      const float * alpha, int32_t zeta, float * e, void * stream) {
  return guard([&] { gap_energies_noalloc(M, N, K, A, B, alpha, zeta, e, static_cast<cudaStream_t>(stream)); });
}

rgpu_status rgpu_set_tile_config(int32_t n_species, int32_t max_radial, int32_t max_angular, const int32_t * values,
                                 int32_t n_values) {
  return guard([&] {
    if (n_values == 0) {
      set_tile_config(n_species, max_radial, max_angular, nullptr);
      return;
    }
    if (n_values != kTileFields || !values)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "tile config: " + std::to_string(kTileFields) + " values expected");
    const TileConfig c = tile_config_from_array(values);
    set_tile_config(n_species, max_radial, max_angular, &c);
  });
}

rgpu_status rgpu_get_tile_config(int32_t n_species, int32_t max_radial, int32_t max_angular, int32_t * values) {
  return guard([&] {
    if (!values) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    tile_config_to_array(tile_config(n_species, max_radial, max_angular), values);
  });
}

rgpu_status rgpu_structures_use_graphs(rgpu_structures * s, int enable) {
  return guard([&] {
    OnDevice on_dev(s);
    if (!s) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    s->use_graphs = enable != 0;
    if (!s->use_graphs) {
      RGPU_CUDA(cudaStreamSynchronize(s->st));
      for (PredictBucket & b : s->pbuckets) pbucket_release(b);
      s->pbuckets.clear();
    }
  });
}

rgpu_status rgpu_structures_graph_info(const rgpu_structures * s, int64_t * info) {
  return guard([&] {
    if (!s || !info) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    info[0] = 0;
    for (const PredictBucket & b : s->pbuckets) info[0] += (b.full.exec ? 1 : 0) + (b.alone.exec ? 1 : 0);
    info[1] = s->pgraph_replays;
    info[2] = s->pgraph_records;
    info[3] = s->pgraph_last_kernels;
  });
}

rgpu_status rgpu_measure_fma_peak(int precision, double * tflops) {
  return guard([&] {
    if (!tflops) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    if (precision != RGPU_PRECISION_FP64 && precision != RGPU_PRECISION_FP32)
      throw Error(RGPU_ERR_INVALID_ARGUMENT, "unknown precision");
    *tflops = measure_fma_peak(precision);
  });
}

rgpu_status rgpu_measure_fp64_tensor_peak(double * tflops) {
  return guard([&] {
    if (!tflops) throw Error(RGPU_ERR_INVALID_ARGUMENT, "null argument");
    *tflops = measure_fp64_tensor_peak();
  });
}

rgpu_status rgpu_synchronize(rgpu_structures * s) {
  return guard([&] {
    OnDevice on_dev(s);
    RGPU_CUDA(cudaStreamSynchronize(s->st));
  });
}

int64_t rgpu_kernel_launches(int reset) { return rgpu::launches(reset != 0); }

rgpu_status rgpu_stage_times(const rgpu_structures * s, double * ms_out, int32_t n_stages) {
  return guard([&] {
    OnDevice on_dev(s);
    RGPU_CUDA(cudaStreamSynchronize(s->st));
    // 0 whole call, 1 neighbour list, 2 expansion, 3 power spectrum,
    // 4 forward GEMMs, 5 backward GEMMs, 6 power-spectrum backward (plain:
    // gradient chunks), 7 pair adjoint
    const int pairs[8][2] = {{0, 8}, {0, 1}, {2, 3}, {3, 4}, {4, 5}, {5, 6}, {6, 7}, {7, 8}};
    for (int i = 0; i < n_stages && i < 8; ++i) {
      float ms = 0.f;
      cudaError_t e = cudaEventElapsedTime(&ms, s->ev[pairs[i][0]], s->ev[pairs[i][1]]);
      ms_out[i] = (e == cudaSuccess) ? ms : -1.0;
    }
  });
}

}  // extern "C"
