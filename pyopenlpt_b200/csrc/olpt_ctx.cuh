// Host-side context shared by all translation units of libolpt_cuda.so.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/olpt.h"
#include "olpt_device.cuh"
#include "olpt_mlp.h"
#include "olpt_prof.h"
#include "olpt_shake.h"
#include "olpt_stb.h"
#include "olpt_stereo.h"
#include "olpt_trackio.h"

namespace olpt {

// Number of kernel launches issued by this library (every launch site wraps its
// grid expression in OLPT_G, which is evaluated exactly once per launch).
extern std::atomic<long long> g_launches;
#define OLPT_G(grid) (::olpt::g_launches.fetch_add(1, std::memory_order_relaxed), (grid))

struct CudaError {
  cudaError_t code;
  std::string where;
};
struct ApiError {
  olpt_status_t code;
  std::string msg;
};

#define OLPT_CUDA(call)                                                             \
  do {                                                                              \
    cudaError_t _e = (call);                                                        \
    if (_e != cudaSuccess) throw ::olpt::CudaError{_e, std::string(#call) + " @ " + \
                                                       __FILE__ + ":" + std::to_string(__LINE__)}; \
  } while (0)

#define OLPT_REQUIRE(cond, code, msg) \
  do {                                \
    if (!(cond)) throw ::olpt::ApiError{(code), (msg)}; \
  } while (0)

// Dynamic shared memory that the current device grants Kernel, raised to at least `bytes`.  The
// limit belongs to the kernel on the device, not to a context: one that another context's
// thread lowered between this call and the launch would refuse the launch, so it only rises.
template <auto Kernel>
void allow_smem(size_t bytes) {
  static std::mutex mu;
  static size_t set[64] = {};
  int dev = 0;
  OLPT_CUDA(cudaGetDevice(&dev));
  OLPT_REQUIRE(dev >= 0 && dev < 64, OLPT_ERR_INVALID_ARG, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(mu);
  if (bytes <= set[dev]) return;
  OLPT_CUDA(cudaFuncSetAttribute((const void*)Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)bytes));
  set[dev] = bytes;
}

// Grow-only device buffer (stream-ordered allocation).
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  void ensure(size_t need, cudaStream_t s) {
    if (need <= bytes) return;
    if (p) OLPT_CUDA(cudaFreeAsync(p, s));
    size_t nb = need + need / 4 + 256;
    OLPT_CUDA(cudaMallocAsync(&p, nb, s));
    bytes = nb;
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
  void release(cudaStream_t s) {
    if (p) cudaFreeAsync(p, s);
    p = nullptr;
    bytes = 0;
  }
};

// Pinned host staging buffer.
struct HostBuf {
  void* p = nullptr;
  size_t bytes = 0;
  void ensure(size_t need) {
    if (need <= bytes) return;
    if (p) cudaFreeHost(p);
    size_t nb = need + need / 4 + 256;
    OLPT_CUDA(cudaMallocHost(&p, nb));
    bytes = nb;
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
  ~HostBuf() {
    if (p) cudaFreeHost(p);
  }
};

// One camera image plane in HBM (row pitch padded to 16 bytes for vector loads).
struct ImagePlane {
  DevBuf buf;
  int dtype = OLPT_U8;
  int H = 0, W = 0;
  int64_t pitch = 0;  // bytes
};

struct OtfDev {
  int nx = 2, ny = 2, nz = 2, n_grid = 8;
  double bmin[3], bmax[3];
  double d[3];  // grid spacing
  int alpha_zero = 0;       // every alpha entry is +0.0 (cos = 1, sin = +0 exactly)
};

// Per-camera 2D detection list (SoA, FP64 like the reference's Pt2D).
struct Dets {
  DevBuf x, y, rc;          // rc: packed (row<<16 | col) is not enough for 2048+; store int2
  int64_t cap = 0;
};

// CSR (start[n_buckets + 1], items[n]) from per-item bucket keys (key < 0: dropped);
// built by count -> exclusive scan -> scatter (scan.cu); items of a bucket in any order.
struct Csr {
  DevBuf start, items, cursor, tmp;
  void build(const int* key, int n, int n_buckets, cudaStream_t s);
  void release(cudaStream_t s) {
    start.release(s);
    items.release(s);
    cursor.release(s);
    tmp.release(s);
  }
};

// Device workspace of the shake (grown on demand).
struct ShakeWork {
  DevBuf otfp;      // n x n_cam x 5 OTF parameters at the object centres
  DevBuf proj;      // projection planes of all cameras, zero between passes
  bool proj_clean = false;
  int proj_esz = 0;
  int64_t proj_bytes = 0;
  const void* proj_at = nullptr;
  DevBuf rep, hkey, has_nb, nb_pos, nb_list, scan_tmp, gpart;
  Csr hash;         // 3D hash grid of object centres
  void release(cudaStream_t s) {
    nb_pos.release(s);
    nb_list.release(s);
    scan_tmp.release(s);
    otfp.release(s);
    proj.release(s);
    proj_clean = false;
    rep.release(s);
    hkey.release(s);
    has_nb.release(s);
    gpart.release(s);
    hash.release(s);
  }
};

// Device workspace of stereo matching (grown on demand, reused across frames).
struct StereoWork {
  DevBuf cell_start, cell_cnt, cell_of, pid, xy, fxy, los, l2d, fl;
  DevBuf counters, scan_tmp;
  DevBuf path_a, path_b, term, pairs;
  DevBuf cand_ids, cand_e, cand_x;
  // near-tolerance decision log: records (olpt_near_record) and a 64-bit counter of
  // every near-tolerance test seen since the last reset (records beyond near_cap are
  // counted, not stored)
  DevBuf near_rec, near_count;
  double near_band = 0.0;
  int64_t near_cap = 0;
  void release(cudaStream_t s) {
    near_rec.release(s);
    near_count.release(s);
    for (DevBuf* b : {&cell_start, &cell_cnt, &cell_of, &pid, &xy, &fxy, &los, &l2d, &fl, &scan_tmp})
      b->release(s);
    counters.release(s);
    path_a.release(s);
    path_b.release(s);
    term.release(s);
    pairs.release(s);
    cand_ids.release(s);
    cand_e.release(s);
    cand_x.release(s);
  }
};

// Per camera: active flag, detection count and offset of its first detection in the
// global point numbering of the prune.
struct PruneView {
  int active[OLPT_MAX_CAM];
  int count[OLPT_MAX_CAM];
  int offset[OLPT_MAX_CAM];
};

// Device workspace of the candidate sort and prune (prune.cu).
struct PruneWork {
  DevBuf key, val, key2, val2, hist, hist2, scan_tmp;
  DevBuf ids_s, e_s, X_s;
  DevBuf fl, slot_key, fcnt, slot_pct, slot_used, pct;
  DevBuf counts;  // PruneCount words (prune.cu)
  DevBuf pcls, ecls, cstart, tiles, mixed;
  DevBuf g_pts, g_cnt, g_pct, g_e, pool_e, pool_i;
  DevBuf gstate, gfirst, gowner, sel, spos, scnt;
  Csr points;
  int n_sel = 0;  // kept candidates of the last device prune
  int cluster = -1;  // the device runs clusters of 16 sort blocks (-1: not asked yet)
  HostBuf pin;    // pinned staging of the sequential greedy's input
  void release(cudaStream_t s) {
    for (DevBuf* b : {&key, &val, &key2, &val2, &hist, &hist2, &scan_tmp, &ids_s, &e_s, &X_s, &fl,
                      &slot_key, &fcnt, &slot_pct, &slot_used, &pct, &counts, &pcls, &ecls,
                      &cstart, &tiles, &mixed, &g_pts, &g_cnt, &g_pct, &g_e, &pool_e, &pool_i,
                      &gstate, &gfirst, &gowner, &sel, &spos, &scnt})
      b->release(s);
    points.release(s);
  }
};

// 3D objects resident on the device (SoA).
struct Objects {
  DevBuf xyz;    // n x 3 double
  DevBuf uv;     // n x n_cam x 2 double: current 2D projections
  DevBuf flags;  // n uint8 (ObjFlag bits)
  DevBuf score;  // n double
  int64_t n = 0;
  void ensure(int64_t cap, int n_cam, cudaStream_t s) {
    xyz.ensure((cap + 1) * 3 * sizeof(double), s);
    uv.ensure((cap + 1) * n_cam * 2 * sizeof(double), s);
    flags.ensure(cap + 16, s);
    score.ensure((cap + 1) * sizeof(double), s);
  }
  void release(cudaStream_t s) {
    xyz.release(s);
    uv.release(s);
    flags.release(s);
    score.release(s);
  }
};

// IPR knobs (IPRParam + tracer threshold, inc/libSTB/Config.h:37-44, 190-195).
struct IprParams {
  double min_obj_int;
  SmParams sm;
  ShakeParams shake;
  int n_cam_reduced, n_loop_ipr, n_loop_ipr_reduced;
  int64_t n_obj2d_process_max;
};

// IPR workspace and the accumulated output objects of the last run.
struct IprWork {
  DevBuf perm, tx, ty, trc, keep, pos, scan_tmp;
  DevBuf out_xyz, out_uv;
  int64_t n_out = 0, cap_out = 0;
  void release(cudaStream_t s) {
    perm.release(s);
    tx.release(s);
    ty.release(s);
    trc.release(s);
    keep.release(s);
    pos.release(s);
    scan_tmp.release(s);
    out_xyz.release(s);
    out_uv.release(s);
    n_out = cap_out = 0;
  }
};

void stereo_match_device(olpt_ctx* ctx, const SmParams& prm, StereoResult& res);
bool prune_select_device(olpt_ctx* ctx, const PruneView& pv, int M, int n_cam,
                         int64_t total_points, char* selected);
// Download a device-resident stereo result (no-op for a host one).
void stereo_result_to_host(olpt_ctx* ctx, StereoResult& r);
// the selected candidates of a result that is on the device, read back to the host
void stereo_matches(olpt_ctx* ctx, const StereoResult& r, int* ids, double* xyz);
// The kept matches become the context's 3D objects (triangulateMatch order); returns
// their number.
int64_t stereo_objects(olpt_ctx* ctx, const StereoResult& r);
void ipr_device(olpt_ctx* ctx, const IprParams& p);
OtfView otf_view(olpt_ctx* ctx);
void shake_device(olpt_ctx* ctx, const ShakeParams& sp);
void residual_device(olpt_ctx* ctx, const ShakeParams& sp, bool use_flags, bool make_current);

// Track files (trackio.cu): device buffers of the row formatter and the writer thread.
// async: the frame loop's track files are written while later frames run (flush_files
// waits for them); otherwise every save returns after its file is written.
constexpr int64_t kMaxRowsPerPass = 1 << 20;
struct TrackIoWork {
  DevBuf ints, xyz, uv, len, off, bad, bytes, tmp;
  bool async = false;
  FileWriter writer;
  void release(cudaStream_t s) {
    for (DevBuf* x : {&ints, &xyz, &uv, &len, &off, &bad, &bytes, &tmp}) x->release(s);
  }
};
// rows of n_int ints, then n1 + n2 doubles from two arrays (device), "%.6f" numbers,
// comma separated, one per line; n <= kMaxRowsPerPass; appended to out
void format_rows_device(olpt_ctx* ctx, const int* ints, int n_int, const double* d1, int n1,
                        const double* d2, int n2, int64_t n, std::string& out);
// bytes -> file on the writer thread (waits for it unless the context writes async)
void write_file(olpt_ctx* ctx, const std::string& file, std::string&& bytes);
// waits for every posted file; throws the first write error
void flush_files(olpt_ctx* ctx);
// OTF estimation from the context's planes (otf_est.cu); false: an image without detections
bool otf_estimate_device(olpt_ctx* ctx, double min_int, double r_pt, int max_det, double abc[3],
                         int64_t* n_samples);

// Device workspace of the STB frame loop (grown on demand, reused across frames).
struct StbWork {
  DevBuf a, b, c, d, ia, link, flag, field, field2, kern, k1, k2;
  Csr g1, g2;
  void release(cudaStream_t s) {
    for (DevBuf* x : {&a, &b, &c, &d, &ia, &link, &flag, &field, &field2, &kern, &k1, &k2})
      x->release(s);
    g1.release(s);
    g2.release(s);
  }
};

// STB state (STB members, inc/libSTB/STB.h:58-70): the four track lists and the
// initial-phase IPR results.
struct StbState {
  StbParams p;
  IprParams ipr;
  bool configured = false;
  TrackList short_active, long_active, long_inactive, exited;
  // capacity kept for the frame loop's temporary lists: one spare per role, so that the
  // long-track and short-track buffers each circulate between their list and its spare
  TrackList spare_long, spare_short;
  std::vector<std::vector<double>> ipr_xyz;   // initial phase, per frame
  std::vector<std::vector<char>> ipr_tracked;
  std::vector<double> linfit_kernel;          // 2 x n_pts
  int64_t last_new = 0, last_extended = 0;
  std::vector<double> last_xyz;               // particles of the last frame
  ImagePlane frame_img[OLPT_MAX_CAM];         // the frame's images as processFrame leaves them
  StbWork w;
};

// Device state of the learned proposal (mlp.cu): f32 master parameters, Adam moments
// and gradients (flat, MlpDims::params), bf16 weight copies for the GEMMs (row-major and
// transposed), and the activations of one batch.
struct MlpWork {
  bool ready = false;
  MlpDims dims = mlp_dims(4);  // network geometry (set from the camera count at init)
  int adam_t = 0;
  LearnedParams lp;
  int64_t n_learned = 0, n_fallback = 0;  // objects through the learned shake / its fallback
  int64_t cap = 0;  // batch capacity of the activation buffers
  DevBuf master, grad, am, av, wb1, wb2, wb3, wt2, wt3;
  DevBuf x, xt, xin, tgt, z1, z2, z3, h1, h2, h3, h1t, h2t, o, dout;
  DevBuf dz2b, dz3b, dz1t, dz2t, dz3t, part, hpart, loss, err;
  // learned shake: keep[i] = 1 for the input objects the network did not drop (the
  // objects left are the kept ones in input order), pos = their exclusive scan; fb =
  // fallback counter
  DevBuf keep, pos, start_xyz, act, nres, ds_x, ds_t, loss_hist, fb;
  void release(cudaStream_t s) {
    for (DevBuf* b : {&master, &grad, &am, &av, &wb1, &wb2, &wb3, &wt2, &wt3, &x, &xt, &xin, &tgt,
                      &z1, &z2, &z3, &h1, &h2, &h3, &h1t, &h2t, &o, &dout, 
                      &dz2b, &dz3b, &dz1t, &dz2t, &dz3t, &part, &hpart, &loss, &err, &keep, &pos,
                      &start_xyz, &act, &nres, &ds_x, &ds_t, &loss_hist, &fb})
      b->release(s);
    ready = false;
    cap = 0;
  }
};

// mlp.cu
// the network geometry of the context's camera count, unless a network is set
void mlp_sync_dims(olpt_ctx* ctx);
void mlp_init(olpt_ctx* ctx, uint64_t seed);
void mlp_set_params(olpt_ctx* ctx, const float* host);
void mlp_get_params(olpt_ctx* ctx, float* host);
// features of the context's objects against residual planes computed with all of
// them (FP32 or FP64 planes per sp.precision); x: n x dims.in_pad bf16 (device),
// f32 (optional, device): n x dims.in
void mlp_features_device(olpt_ctx* ctx, const ShakeParams& sp, __nv_bfloat16* x, float* f32);
void gelu_inplace_device(float* p, int64_t n, cudaStream_t s);
// residual planes of the current images with every object projected (the first step
// of a shake iteration)
void residual_all_device(olpt_ctx* ctx, const ShakeParams& sp);
// o (device, n x 4) = network(x), for f32 rows of dims.in or bf16 rows of dims.in_pad (device;
// the other one null); waits for the result
void mlp_infer_device(olpt_ctx* ctx, const float* x_f32, const __nv_bfloat16* x, int64_t n,
                      float* o);
// the same enqueued in one kernel (mlp_fused.cu); MlpWork::err reports a timed-out wait
void mlp_fused_forward(olpt_ctx* ctx, const float* x_f32, const __nv_bfloat16* x, int64_t n,
                       float* o);
// one training batch: loss (mean), gradients into MlpWork::grad, Adam update when lr > 0
double mlp_train_device(olpt_ctx* ctx, const float* x_f32, const float* tgt, int64_t n, double lr,
                        double ghost_weight, bool update);
// steps Adam steps on uniform mini-batches of a device-resident dataset (cosine
// learning-rate decay to 5%); losses (host, optional) per step
void mlp_train_many(olpt_ctx* ctx, const float* x, const float* t, int64_t n, int batch, int steps,
                    double lr, double ghost_weight, uint64_t seed, float* losses);
// the learned shake: features -> network -> correction and ghost pruning -> short
// plain refinement -> full plain shake for objects whose residue stays high
void learned_shake_device(olpt_ctx* ctx, const ShakeParams& sp);

void stb_configure(olpt_ctx* ctx, const StbParams& p, const IprParams& ipr);
void stb_process_frame(olpt_ctx* ctx, int frame);
TrackList& stb_list(olpt_ctx* ctx, int which);
void stb_save_tracks(olpt_ctx* ctx, int which, const std::string& path);
void stb_load_tracks(olpt_ctx* ctx, int which, const std::string& path);

}  // namespace olpt

struct olpt_ctx {
  int device = 0;
  // launch shapes chosen by olpt_autotune_ipr (they never change results)
  olpt_tuning tune{4, 256, 64};
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;

  int n_cam = 0;
  std::vector<olpt::CamDev> cams_h;
  olpt::DevBuf cams_d;

  olpt::OtfDev otf;
  olpt::DevBuf otf_table;

  olpt::ImagePlane img[OLPT_MAX_CAM];  // current working image per camera

  // detections
  olpt::Dets dets[OLPT_MAX_CAM];
  // int64 words: [OLPT_MAX_CAM] detection counts, then the staged detector's error
  // word, band ticket and per-band look-back states
  olpt::DevBuf det_counts;
  std::vector<int64_t> det_counts_h;
  struct DetMap {  // TMA descriptor of one camera plane, re-encoded when the plane changes
    const void* p = nullptr;
    int dtype = -1, H = 0, W = 0, box_w = 0, box_h = 0;
    int64_t pitch = 0;
    CUtensorMap map;
  } det_map[OLPT_MAX_CAM];
  olpt::DevBuf band_counts, band_offsets;
  olpt::DevBuf lut_u8, lut_u16;  // log(max(v, 1e-4)) of every integer level
  // failure-detection test hook of the next staged detection launch (-1 = off)
  int test_hold_ticket = -1;
  unsigned long long test_wait_limit_ns = 0;

  // stereo matching
  olpt::StereoWork sm;
  olpt::StereoResult sm_result;
  olpt::PruneWork prune;

  // 3D objects (stereo output / shake input and output)
  olpt::Objects obj;

  // shake: residual planes (FP32 or FP64) and workspace
  olpt::ImagePlane resid[OLPT_MAX_CAM];
  olpt::ShakeWork shk;

  // IPR workspace and output
  olpt::IprWork ipr;

  // Shake-the-Box frame loop
  olpt::StbState stb;
  olpt::TrackIoWork tio;

  // learned proposal
  olpt::MlpWork mlp;

  // optional per-kernel event timing
  olpt::Prof prof;

  // scratch, and the pinned block of the read-backs
  olpt::DevBuf scratch;
  olpt::HostBuf pinned;
};

namespace olpt {

// Results read back to the host: copies into the context's pinned block, one synchronisation,
// and from there to where they belong.  A copy to pageable memory waits for the stream by
// itself, and goes through a staging area of the driver (a detection list of 1,700 spots in
// three of them: 30 us, this way 12 us).  What does not fit into the block (results so large
// that the copy itself counts) is copied directly.  The block starts with the first read-back
// and grows to what they need, because pinning is paid by the page (64 KB 60 us, 1 MB 1.1 ms):
// a context that only runs the network has none.  One user at a time, like the context.
constexpr size_t kReadBackFirst = 64 << 10, kReadBackBytes = 1 << 20;

class ReadBack {
 public:
  explicit ReadBack(olpt_ctx* c) : c_(c) {}
  void add(void* dst, const void* src, size_t bytes) {
    if (!bytes) return;
    if (n_ < kMax && room(bytes)) {
      char* at = c_->pinned.as<char>() + used_;
      OLPT_CUDA(cudaMemcpyAsync(at, src, bytes, cudaMemcpyDeviceToHost, c_->stream));
      part_[n_++] = {dst, at, bytes};
      used_ += (bytes + 15) / 16 * 16;
    } else {
      OLPT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c_->stream));
    }
  }
  void finish() {
    OLPT_CUDA(cudaStreamSynchronize(c_->stream));
    for (int i = 0; i < n_; ++i) std::memcpy(part_[i].dst, part_[i].at, part_[i].bytes);
    n_ = 0;
    used_ = 0;
  }

 private:
  static constexpr int kMax = 8;
  // the block holds `bytes` more, after growing where it may
  bool room(size_t bytes) {
    HostBuf& b = c_->pinned;
    if (used_ + bytes <= b.bytes) return true;
    if (used_ + bytes > kReadBackBytes) return false;
    size_t size = kReadBackFirst;
    while (size < used_ + bytes) size *= 2;
    finish();  // no copy into the block that goes is under way
    void* p = nullptr;
    if (cudaMallocHost(&p, size) != cudaSuccess) {
      cudaGetLastError();
      return bytes <= b.bytes;
    }
    if (b.p) cudaFreeHost(b.p);
    b.p = p;
    b.bytes = size;
    return true;
  }
  struct Part {
    void* dst;
    const void* at;
    size_t bytes;
  };
  olpt_ctx* c_;
  Part part_[kMax];
  int n_ = 0;
  size_t used_ = 0;
};

template <class T>
T read_back(olpt_ctx* c, const T* src) {
  T v;
  ReadBack rb(c);
  rb.add(&v, src, sizeof(T));
  rb.finish();
  return v;
}

}  // namespace olpt
