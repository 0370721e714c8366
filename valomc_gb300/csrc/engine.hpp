// engine.hpp -- internal interface between the C ABI, the batch path and the serving loop.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <string>
#include <vector>

#include "host_setup.hpp"

namespace vmc {

void set_error(const std::string &msg);
int cuda_status(cudaError_t e, const char *what);
// bytes this thread's call has copied to and from the device
extern thread_local int64_t g_h2d_bytes, g_d2h_bytes;

#define VMC_CK(call)                                      \
  do {                                                    \
    cudaError_t _e = (call);                              \
    if (_e != cudaSuccess) return cuda_status(_e, #call); \
  } while (0)

int select_device(int device, int *num_sms = nullptr);
uint64_t clock_seed();

// Resident geometry (the opaque vmc_mesh).
struct DeviceMesh {
  int device = 0;
  int dim = 3;
  HostMesh host;
  void *d_geom[2] = {nullptr, nullptr};  // [precision]
  double *d_bnorm = nullptr;
  int64_t bytes = 0;
  // a mesh that lives for one call: allocated from `pool` and copied, then freed, in order
  // on `st` (no device-wide synchronisation); resident meshes keep plain allocations
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;
  ~DeviceMesh();
  // FP64: the plane records are made (then d_geom holds them, and the vertex records behind them)
  bool planes = true;
  // what a walk reads: the plain FP64 one the plane records, the literal one the vertex records
  const void *geom(int precision, bool literal) const;
  // device bytes of an element's records
  size_t record_bytes(int precision) const;
};
// Whether an FP64 mesh gets plane records beside the vertex records (320 bytes a tetrahedron, 112
// without, 192 and 64 a triangle): only where such a mesh and the arrays of a job on it (48 bytes
// an element) leave half of the device's free memory.  One that does not, or for which there is no
// memory when it is made, is the size it was before there were planes, and its jobs take the
// literal walk, which needs none.  Up to kPlanesAlways bytes the memory is not asked for.
constexpr size_t kPlanesAlways = 1ull << 30;
bool planes_fit(int dim, int64_t Ne);
int upload_mesh(DeviceMesh &m, int precision_mask);
// The same from the input's arrays with neighbours and records made on the device (m.device is
// current, m.st and m.pool are set).  keep_HN: the host gets HN too.  Out of memory leaves nothing
// on the device, and the host can build.
int build_mesh_on_device(const vmc_input *in, int precision_mask, DeviceMesh &m, bool own, bool keep_HN);
// Whether that pays.  A call with one photon takes on the host / with the device, in ms: 0.33 /
// 0.35 at 800 triangles in FP64 (0.33 / 0.30 in FP32), 0.40 / 0.37 at 1250 (0.40 / 0.31), 1.45 /
// 0.64 at 20000; 0.61 / 0.40 at 750 tetrahedra, 11.0 / 2.1 at 162k, 95 / 32 at 1.3M: launches and
// copies cost 0.1 ms, the host's search some 50 ns a face on its 16 cores and its records 5 more.
// Above 2^26 elements the scratch of 90 bytes an element could be what a mesh that fits by itself
// lacks.
inline bool builds_on_device(int64_t Ne) { return Ne >= 1000 && Ne <= (int64_t)1 << 26; }
// TetRec / TriRec [Ne] at `geom` from the Tet64 / Tri64 [Ne] behind them (planes)
cudaError_t make_plane_records(int dim, void *geom, int64_t Ne, cudaStream_t st);

// Memory of calls and launches: a pool of this library's per device, so that a call's buffers
// are not mapped and unmapped each time.  It keeps at most kPoolKeep bytes between calls (what is
// freed beyond that goes back at the next synchronisation), and all of it when an allocation fails.
// It belongs to the device's current context (the device is selected): another one after
// cudaDeviceReset.
constexpr uint64_t kPoolKeep = 256ull << 20;
int call_pool(int device, cudaMemPool_t *pool);
// cudaMallocFromPoolAsync; gives the kept memory back and tries again when there is none
cudaError_t pool_alloc(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st);

// Device state of one job, in one allocation: what is uploaded, then what the kernel adds to.
struct JobBuffers {
  void *d_block = nullptr;
  Raw<unsigned char> staged;  // host image of the uploaded part (alive while its copy may run)
  void *d_optics = nullptr;
  uint8_t *d_bctype = nullptr;
  double *d_bcn = nullptr, *d_cdf = nullptr;
  SourceRec *d_src = nullptr;
  float *d_cdf_f = nullptr;
  SourceRecF *d_src_f = nullptr;
  // counters, ledger and accumulators lie back to back: cleared and read back at once
  unsigned long long *d_jc = nullptr;
  double *d_ledger = nullptr;
  double *d_acc = nullptr;  // ER, EI [Ne]; EBR, EBI, DEBR, DEBI [Nb]
  size_t result_bytes() const { return sizeof(double) * (size_t)(kSlots * (kJcN + kLgN) + 2 * Ne + 4 * Nb); }
  uint32_t *d_tape = nullptr;
  int64_t *d_tape_off = nullptr, *d_trace = nullptr, *d_trace_len = nullptr;
  int64_t bytes = 0;
  int64_t Ne = 0, Nb = 0;
  // Stream-ordered allocation (the serving loop): buffers come from `pool` on the upload
  // stream and go back with cudaFreeAsync on `free_stream`, so that freeing a finished
  // request never waits for the device (cudaFree would, and stall the launches in flight).
  cudaMemPool_t pool = nullptr;
  cudaStream_t free_stream = nullptr;
  ~JobBuffers();
  void release();
};
// bytes of device state a job on mesh m needs (admission control)
int64_t job_footprint(const HostJob &j, const HostMesh &m);
int upload_job(const HostJob &j, const DeviceMesh &m, int precision, JobBuffers &b, cudaStream_t st);
JobDev describe_job(const HostJob &j, const DeviceMesh &m, int precision, bool literal, const JobBuffers &b);
// Whether a job runs the literal FP64 walk (rough_optics, or a mesh without plane records).
bool runs_literal(const vmc_input *in, const DeviceMesh &m, int precision);
int zero_job(JobBuffers &b, cudaStream_t st);

struct LaunchSpec {
  int dim = 3, precision = VMC_FP32;
  bool fd = false, tape = false;
  bool literal = false; // FP64: the reference's operation sequence (runs_literal)
  bool graph = false;  // launch through a (reused) CUDA graph
  int stage_slots = 0; // shared-memory staging slots per CTA (0: off)
  int block = 0, blocks_per_sm = 0, chunk = 0;
  int refill = 0;      // idle lanes a warp waits for before relaunching (0: default)
  int64_t max_steps = 0;
};
struct LaunchResult {
  uint64_t steps = 0, scatters = 0, done = 0;
  double kernel_ms = 0;
  int grid = 0, block = 0;
};
// Runs the pool kernel over jobs (device descriptors are uploaded here) and waits,
// polling progress / cancel / timeout from opt (may be null).  Stream-ordered.  meanwhile: host
// work to do while the kernel runs.
int launch_jobs(int device, const LaunchSpec &spec, const std::vector<JobDev> &jobs, const vmc_options *opt,
                cudaStream_t st, LaunchResult &res, const std::function<void()> &meanwhile = nullptr);

// Device and pinned buffers of one launch at a time, reused across launches: the job
// table, its photon prefix, the control block, the timing events and a graph.  Lets a
// caller keep a launch in flight while it prepares the next on another arena and stream.
struct LaunchArena {
  JobDev *djobs = nullptr, *hjobs = nullptr;
  int64_t *dbegin = nullptr, *hbegin = nullptr;
  Ctl *dctl = nullptr, *hctl = nullptr;
  size_t cap_jobs = 0;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaStream_t cap_stream = nullptr;  // graph capture
  cudaGraphExec_t exec = nullptr;
  int64_t total = 0, next0 = 0;  // photons, and those dealt out before the fetch counter starts
  bool pending = false;
  LaunchArena() = default;
  LaunchArena(const LaunchArena &) = delete;
  LaunchArena &operator=(const LaunchArena &) = delete;
  ~LaunchArena();
};
// Enqueues the pool kernel over jobs on `st` without waiting (no progress polling).
int launch_start(int device, const LaunchSpec &spec, const std::vector<JobDev> &jobs, LaunchArena &a,
                 cudaStream_t st, LaunchResult &res);
// Waits for the arena's launch and reads its counters (no-op when nothing is in flight).
int launch_finish(LaunchArena &a, cudaStream_t st, LaunchResult &res);

// Copies a job's accumulators and counters back (into `back`, kept by the caller for the next)
// and fills out/stats.
int collect_job(const HostJob &j, const DeviceMesh &m, const JobBuffers &b, int64_t nphoton, bool normalize,
                vmc_output *out, vmc_stats *st, cudaStream_t stream, Raw<double> &back);
// Touches the pages that collect_job will fill, so that they are mapped while the kernel runs and
// not by the copy (10 MB into fresh pages took 2 to 10 ms, into mapped ones 0.07).
void touch_results(const HostMesh &m, const JobBuffers &b, const vmc_output *out, Raw<double> &back);

const void *kernel_3d64(bool fd, bool tape, bool one, bool tab);
const void *kernel_3d64_literal(bool fd, bool tape, bool one, bool tab);
const void *kernel_3d32(bool fd, bool tape, bool one, bool tab);
const void *kernel_2d64(bool fd, bool tape, bool one, bool tab);
const void *kernel_2d64_literal(bool fd, bool tape, bool one, bool tab);
const void *kernel_2d32(bool fd, bool tape, bool one, bool tab);
// one: the single-job form (descriptor and round keys in LaunchParams::job0 / rk);
// tab: the per-job form with the job table copied into each CTA's shared memory
const void *select_kernel(const LaunchSpec &s, bool one = false, bool tab = false);
void set_single_job(LaunchParams &lp, const JobDev &job);
// the photons that the warps of a launch start with (lp.total is set)
void deal_photons(LaunchParams &lp, int grid, int block, int per_sm, int sms);
// the L1 / shared-memory split of a pool kernel: reset to the driver's default before the
// occupancy query, then the smallest split holding per_sm CTAs' shared memory
void reset_carveout(const void *fn);
void fit_carveout(const void *fn, int device, int per_sm, size_t dyn_smem);

}  // namespace vmc
