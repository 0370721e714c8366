// host_setup.hpp -- host half of the drop-in: ErrorChecks, Init and the normalisation of
// MC3D/MC2D (cpp/3d/MC3D.hpp:460-738, :1792-1818; cpp/2d/MC2D.hpp:390-643, :1672-1703),
// producing the device records of vmc_types.hpp.  Compiled with -ffp-contract=off so the
// per-face launch quantities are the reference's doubles bit for bit.
#pragma once
#include <stdint.h>

#include <cstddef>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/valomc_gb300.h"
#include "vmc_types.hpp"

namespace vmc {

// An array of plain values that starts uninitialised: its pages are first touched by the threads
// that fill it, not by a zeroing constructor.
template <class T>
class Raw {
 public:
  void resize(size_t n) {
    if (n != n_) p_.reset(n ? new T[n] : nullptr);
    n_ = n;
  }
  void clear() { resize(0); }
  T *data() { return p_.get(); }
  const T *data() const { return p_.get(); }
  size_t size() const { return n_; }
  T &operator[](size_t i) { return p_[i]; }
  const T &operator[](size_t i) const { return p_[i]; }

 private:
  std::unique_ptr<T[]> p_;
  size_t n_ = 0;
};

// A face of element el on the boundary (face f behind boundary element ib); first: the lowest
// face of el on ib.
struct BoundaryFace {
  int32_t el, ib;
  int8_t f, first;
};

// Geometry shared by every job on a mesh.
struct HostMesh {
  int dim = 3;
  int64_t Ne = 0, Nb = 0, Nr = 0;
  // column-major; the caller's arrays for a mesh that lives for one call, else copies
  const int64_t *H = nullptr, *BH = nullptr;
  const double *r = nullptr;
  Raw<int64_t> own_H, own_BH;
  Raw<double> own_r;
  Raw<int64_t> HN;              // column-major [Ne x (dim+1)]
  std::vector<BoundaryFace> faces;  // in (element, face) order
  Raw<double> volume;           // ElementVolume / ElementArea(el)
  Raw<double> area;             // ElementArea(ib) / ElementLength(ib)
  std::vector<double> bnorm;    // [Nb x 4] Normal(ib)
  // device records, until they are uploaded
  Raw<Tet64> tet64;
  Raw<Tet32> tet32;
  Raw<Tri64> tri64;
  Raw<Tri32> tri32;
};

// One problem on a mesh: optics, boundary conditions, sources, scalars.
struct HostJob {
  int dim = 3;
  int64_t Ne = 0, Nb = 0;
  bool homogeneous = false;
  // optics of the elements (a single one each when homogeneous): the caller's arrays, or the
  // job's own after keep()
  const double *mua = nullptr, *mus = nullptr, *g = nullptr, *n = nullptr;
  Raw<double> own;
  size_t rows() const { return homogeneous ? 1 : (size_t)Ne; }
  double mua_of(int64_t i) const { return mua[homogeneous ? 0 : i]; }
  double k_of(int64_t i) const;  // omega / c0 * n (MC3D.hpp:660-662)
  void keep();                   // copies the optics out of the caller's arrays
  // rows of (mua, mus, g, n)
  void optics_rows(float *out) const;
  void optics_rows(double *out) const;
  std::vector<uint8_t> bctype;
  std::vector<double> bcn;
  std::vector<SourceRec> src;
  std::vector<double> cdf;
  std::vector<SourceRecF> src_f;  // FP32 copies for the tracking form
  std::vector<float> cdf_f;
  double f = 0, omega = 0, k_scale = 0, phase0 = 0;
  double k_turn = 0;            // f / c0, turns a millimetre in vacuum
  uint64_t turn0 = 0;           // phase0 in 2^-64 turns
  int64_t Nphoton = 0;
  uint64_t seed = 0;
  float walk = 0;               // about how long its walks are: scatterings per absorption length
};

// Memory that a call writes its results to.  A job reads its optics from the caller's arrays until
// the results are normalised: where a caller has results written over those arrays, the job keeps
// its own copy (HostJob::keep).
class ResultSpans {
 public:
  ResultSpans(const vmc_output *outs, const HostMesh *const *meshes, int n);
  bool meets(const HostJob &j) const;  // an array of j's optics overlaps one of the results

 private:
  struct Span { uintptr_t begin, end; };
  std::vector<Span> spans_;  // by their begin, each end the largest so far
};

// Whether the scattering coefficient or the index changes across more than an eighth of the mesh's
// interior faces: such jobs run the literal FP64 walk.  A photon's remaining path is multiplied
// by mus / mus2 at each of these faces, so rounding differences are too: on the 648k-tet phantom
// with mus drawn per element (every face) walks of some thousand steps end elsewhere after any
// change of rounding, while with one or two inclusions (2-4 % of the faces) results move by 1e-14.
// Both sides of the line, in a box of 16 x 16 x 12 cells with layers of mus 9 and 11: two cells thick
// (7 % of the faces) and one (16 %), the two walks differ by 1.4e-13 to 1.9e-13 (L2), the plain one is
// 2e-14 to 5e-14 off 80-bit arithmetic and the literal one 1.4e-13 to 1.9e-13, and 5e4 photons take 20
// and 77 ms.  So in a small body either would do: the line is there for the reference's own
// trajectories in large ones, and optics that differ in their last digits alone count as changes.
bool rough_optics(const vmc_input *in, const HostMesh &m);

// ErrorChecks (same checks, same order, same codes).  Returns VMC_OK or 1 + mcerror.
// indices: also that H and BH name nodes (done once, when a resident mesh was made).
int check_input(const vmc_input *in, bool indices = true);
bool nodes_in_range(const int64_t *idx, int64_t n, int64_t Nr);
// an input's geometry replaced by a resident mesh's
void use_mesh(vmc_input &in, const HostMesh &m);

// BuildNeighbourhoods: HN [Ne x (dim+1)] column-major with the reference's semantics
// (boundary -1 - ib, 3D open faces INT64_MAX, 2D open edges -> MISSING_BOUNDARY,
// two different candidates for one face -> INCONSISTENT_MESH[_DUPLICATE_NEIGHBORS]).
int build_neighbours(int dim, int64_t Ne, int64_t Nb, int64_t Nr, const int64_t *H, const int64_t *BH, int64_t *HN);

// Mesh from the geometry arrays of an input (HN built unless given).  precision_mask:
// bit 0 builds the FP64 records, bit 1 the FP32 records.  own: the mesh outlives the input's
// arrays and copies them.
int build_mesh(const vmc_input *in, int precision_mask, HostMesh &m, bool own);
// Its parts, for a mesh whose neighbours and records are made on the device: sizes and arrays, the
// boundary's areas and normals, the order of the faces, the elements' volumes.
int take_geometry(const vmc_input *in, HostMesh &m, bool own);
void measure_boundary(HostMesh &m);
void list_boundary_faces(HostMesh &m);  // from HN, in any order
void sort_faces(HostMesh &m);
void measure_elements(HostMesh &m);

// Job from the problem arrays of an input on mesh m (Init's light sources, BCLNormal
// processing and wave numbers).  The job reads the input's optics arrays until keep().
int build_job(const vmc_input *in, const HostMesh &m, HostJob &j);

// MonteCarlo's normalisation of raw accumulators into the caller's output arrays.
void normalise(const HostMesh &m, const HostJob &j, int64_t nphoton, const double *ER, const double *EI,
               const double *EBR, const double *EBI, const double *DEBR, const double *DEBI, vmc_output *out,
               bool apply);

const char *mcerror_string(int status);

}  // namespace vmc
