// geometry.cu -- kernels that derive the element records of a mesh on the device.
#include <cuda_runtime.h>
#include <math.h>

#include "engine.hpp"

namespace vmc {

namespace {

// below this face size (twice the area, or the edge length) the reference's parallel test can
// take part in its choice of the exit face: the FP32 normals are left out
constexpr double kMinFace = 1e-9;

__device__ void store_normal(double *n, float *nf, const double *v, int dim, double size, bool use) {
  for (int c = 0; c < dim; c++) {
    n[c] = v[c];
    nf[c] = use ? (float)(v[c] / size) : NAN;
  }
}

__global__ void tet_records(TetRec *rec, const Tet64 *tet, int64_t Ne) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= Ne) return;
  const Tet64 &T = tet[e];
  TetRec R;
  for (int c = 0; c < 3; c++) R.v0[c] = T.v[0][c];
  double size[4], smallest = INFINITY;
  double nn[4][3];
  for (int f = 0; f < 4; f++) {
    // face (0,1,2), (0,1,3), (0,2,3) or (1,2,3), opposite vertex 3 - f; Normal(el, f), MC3D.hpp:408-457
    const int i0 = f == 3, i1 = f < 2 ? 1 : 2, i2 = f == 0 ? 2 : 3, o = 3 - f;
    double a[3], b[3], t[3];
    for (int c = 0; c < 3; c++) {
      a[c] = T.v[i1][c] - T.v[i0][c];
      b[c] = T.v[i2][c] - T.v[i0][c];
      t[c] = T.v[o][c] - T.v[i0][c];
    }
    double n[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    size[f] = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    smallest = fmin(smallest, size[f]);
    const bool in = n[0] * t[0] + n[1] * t[1] + n[2] * t[2] > 0.0;  // out: away from o
    for (int c = 0; c < 3; c++) nn[f][c] = in ? -n[c] : n[c];
  }
  for (int f = 0; f < 4; f++) store_normal(R.n[f], R.nf[f], nn[f], 3, size[f], smallest >= kMinFace);
  R.off = 0.0;
  for (int c = 0; c < 3; c++) R.off += R.n[3][c] * (T.v[1][c] - T.v[0][c]);
  R.off_size = (float)(R.off / size[3]);
  for (int f = 0; f < 4; f++) R.nbr[f] = T.nbr[f];
  rec[e] = R;
}

__global__ void tri_records(TriRec *rec, const Tri64 *tri, int64_t Ne) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= Ne) return;
  const Tri64 &T = tri[e];
  TriRec R;
  for (int c = 0; c < 2; c++) R.v0[c] = T.v[0][c];
  R.pad = 0.0;
  R.padf = 0.0f;
  double size[3], smallest = INFINITY;
  double nn[3][2];
  for (int f = 0; f < 3; f++) {
    // edge (0,1), (1,2) or (2,0); Normal(el, f), MC2D.hpp:358-387
    const int i0 = f, i1 = f == 2 ? 0 : f + 1, o = f == 0 ? 2 : f - 1;
    const double dx = T.v[i1][0] - T.v[i0][0], dy = T.v[i1][1] - T.v[i0][1];
    size[f] = sqrt(dx * dx + dy * dy);
    smallest = fmin(smallest, size[f]);
    const bool in = dy * (T.v[o][0] - T.v[i0][0]) - dx * (T.v[o][1] - T.v[i0][1]) > 0.0;
    nn[f][0] = in ? -dy : dy;
    nn[f][1] = in ? dx : -dx;
  }
  for (int f = 0; f < 3; f++) store_normal(R.n[f], R.nf[f], nn[f], 2, size[f], smallest >= kMinFace);
  R.off = R.n[1][0] * (T.v[1][0] - T.v[0][0]) + R.n[1][1] * (T.v[1][1] - T.v[0][1]);
  R.off_size = (float)(R.off / size[1]);
  for (int f = 0; f < 4; f++) R.nbr[f] = T.nbr[f];
  rec[e] = R;
}

}  // namespace

cudaError_t make_plane_records(int dim, void *geom, int64_t Ne, cudaStream_t st) {
  if (Ne == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((Ne + 127) / 128);
  if (dim == 3) {
    TetRec *r = static_cast<TetRec *>(geom);
    tet_records<<<grid, 128, 0, st>>>(r, reinterpret_cast<const Tet64 *>(r + Ne), Ne);
  } else {
    TriRec *r = static_cast<TriRec *>(geom);
    tri_records<<<grid, 128, 0, st>>>(r, reinterpret_cast<const Tri64 *>(r + Ne), Ne);
  }
  return cudaGetLastError();
}

}  // namespace vmc
