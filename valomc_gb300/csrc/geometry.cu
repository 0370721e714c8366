// geometry.cu -- a mesh's neighbours and element records, made on the device.
//
// The host's search for the neighbours of the 648k-tet phantom takes 30 ms on 16 Grace cores (60
// million candidates compared) and its records 3 ms more.  Here a thread searches a face, the
// candidates' vertices come out of the L2, and only the list of boundary faces goes back: all of a
// call's preparation on that mesh is 3 ms (38 on the host), most of it the copies of the input.
#include <cuda_runtime.h>
#include <math.h>

#include <vector>

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

// ---- neighbours: BuildNeighbourhoods as host_setup.cpp's build_neighbours, a thread a face ----

struct Geometry {
  const int64_t *H, *BH, *HN;  // column-major
  const double *r;
  int64_t Ne, Nb, Nr;
  __device__ int64_t h(int64_t e, int c) const { return H[e + Ne * c]; }
  __device__ double x(int64_t v, int c) const { return r[v + Nr * c]; }
};

__global__ void count_incidences(const int64_t *idx, int64_t n, uint32_t *count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(count + idx[i], 1u);
}

// off[v] = count[0] + ... + count[v - 1], and count = a copy of it; one block
__global__ void __launch_bounds__(1024) scan_counts(uint32_t *count, uint32_t *off, int64_t n) {
  __shared__ uint32_t part[1024];
  const int64_t each = (n + 1023) / 1024, lo = min(n, each * threadIdx.x), hi = min(n, lo + each);
  uint32_t sum = 0;
  for (int64_t i = lo; i < hi; i++) sum += count[i];
  part[threadIdx.x] = sum;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const uint32_t v = threadIdx.x >= d ? part[threadIdx.x - d] : 0u;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t at = part[threadIdx.x] - sum;
  for (int64_t i = lo; i < hi; i++) {
    const uint32_t c = count[i];
    off[i] = count[i] = at;
    at += c;
  }
  if (hi == n && lo < hi) off[n] = at;
  if (n == 0 && threadIdx.x == 0) off[0] = 0;
}

// rows: elements (sign >= 0: i) or boundary elements (-1 - i); the order in a list does not matter
__global__ void fill_lists(const int64_t *idx, int64_t rows, int cols, bool boundary, uint32_t *at, int32_t *lst) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= rows * cols) return;
  const int32_t i = (int32_t)(k % rows);
  lst[atomicAdd(at + idx[k], 1u)] = boundary ? -1 - i : i;
}

// HN[el, f]: the one element or boundary element that holds all vertices of the face, from the
// shortest incidence list among them; bad: smallest (element * 32 + code) of two candidates
__global__ void find_neighbours(Geometry g, int dim, const uint32_t *off, const int32_t *lst, int64_t *HN, int dup_code,
                                int open_code, unsigned long long *bad) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int NF = dim + 1;
  if (k >= g.Ne * NF) return;
  const int64_t el = k % g.Ne;
  const int f = (int)(k / g.Ne);
  int64_t fv[3];
  if (dim == 3) {
    fv[0] = g.h(el, f == 3); fv[1] = g.h(el, f < 2 ? 1 : 2); fv[2] = g.h(el, f == 0 ? 2 : 3);
  } else {
    fv[0] = g.h(el, f); fv[1] = g.h(el, f == 2 ? 0 : f + 1); fv[2] = fv[1];
  }
  int64_t best = fv[0];
  for (int q = 1; q < dim; q++)
    if (off[fv[q] + 1] - off[fv[q]] < off[best + 1] - off[best]) best = fv[q];
  int64_t found = INT64_MAX;
  for (uint32_t q = off[best]; q < off[best + 1]; q++) {
    const int64_t cand = lst[q];
    if (cand == el) continue;
    bool all = true;
    for (int v = 0; v < dim && all; v++) {
      bool hit = false;
      if (cand >= 0) {
        for (int c = 0; c < NF; c++) hit |= g.h(cand, c) == fv[v];
      } else {
        for (int c = 0; c < dim; c++) hit |= g.BH[-1 - cand + g.Nb * c] == fv[v];
      }
      all = hit;
    }
    if (!all) continue;
    if (found != INT64_MAX && found != cand) {
      atomicMin(bad, (unsigned long long)el * 32u + (unsigned)dup_code);
      break;
    }
    found = cand;
  }
  HN[k] = found;
  if (dim == 2 && found == INT64_MAX) atomicMin(bad, (unsigned long long)el * 32u + (unsigned)open_code);
}

// the faces on the boundary, in any order
__global__ void list_faces(Geometry g, int NF, BoundaryFace *list, unsigned *n, unsigned cap) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.Ne * NF) return;
  const int64_t h = g.HN[k];
  if (h > -1 || h < -g.Nb) return;
  const int64_t el = k % g.Ne;
  const int f = (int)(k / g.Ne);
  int first = f;
  for (int q = f - 1; q >= 0; q--)
    if (g.HN[el + g.Ne * q] == h) first = q;
  const unsigned at = atomicAdd(n, 1u);
  if (at < cap) list[at] = BoundaryFace{(int32_t)el, (int32_t)(-1 - h), (int8_t)f, (int8_t)first};
}

__device__ int32_t nbr32(const Geometry &g, int64_t el, int f) {
  const int64_t h = g.HN[el + g.Ne * f];
  return h >= g.Ne || h < -g.Nb ? kOpenFace : (int32_t)h;
}

// ---- records; products and sums in the order and roundings of the host's (no fused operations),
// so that the FP32 planes are the same bits wherever they are made ----
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dot3(const double *a, const double *b) {
  return add(add(mul(a[0], b[0]), mul(a[1], b[1])), mul(a[2], b[2]));
}

__global__ void tet32_records(Geometry g, Tet32 *out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.Ne * 4) return;
  const int64_t el = k >> 2;
  const int f = (int)(k & 3);
  // the face's vertices in ascending id order: both elements of a face store exactly opposite planes
  int64_t i0 = g.h(el, f == 3), i1 = g.h(el, f < 2 ? 1 : 2), i2 = g.h(el, f == 0 ? 2 : 3);
  const int64_t o = g.h(el, 3 - f);
  int64_t t;
  if (i0 > i1) { t = i0; i0 = i1; i1 = t; }
  if (i1 > i2) { t = i1; i1 = i2; i2 = t; }
  if (i0 > i1) { t = i0; i0 = i1; i1 = t; }
  double p[3], a[3], b[3], q[3];
  for (int c = 0; c < 3; c++) {
    p[c] = g.x(i0, c);
    a[c] = sub(g.x(i1, c), p[c]);
    b[c] = sub(g.x(i2, c), p[c]);
    q[c] = sub(g.x(o, c), p[c]);
  }
  double n[3] = {sub(mul(a[1], b[2]), mul(a[2], b[1])), sub(mul(a[2], b[0]), mul(a[0], b[2])),
                 sub(mul(a[0], b[1]), mul(a[1], b[0]))};
  const double nn = __dsqrt_rn(dot3(n, n));
  for (int c = 0; c < 3; c++) n[c] = __ddiv_rn(n[c], nn);
  const double d = dot3(n, p);
  const float s = dot3(n, q) > 0.0 ? -1.0f : 1.0f;  // outward: away from the opposite vertex
  Tet32 &T = out[el];
  *reinterpret_cast<float4 *>(T.pl[f]) =
      make_float4(s * (float)n[0], s * (float)n[1], s * (float)n[2], s * (float)d);
  T.nbr[f] = nbr32(g, el, f);
}

__global__ void tri32_records(Geometry g, Tri32 *out) {
  const int64_t el = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (el >= g.Ne) return;
  Tri32 T;
  for (int f = 0; f < 3; f++) {
    int64_t i0 = g.h(el, f), i1 = g.h(el, f == 2 ? 0 : f + 1);
    const int64_t o = g.h(el, f == 0 ? 2 : f - 1);
    if (i0 > i1) { const int64_t t = i0; i0 = i1; i1 = t; }
    const double px = g.x(i0, 0), py = g.x(i0, 1);
    const double tx = sub(g.x(i1, 0), px), ty = sub(g.x(i1, 1), py);
    const double nn = __dsqrt_rn(add(mul(tx, tx), mul(ty, ty)));
    const double n0 = __ddiv_rn(ty, nn), n1 = __ddiv_rn(-tx, nn);
    const double d = add(mul(n0, px), mul(n1, py));
    const double side = add(mul(n0, sub(g.x(o, 0), px)), mul(n1, sub(g.x(o, 1), py)));
    const float s = side > 0.0 ? -1.0f : 1.0f;
    T.ln[f][0] = s * (float)n0;
    T.ln[f][1] = s * (float)n1;
    T.ln[f][2] = s * (float)d;
    T.ln[f][3] = 0.0f;
    T.nbr[f] = nbr32(g, el, f);
  }
  T.nbr[3] = kOpenFace;
  out[el] = T;
}

__global__ void vertex_records(Geometry g, int dim, void *out) {
  const int64_t el = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (el >= g.Ne) return;
  if (dim == 3) {
    Tet64 T;
    for (int v = 0; v < 4; v++)
      for (int c = 0; c < 3; c++) T.v[v][c] = g.x(g.h(el, v), c);
    for (int f = 0; f < 4; f++) T.nbr[f] = nbr32(g, el, f);
    static_cast<Tet64 *>(out)[el] = T;
  } else {
    Tri64 T;
    for (int v = 0; v < 3; v++)
      for (int c = 0; c < 2; c++) T.v[v][c] = g.x(g.h(el, v), c);
    for (int f = 0; f < 3; f++) T.nbr[f] = nbr32(g, el, f);
    T.nbr[3] = kOpenFace;
    static_cast<Tri64 *>(out)[el] = T;
  }
}

unsigned blocks(int64_t n) { return (unsigned)((n + 255) / 256); }

// device memory of one build, given back in order on the stream
struct Temp {
  cudaMemPool_t pool;
  cudaStream_t st;
  std::vector<void *> all;
  ~Temp() {
    if (!all.empty()) cudaStreamSynchronize(st);  // after an error: nothing still reads or writes the caller's arrays
    for (void *p : all) cudaFreeAsync(p, st);
  }
  template <class T>
  int get(T **p, size_t n) {
    VMC_CK(pool_alloc(reinterpret_cast<void **>(p), (n ? n : 1) * sizeof(T), pool, st));
    all.push_back(*p);
    return VMC_OK;
  }
};

int build(const vmc_input *in, int mask, DeviceMesh &m, bool keep_HN, Temp &t) {
  HostMesh &h = m.host;
  const int D = h.dim, NF = D + 1;
  const int64_t Ne = h.Ne, Nb = h.Nb, Nr = h.Nr;
  cudaStream_t st = t.st;
  Geometry g{nullptr, nullptr, nullptr, nullptr, Ne, Nb, Nr};
  int64_t *dH, *dBH, *dHN;
  double *dr;
  int s;
  const auto up = [st](auto *d, const auto *src, size_t n) {
    if (!n) return cudaSuccess;
    g_h2d_bytes += (int64_t)(n * sizeof(*d));
    return cudaMemcpyAsync(d, src, n * sizeof(*d), cudaMemcpyHostToDevice, st);
  };
  const auto down = [st](auto *dst, const auto *d, size_t n) {
    if (!n) return cudaSuccess;
    g_d2h_bytes += (int64_t)(n * sizeof(*d));
    return cudaMemcpyAsync(dst, d, n * sizeof(*d), cudaMemcpyDeviceToHost, st);
  };
  if ((s = t.get(&dH, (size_t)(Ne * NF))) || (s = t.get(&dBH, (size_t)(Nb * D))) || (s = t.get(&dr, (size_t)(Nr * D))) ||
      (s = t.get(&dHN, (size_t)(Ne * NF))))
    return s;
  VMC_CK(up(dH, h.H, (size_t)(Ne * NF)));
  VMC_CK(up(dBH, h.BH, (size_t)(Nb * D)));
  VMC_CK(up(dr, h.r, (size_t)(Nr * D)));
  g.H = dH; g.BH = dBH; g.r = dr; g.HN = dHN;
  // what comes back: the smallest error key, the number of boundary faces
  struct Found { unsigned long long bad; unsigned faces; unsigned pad; };
  Found *df;
  BoundaryFace *dlist;
  const unsigned cap = (unsigned)(2 * Nb + 1024);
  if ((s = t.get(&df, 1)) || (s = t.get(&dlist, cap))) return s;
  Found found{~0ull, 0, 0};
  VMC_CK(up(df, &found, 1));
  const bool given = in->HN && in->n_HN == Ne;
  if (given) {
    VMC_CK(up(dHN, in->HN, (size_t)(Ne * NF)));
  } else {
    uint32_t *count, *off;
    int32_t *lst;
    if ((s = t.get(&count, (size_t)Nr)) || (s = t.get(&off, (size_t)Nr + 1)) || (s = t.get(&lst, (size_t)(Ne * NF + Nb * D))))
      return s;
    VMC_CK(cudaMemsetAsync(count, 0, sizeof(uint32_t) * (size_t)Nr, st));
    count_incidences<<<blocks(Ne * NF), 256, 0, st>>>(dH, Ne * NF, count);
    if (Nb) count_incidences<<<blocks(Nb * D), 256, 0, st>>>(dBH, Nb * D, count);
    scan_counts<<<1, 1024, 0, st>>>(count, off, Nr);
    fill_lists<<<blocks(Ne * NF), 256, 0, st>>>(dH, Ne, NF, false, count, lst);
    if (Nb) fill_lists<<<blocks(Nb * D), 256, 0, st>>>(dBH, Nb, D, true, count, lst);
    find_neighbours<<<blocks(Ne * NF), 256, 0, st>>>(g, D, off, lst, dHN,
                                                     D == 3 ? VMC_INCONSISTENT_MESH_DUPLICATE_NEIGHBORS : VMC_INCONSISTENT_MESH,
                                                     VMC_MISSING_BOUNDARY, &df->bad);
  }
  list_faces<<<blocks(Ne * NF), 256, 0, st>>>(g, NF, dlist, &df->faces, cap);
  // the records
  for (int prec = 0; prec < 2; prec++) {
    if (!(mask & (1 << prec))) continue;
    const size_t size = m.record_bytes(prec);
    void *p = nullptr;
    if (m.pool) VMC_CK(pool_alloc(&p, size * (size_t)Ne, m.pool, m.st));
    else VMC_CK(cudaMalloc(&p, size * (size_t)Ne));
    m.d_geom[prec] = p;
    m.bytes += (int64_t)(size * (size_t)Ne);
    if (prec == VMC_FP64) {
      vertex_records<<<blocks(Ne), 256, 0, st>>>(g, D, const_cast<void *>(m.geom(VMC_FP64, true)));
      if (m.planes) VMC_CK(make_plane_records(D, p, Ne, st));
    } else if (D == 3) {
      tet32_records<<<blocks(Ne * 4), 256, 0, st>>>(g, static_cast<Tet32 *>(p));
    } else {
      tri32_records<<<blocks(Ne), 256, 0, st>>>(g, static_cast<Tri32 *>(p));
    }
  }
  VMC_CK(cudaGetLastError());
  VMC_CK(down(&found, df, 1));
  // meanwhile the host measures what the jobs need first
  measure_boundary(h);
  VMC_CK(cudaStreamSynchronize(st));
  if (found.bad != ~0ull) return (int)(found.bad % 32u);
  if (found.faces <= cap) {
    h.faces.resize(found.faces);
    VMC_CK(down(h.faces.data(), dlist, found.faces));
  }
  if (keep_HN || found.faces > cap) {
    h.HN.resize((size_t)(Ne * NF));
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < Ne * NF; i += 512) h.HN[(size_t)i] = 0;  // map the pages
    VMC_CK(down(h.HN.data(), dHN, (size_t)(Ne * NF)));
  }
  VMC_CK(cudaStreamSynchronize(st));
  if (found.faces > cap) list_boundary_faces(h);  // a given neighbourhood with more faces than it should have
  sort_faces(h);
  return VMC_OK;
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

int build_mesh_on_device(const vmc_input *in, int precision_mask, DeviceMesh &m, bool own, bool keep_HN) {
  int s = take_geometry(in, m.host, own);
  if (s) return s;
  m.dim = in->dim;
  cudaMemPool_t pool = nullptr;
  if ((s = call_pool(m.device, &pool))) return s;
  m.planes = planes_fit(m.dim, m.host.Ne);
  Temp t{pool, m.st, {}};
  const int64_t before = m.bytes;
  s = build(in, precision_mask, m, keep_HN, t);
  if (s) {
    m.bytes = before;
    for (void *&p : m.d_geom) {
      if (p && m.pool) cudaFreeAsync(p, m.st);
      else if (p) cudaFree(p);
      p = nullptr;
    }
  }
  return s;
}

}  // namespace vmc
