// mesh.cu -- the mesh collocation operator assembled on the device.
//
// The reference builds the collocation matrix of a triangle-mesh scene in
// torch every step (core/KTAB_Mfs_spclf1d.py:95-113): the solid angle of every
// face seen from every source (utils/torch_utils.py:306-334,
// compute_solid_angle, through faces x sources x 3 temporaries) and the
// rigid-mode right-hand side FL @ IQ (compute_FL_matrix, :62-75, and
// compute_face_centers, :49-60).  Here every entry is computed in FP64 from
// float32 coordinates and stored as FP32 or FP64, with no temporaries in
// global memory.
#include <cmath>
#include <cstdint>
#include <string>

#include <cuda_runtime.h>

#include "mbc_internal.h"

namespace {

template <typename T>
__device__ __forceinline__ T to_out(double v);
template <>
__device__ __forceinline__ float to_out<float>(double v) { return (float)v; }
template <>
__device__ __forceinline__ double to_out<double>(double v) { return v; }

// M[f, j] = 2 atan2(R1 . (R2 x R3), l1 l2 l3 + (R1.R2) l3 + (R1.R3) l2 + (R2.R3) l1),
// Rk = V[F[f, k]] - S[j] (van Oosterom and Strackee).  Block: 128 sources of
// one face; faces loop over gridDim.y so any face count fits the grid.
template <typename T>
__global__ void __launch_bounds__(128) solid_angle_kernel(int n_vert, const float *__restrict__ V, int n_faces,
                                                          const int32_t *__restrict__ F, int n_src,
                                                          const float *__restrict__ S, T *__restrict__ M,
                                                          int64_t ldm)
{
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_src) return;
  const double sx = S[3 * (size_t)j], sy = S[3 * (size_t)j + 1], sz = S[3 * (size_t)j + 2];
  for (int f = blockIdx.y; f < n_faces; f += gridDim.y) {
    const int i1 = F[3 * (size_t)f], i2 = F[3 * (size_t)f + 1], i3 = F[3 * (size_t)f + 2];
    double out;
    if (i1 < 0 || i1 >= n_vert || i2 < 0 || i2 >= n_vert || i3 < 0 || i3 >= n_vert) {
      out = nan("");  // a face naming a vertex that does not exist
    } else {
      const double ax = V[3 * (size_t)i1] - sx, ay = V[3 * (size_t)i1 + 1] - sy, az = V[3 * (size_t)i1 + 2] - sz;
      const double bx = V[3 * (size_t)i2] - sx, by = V[3 * (size_t)i2 + 1] - sy, bz = V[3 * (size_t)i2 + 2] - sz;
      const double cx = V[3 * (size_t)i3] - sx, cy = V[3 * (size_t)i3 + 1] - sy, cz = V[3 * (size_t)i3 + 2] - sz;
      const double num = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
      const double la = sqrt(ax * ax + ay * ay + az * az);
      const double lb = sqrt(bx * bx + by * by + bz * bz);
      const double lc = sqrt(cx * cx + cy * cy + cz * cz);
      const double ab = ax * bx + ay * by + az * bz;
      const double ac = ax * cx + ay * cy + az * cz;
      const double bc = bx * cx + by * cy + bz * cz;
      out = 2.0 * atan2(num, la * lb * lc + ab * lc + ac * lb + bc * la);
    }
    M[(size_t)f * ldm + j] = to_out<T>(out);
  }
}

// ---------------------------------------------------------------------------
// FP32 matrices.  What bounds them: FP64 instructions (the 1.9 GB of 30720 x
// 15372 entries take 0.29 ms to store; three square roots, an arc tangent and
// the products of three vectors per entry took 4.9 ms).  A block takes 16
// faces x 128 sources at a time, a thread two sources of every fourth face, and
//   * evaluates each distinct vertex of its faces once per source (faces that
//     follow one another share theirs): q = |v - s|^2 and y = 1 / |v - s|, the
//     FP32 estimate after one Newton step (1e-14), kept in shared memory;
//   * has R1 . (R2 x R3) = R1 . n with the face's n = (v2 - v1) x (v3 - v1), and
//     Ri . Rj = (qi + qj - |vi - vj|^2) / 2, so that an entry divided by
//     l1 l2 l3 is num = (R1 . n) y1 y2 y3 over den = 1 + sum (Ri . Rj) yi yj.
//     Only differences of a face's own vertices and a source enter an entry: a
//     vertex that is NaN, infinite or far from the others changes the faces
//     that name it and no others of its tile;
//   * for |num| <= (den - 0.01) / 4 (all but the few sources next to a face or
//     its edges) takes atan(num / den) from its Maclaurin series, 4 terms below
//     0.02 and 10 up to 0.25 (errors 3e-15 and 5e-14 of the value); the other
//     entries take the formula with square roots and atan2.  So do those where
//     the form above cancels: den has an absolute error of ~3e-13 (from y, up to
//     4e-14 each) and ~3e-16 times the ratio of the longest to the shortest of
//     l1, l2, l3, and R1 . n loses that ratio too.  With den at least 0.01 and
//     the ratio at most 256 an entry keeps 1e-10, a thousandth of the FP32
//     rounding.  Distances outside 1e-17 .. 1e17, whose squares leave FP32's
//     range, and faces without a vertex (NaN) take the formula as well.
// About 40 FP64 instructions an entry instead of 190; the error is the FP32
// rounding of the stored value, as before.  Measured (B200, 30720 x 15372):
// 4.90 -> 2.49 ms; the FP64 pipe is 40 to 45 % busy, the rest waits for the chains of
// FP64 results (16 warps per SM).  FP64 matrices keep the kernel
// above.
constexpr int kFT = 16, kST = 128, kMaxV = 3 * kFT, kAsmThreads = 256;
constexpr int kFG = kAsmThreads / (kST / 2);  // groups of faces; a thread takes two sources
constexpr int kAsmSmem = 2 * kMaxV * kST * (int)sizeof(double);

constexpr double kMinDen = 0.01;
// upper words of positive doubles order as integers: the smallest y = 1 / l in
// 1e-17 .. 1e17 / 2^8 (a NaN's word lies outside), the largest within a factor
// of 2^8 of it
constexpr int kYLow = 0x3c670ef5;
constexpr unsigned kYRatio = 8u << 20, kYSpan = 0x43763457u - kYLow - kYRatio;

// atan(t), |t| <= 1/4, from its Maclaurin series
__device__ __forceinline__ double atan_quarter(double t)
{
  const double t2 = t * t;
  double s = fma(t2, -1.0 / 19.0, 1.0 / 17.0);
  s = fma(t2, s, -1.0 / 15.0);
  s = fma(t2, s, 1.0 / 13.0);
  s = fma(t2, s, -1.0 / 11.0);
  s = fma(t2, s, 1.0 / 9.0);
  s = fma(t2, s, -1.0 / 7.0);
  s = fma(t2, s, 1.0 / 5.0);
  s = fma(t2, s, -1.0 / 3.0);
  return fma(t * t2, s, t);
}

// half the solid angle by the formula itself; corners c as slots times kST
__device__ __noinline__ double angle(const double (&v)[3][kMaxV], int4 c, double sx, double sy, double sz)
{
  const int a = c.x / kST, b = c.y / kST, d = c.z / kST;
  const double ax = v[0][a] - sx, ay = v[1][a] - sy, az = v[2][a] - sz;
  const double bx = v[0][b] - sx, by = v[1][b] - sy, bz = v[2][b] - sz;
  const double cx = v[0][d] - sx, cy = v[1][d] - sy, cz = v[2][d] - sz;
  const double num = ax * (by * cz - bz * cy) + ay * (bz * cx - bx * cz) + az * (bx * cy - by * cx);
  const double la = sqrt(ax * ax + ay * ay + az * az);
  const double lb = sqrt(bx * bx + by * by + bz * bz);
  const double lc = sqrt(cx * cx + cy * cy + cz * cz);
  const double ab = ax * bx + ay * by + az * bz, ac = ax * cx + ay * cy + az * cz, bc = bx * cx + by * cy + bz * cz;
  return atan2(num, la * lb * lc + ab * lc + ac * lb + bc * la);
}

__global__ void __launch_bounds__(kAsmThreads, 2) solid_angle_f32_kernel(int n_vert, const float *__restrict__ V,
                                                                      int n_faces, const int32_t *__restrict__ F,
                                                                      int n_src, const float *__restrict__ S,
                                                                      float *__restrict__ M, int64_t ldm, int tiles_per)
{
  extern __shared__ double dyn[];
  double *vq = dyn, *vy = dyn + kMaxV * kST;  // [vertex][source]
  __shared__ int s_id[kMaxV], s_first[kMaxV], s_slot[kMaxV], s_nu;
  __shared__ double s_v[3][kMaxV];   // distinct vertices
  __shared__ __align__(16) double s_f[kFT][10];  // n, v1, half the squared edges of a face
  __shared__ __align__(16) int4 s_c[kFT];       // its corners' slots, times kST
  const int tid = threadIdx.x;
  const int j = tid & (kST / 2 - 1), fg = tid / (kST / 2);  // sources j and j + kST / 2
  for (int ft = blockIdx.y; ft * kFT < n_faces; ft += gridDim.y) {
    const int f0 = ft * kFT, nfc = min(kFT, n_faces - f0);
    // distinct vertices of the faces (an invalid index is one more vertex, NaN)
    __syncthreads();
    if (tid < kMaxV) {
      int v = tid < 3 * nfc ? F[3 * (size_t)f0 + tid] : F[3 * (size_t)f0];
      s_id[tid] = v >= 0 && v < n_vert ? v : -1;
    }
    __syncthreads();
    if (tid < kMaxV) {
      int k = 0;
      while (s_id[k] != s_id[tid]) ++k;
      s_first[tid] = k;
    }
    __syncthreads();
    if (tid < kMaxV) {
      int slot = 0;
      for (int k = 0; k < s_first[tid]; ++k) slot += s_first[k] == k;
      s_slot[tid] = slot;
      if (s_first[tid] == tid) {
        const int v = s_id[tid];
#pragma unroll
        for (int d = 0; d < 3; ++d) s_v[d][slot] = v < 0 ? nan("") : V[3 * (size_t)v + d];
      }
      if (tid == kMaxV - 1) {
        int nu = 0;
        for (int k = 0; k < kMaxV; ++k) nu += s_first[k] == k;
        s_nu = nu;
      }
    }
    __syncthreads();
    if (tid < nfc) {
      double v[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) v[k][d] = s_v[d][s_slot[3 * tid + k]];
      double e1[3], e2[3], e3[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        e1[d] = v[1][d] - v[0][d];
        e2[d] = v[2][d] - v[0][d];
        e3[d] = v[2][d] - v[1][d];
      }
      const double n0 = e1[1] * e2[2] - e1[2] * e2[1], n1 = e1[2] * e2[0] - e1[0] * e2[2],
                   n2 = e1[0] * e2[1] - e1[1] * e2[0];
      s_c[tid] = make_int4(s_slot[3 * tid] * kST, s_slot[3 * tid + 1] * kST, s_slot[3 * tid + 2] * kST, 0);
      s_f[tid][0] = n0;
      s_f[tid][1] = n1;
      s_f[tid][2] = n2;
#pragma unroll
      for (int d = 0; d < 3; ++d) s_f[tid][3 + d] = v[0][d];
      s_f[tid][6] = 0.5 * (e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
      s_f[tid][7] = 0.5 * (e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]);
      s_f[tid][8] = 0.5 * (e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2]);
    }
    const int nu = s_nu;
    for (int tl = 0; tl < tiles_per; ++tl) {
      const int j0 = (blockIdx.x * tiles_per + tl) * kST;
      if (j0 >= n_src) break;
      double sx[2], sy[2], sz[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int js = min(j0 + j + h * (kST / 2), n_src - 1);
        sx[h] = S[3 * (size_t)js];
        sy[h] = S[3 * (size_t)js + 1];
        sz[h] = S[3 * (size_t)js + 2];
      }
      __syncthreads();  // the face constants, or the last tile's readers
      for (int u = fg; u < nu; u += kFG) {
        const double ux = s_v[0][u], uy = s_v[1][u], uz = s_v[2][u];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double dx = ux - sx[h], dy = uy - sy[h], dz = uz - sz[h];
          const double q = fma(dz, dz, fma(dy, dy, dx * dx));
          const double y0 = (double)rsqrtf((float)q);
          const double e = fma(-q * y0, y0, 1.0);
          vq[u * kST + j + h * (kST / 2)] = q;
          vy[u * kST + j + h * (kST / 2)] = fma(0.5 * y0, e, y0);
        }
      }
      __syncthreads();
      float *row = M + (size_t)(f0 + fg) * ldm + j0 + j;
      for (int f = fg; f < nfc; f += kFG, row += kFG * ldm) {
        const int4 c = s_c[f];
        const double2 n01 = *reinterpret_cast<const double2 *>(&s_f[f][0]);
        const double2 n2v = *reinterpret_cast<const double2 *>(&s_f[f][2]);
        const double2 v12 = *reinterpret_cast<const double2 *>(&s_f[f][4]);
        const double2 c01 = *reinterpret_cast<const double2 *>(&s_f[f][6]);
        const double c2 = s_f[f][8];
        double num[2], t[2];
        bool fine[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double *pq = vq + j + h * (kST / 2), *py = vy + j + h * (kST / 2);
          const double q1 = pq[c.x], q2 = pq[c.y], q3 = pq[c.z];
          const double y1 = py[c.x], y2 = py[c.y], y3 = py[c.z];
          const double p12 = y1 * y2, p = p12 * y3;
          const double d12 = fma(0.5, q1 + q2, -c01.x), d13 = fma(0.5, q1 + q3, -c01.y), d23 = fma(0.5, q2 + q3, -c2);
          const double den = fma(d12, p12, fma(d13, y1 * y3, fma(d23, y2 * y3, 1.0)));
          num[h] = fma(n2v.y - sx[h], n01.x, fma(v12.x - sy[h], n01.y, (v12.y - sz[h]) * n2v.x)) * p;
          const double r0 = (double)__fdividef(1.0f, (float)den);
          t[h] = num[h] * fma(r0, fma(-den, r0, 1.0), r0);
          const int e1 = __double2hiint(y1), e2 = __double2hiint(y2), e3 = __double2hiint(y3);
          const int ya = min(e1, min(e2, e3)), yb = max(e1, max(e2, e3));
          fine[h] = fabs(num[h]) <= fma(0.25, den, -0.25 * kMinDen) && (unsigned)(ya - kYLow) <= kYSpan &&
                    (unsigned)(yb - ya) <= kYRatio;
        }
        double out[2];
        if (__all_sync(0xffffffffu, fine[0] && fine[1] && fabs(t[0]) < 0.02 && fabs(t[1]) < 0.02)) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const double t2 = t[h] * t[h];
            out[h] = fma(t[h] * t2, fma(t2, fma(t2, -1.0 / 7.0, 1.0 / 5.0), -1.0 / 3.0), t[h]);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) out[h] = fine[h] ? atan_quarter(t[h]) : angle(s_v, c, sx[h], sy[h], sz[h]);
        }
        if (j0 + j < n_src) row[0] = (float)(2.0 * out[0]);
        if (j0 + j + kST / 2 < n_src) row[kST / 2] = (float)(2.0 * out[1]);
      }
    }
  }
}

// rhs[f, 6b .. 6b+5] = (s, r x s) for the face's body b, zero elsewhere:
// s = (v2 - v1) x (v3 - v1) / 2, r = (v1 + v2 + v3) / 3 - y_b.  One thread
// per face writes its whole row (6 n_bodies entries).
template <typename T>
__global__ void rhs_kernel(int n_vert, const float *__restrict__ V, int n_faces, const int32_t *__restrict__ F,
                           const int32_t *__restrict__ face_body, int n_bodies, const float *__restrict__ body_pos,
                           T *__restrict__ rhs)
{
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces) return;
  const int ncol = 6 * n_bodies;
  T *row = rhs + (size_t)f * ncol;
  const int i1 = F[3 * (size_t)f], i2 = F[3 * (size_t)f + 1], i3 = F[3 * (size_t)f + 2];
  const int b = face_body[f];
  if (i1 < 0 || i1 >= n_vert || i2 < 0 || i2 >= n_vert || i3 < 0 || i3 >= n_vert || b < 0 || b >= n_bodies) {
    for (int c = 0; c < ncol; ++c) row[c] = to_out<T>(nan(""));
    return;
  }
  for (int c = 0; c < ncol; ++c) row[c] = to_out<T>(0.0);
  const double v1x = V[3 * (size_t)i1], v1y = V[3 * (size_t)i1 + 1], v1z = V[3 * (size_t)i1 + 2];
  const double v2x = V[3 * (size_t)i2], v2y = V[3 * (size_t)i2 + 1], v2z = V[3 * (size_t)i2 + 2];
  const double v3x = V[3 * (size_t)i3], v3y = V[3 * (size_t)i3 + 1], v3z = V[3 * (size_t)i3 + 2];
  const double e1x = v2x - v1x, e1y = v2y - v1y, e1z = v2z - v1z;
  const double e2x = v3x - v1x, e2y = v3y - v1y, e2z = v3z - v1z;
  const double sx = (e1y * e2z - e1z * e2y) / 2.0, sy = (e1z * e2x - e1x * e2z) / 2.0,
               sz = (e1x * e2y - e1y * e2x) / 2.0;
  const double rx = (v1x + v2x + v3x) / 3.0 - body_pos[3 * b];
  const double ry = (v1y + v2y + v3y) / 3.0 - body_pos[3 * b + 1];
  const double rz = (v1z + v2z + v3z) / 3.0 - body_pos[3 * b + 2];
  T *o = row + 6 * b;
  o[0] = to_out<T>(sx);
  o[1] = to_out<T>(sy);
  o[2] = to_out<T>(sz);
  o[3] = to_out<T>(ry * sz - rz * sy);
  o[4] = to_out<T>(rz * sx - rx * sz);
  o[5] = to_out<T>(rx * sy - ry * sx);
}

template <typename T>
cudaError_t launch(int32_t n_vert, const float *V, int32_t n_faces, const int32_t *F, const int32_t *face_body,
            int32_t n_bodies, const float *body_pos, int32_t n_src, const float *S, void *M, int64_t ldm, void *rhs,
            cudaStream_t st)
{
  if constexpr (sizeof(T) == 4) {
    const cudaError_t e =
        cudaFuncSetAttribute(solid_angle_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAsmSmem);
    if (e != cudaSuccess) return e;
    // up to 8 source tiles per block, which spread its vertex search, while
    // there are four blocks per SM
    const int64_t ftiles = (n_faces + kFT - 1) / kFT, stiles = (n_src + kST - 1) / kST;
    int per = 8;
    while (per > 1 && ftiles * ((stiles + per - 1) / per) < 4 * 148) per /= 2;
    const dim3 grid((unsigned)((stiles + per - 1) / per), (unsigned)(ftiles < 65535 ? ftiles : 65535));
    solid_angle_f32_kernel<<<grid, kAsmThreads, kAsmSmem, st>>>(n_vert, V, n_faces, F, n_src, S, (float *)M, ldm, per);
  } else {
    const dim3 grid((unsigned)((n_src + 127) / 128), (unsigned)(n_faces < 65535 ? n_faces : 65535));
    solid_angle_kernel<T><<<grid, 128, 0, st>>>(n_vert, V, n_faces, F, n_src, S, (T *)M, ldm);
  }
  if (rhs)
    rhs_kernel<T><<<(unsigned)((n_faces + 127) / 128), 128, 0, st>>>(n_vert, V, n_faces, F, face_body, n_bodies,
                                                                       body_pos, (T *)rhs);
  return cudaGetLastError();
}

}  // namespace

extern "C" mbc_status mbc_mesh_assemble(int32_t n_vert, const float *V, int32_t n_faces, const int32_t *F,
                                        const int32_t *face_body, int32_t n_bodies, const float *body_pos,
                                        int32_t n_src, const float *S, int32_t dtype, void *M, int64_t ldm,
                                        void *rhs, mbc_stream stream)
{
  if (n_vert <= 0 || n_faces <= 0 || n_src <= 0 || !V || !F || !S || !M)
    return mbc::fail(MBC_BAD_ARG, "mbc_mesh_assemble: NULL pointer or non-positive size");
  if (ldm < n_src) return mbc::fail(MBC_BAD_ARG, "mbc_mesh_assemble: ldm below n_src");
  if (dtype != MBC_F32 && dtype != MBC_F64) return mbc::fail(MBC_BAD_ARG, "mbc_mesh_assemble: dtype must be MBC_F32 or MBC_F64");
  if (rhs && (n_bodies <= 0 || !face_body || !body_pos))
    return mbc::fail(MBC_BAD_ARG, "mbc_mesh_assemble: the right-hand side needs face_body, n_bodies and body_pos");
  const cudaStream_t st = (cudaStream_t)stream;
  const cudaError_t e =
      dtype == MBC_F64
          ? launch<double>(n_vert, V, n_faces, F, face_body, n_bodies, body_pos, n_src, S, M, ldm, rhs, st)
          : launch<float>(n_vert, V, n_faces, F, face_body, n_bodies, body_pos, n_src, S, M, ldm, rhs, st);
  if (e != cudaSuccess) return mbc::fail(MBC_CUDA_ERROR, std::string("mbc_mesh_assemble: ") + cudaGetErrorString(e));
  return MBC_OK;
}
