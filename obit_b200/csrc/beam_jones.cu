// Jones matrices of every (antenna type, component, beam plane) interpolated
// from beam images: the computation of GetJonesKernel
// (ObitCUDABeamModel.cu:1228-1299) with its pixel geometry (CUDAPositionXYpix,
// CUDASkyGeom.h:91-286; linear grids and the eight projections) and Lagrange interpolator
// (CUDABeamInterpPixel / SetConvKernal, CUDABeamInterp.h), written anew.
// The position, its pixel, the interpolation weights and the primary-beam
// factor's offset are computed once per component, then every plane's 8 images
// are interpolated with the same taps.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <string>

#include "abi_internal.h"
#include "obit_dft.h"

namespace obit {
namespace {

constexpr int kMaxTaps = 9;  // 2 hwidth + 1, hwidth <= 4

struct JonesParams {
  int numAntType, nx, ny, nplane, ncomp, hwidth, projection;
  float fblank, refSizeFact, parAng, crota;
  double crval0, crval1;
  float crpix0, crpix1, cdelt0, cdelt1;
  const float* pixels;
  const float* pos;
  float* jones;
  float planeFreq[64];
};
constexpr int kMaxPlanes = 64;

// Offsets (deg) of a position (deg) from the grid's reference position in
// the grid's projection, or false where it cannot be projected: the linear
// offsets after the 0 h wrap, or for projections 1..8 (-SIN, -TAN, -ARC,
// -NCP, -GLS, -MER, -AIT, -STG) the projected coordinates of the standard
// AIPS definitions scaled back to degrees, as CUDAPositionXYpixLM
// (CUDASkyGeom.h:91-250) forms them; crota (deg) enters only the -MER and
// -AIT scale factors.
__device__ bool grid_offsets(const JonesParams& p, double x, double y, double& l, double& m) {
  const double d2r = 1.745329252e-2, halfPi = 6.28318530717959 / 4.0, eps = 1.0e-5;
  const double dx = x - p.crval0;
  if (dx > 180.0) x -= 360.0;
  if (dx < -180.0) x += 360.0;
  l = x - p.crval0;
  m = y - p.crval1;
  if (p.projection == 0) return true;
  const double ra0 = p.crval0 * d2r, dec0 = p.crval1 * d2r, ra = x * d2r, dec = y * d2r;
  const double cd = cos(dec), sd = sin(dec), cd0 = cos(dec0), sd0 = sin(dec0);
  const double da = ra - ra0, ca = cos(da);
  const double cosAlt = sd * sd0 + cd * cd0 * ca;  // cosine of the angle from the reference
  const double mNorth = sd * cd0 - cd * sd0 * ca;   // north component of the direction
  double L = sin(da) * cd, M = 0.0;
  switch (p.projection) {
    case 1:  // -SIN: orthographic
      if (cosAlt < 0.0) return false;
      M = mNorth;
      break;
    case 2:  // -TAN: gnomonic
      if (cosAlt <= 0.0) return false;
      L /= cosAlt;
      M = mNorth / cosAlt;
      break;
    case 3: {  // -ARC: zenithal equidistant
      const double th = acos(fmin(1.0, fmax(-1.0, cosAlt)));
      const double f = th != 0.0 ? th / sin(th) : 1.0;
      L *= f;
      M = mNorth * f;
      break;
    }
    case 4:  // -NCP: north celestial pole
      if (dec0 == 0.0) return false;
      M = (cd0 - cd * ca) / sd0;
      break;
    case 5:  // -GLS: global sinusoid
      if (fabs(dec) > halfPi || fabs(dec0) > halfPi) return false;
      L = da * cd;
      M = dec - dec0;
      break;
    case 6: {  // -MER: Mercator, scaled to the grid's increment along y
      const double r = p.crota * d2r;
      double step = p.cdelt1 * cos(r) + p.cdelt0 * sin(r);
      if (step == 0.0) step = 1.0;
      const double y0 = (p.crval1 / 2.0 + 45.0) * d2r;
      const double ly0 = log(tan(y0)), ly1 = log(tan(y0 + step / 2.0 * d2r));
      const double gy = step * d2r / (ly1 - ly0);
      double gx = cos(p.crval1 * d2r);
      if (gx <= 0.0) gx = 1.0;
      const double t = tan(dec / 2.0 + halfPi / 2.0);
      if (t < eps) return false;
      L = gx * da;
      M = gy * log(t) - gy * ly0;
      break;
    }
    case 7: {  // -AIT: Hammer-Aitoff, scaled to the grid's increments
      const double half = da / 2.0;
      if (fabs(half) > halfPi) return false;
      const double r = p.crota * d2r, cr = cos(r), sr = sin(r);
      const double yc = p.crval1 * d2r;
      double sy = p.cdelt1 * cr + p.cdelt0 * sr;
      if (sy == 0.0) sy = 1.0;
      sy *= d2r;
      double ny = sin(yc + sy) / sqrt((1.0 + cos(yc + sy)) / 2.0) - sin(yc) / sqrt((1.0 + cos(yc)) / 2.0);
      if (ny == 0.0) ny = 1.0;
      const double gy = sy / ny;
      double sx = p.cdelt0 * cr - p.cdelt1 * sr;
      if (sx == 0.0) sx = 1.0;
      sx *= d2r;
      double nx = 2.0 * cos(yc) * sin(sx / 2.0);
      if (nx == 0.0) nx = 1.0;
      const double gx = sx * sqrt((1.0 + cos(yc) * cos(sx / 2.0)) / 2.0) / nx;
      const double y0 = gy * sin(yc) / sqrt((1.0 + cos(yc)) / 2.0);
      const double z = sqrt((1.0 + cd * cos(half)) / 2.0);
      if (fabs(z) < eps) return false;
      L = 2.0 * gx * cd * sin(half) / z;
      M = gy * sd / z - y0;
      break;
    }
    case 8: {  // -STG: stereographic
      if (fabs(dec) > halfPi) return false;
      const double den = 1.0 + cosAlt;
      if (fabs(den) < eps) return false;
      L *= 2.0 / den;
      M = mNorth * 2.0 / den;
      break;
    }
    default:
      return false;
  }
  l = L / d2r;
  m = M / d2r;
  return true;
}

// Pixel (1-relative) of a position (deg), or false when it cannot be
// projected: the grid offsets rotated by the parallactic angle, then the
// grid's increments and reference pixel (CUDAPositionXYpix,
// CUDASkyGeom.h:266-286).
__device__ bool pixel_of(const JonesParams& p, double x, double y, float& px, float& py) {
  double l, m;
  if (!grid_offsets(p, x, y, l, m)) return false;
  float sr, cr;
  sincosf(p.parAng, &sr, &cr);
  const double lr = l * cr + m * sr;
  const double mr = m * cr - l * sr;
  px = (float)(lr / p.cdelt0 + p.crpix0);
  py = (float)(mr / p.cdelt1 + p.crpix1);
  return true;
}

// First (0-relative) of the taps about pixel pix (1-relative) on an axis of n pixels.
__device__ int first_tap(float pix, int n, int hw) {
  const int iwid = 2 * hw + 1;
  const int cen = (int)(pix + 0.5f) - hw;
  return max(1, min(cen, n - iwid + 1)) - 1;
}

// Lagrange weight of tap j of iwid whose first is `start`.
__device__ float lagrange_weight(float pix, int start, int iwid, int j) {
  const float xx = pix - (float)start;  // 1 at the first tap
  float prod = 1.0f, den = 1.0f;
  for (int i = 0; i < iwid; i++)
    if (i != j) {
      prod *= xx - (float)(i + 1);
      den *= (float)(j - i);
    }
  return prod / den;
}

// Inverse square root of the cos^2 primary-beam gain at offset ang (deg):
// InvBeam (ObitCUDABeamModel.cu:66-72), 100 past the 10 % point.
__device__ float inv_beam(float fact, float freq, float ang) {
  const double arg = (double)fact * freq * ang;
  if (arg > 1.02) return 100.0f;
  return (float)((1.0 - 4.0 * arg * arg) / cos(3.141592653589793 * arg));
}

// a blank interpolant in the exchange between lanes: a NaN no arithmetic produces
constexpr int kBlankBits = 0x7fc0beef;

// Units: one interpolation of (component, plane, image).  A CTA takes CB
// components of one antenna type: a thread per component finds the pixel, a
// thread per tap its weight on an axis, all threads the (offset, weight) table, then eight lanes share a unit, each every eighth tap, and at last a
// thread per (component, plane) applies the gain and the limits.  The images
// come from L2 (1.9 MB at 2 types x 8 planes x 61 x 61 pixels); a warp's load
// touches 4 units of two rows each.  A thread per (component, type) over all
// planes, images and taps kept 8,000 threads on 200 dependent loads a plane:
// 160 us for 4,000 components x 2 types x 8 planes of 61 x 61 pixels, now 35.
constexpr int kJonesThreads = 256;
constexpr int kMaxCB = 32;

__host__ __device__ inline int jones_comps_per_cta(int nplane) {
  const int cb = 2 * kJonesThreads / (8 * nplane);
  return cb < 1 ? 1 : (cb > kMaxCB ? kMaxCB : cb);
}

__global__ void __launch_bounds__(kJonesThreads) beam_jones_kernel(const __grid_constant__ JonesParams p) {
  __shared__ float sW[kMaxCB][2][kMaxTaps];
  __shared__ int sFirst[kMaxCB];  // offset of the first tap, or -1 off the grid
  __shared__ float sAng[kMaxCB], sSum[kMaxCB], sPix[kMaxCB][2];
  extern __shared__ __align__(8) float dynJ[];
  const int CB = jones_comps_per_cta(p.nplane);
  const int iwid = 2 * p.hwidth + 1, ntap = iwid * iwid;
  float2* sTap = reinterpret_cast<float2*>(dynJ);           // [CB][ntap]: offset (as bits), weight
  float* sV = dynJ + 2 * CB * ntap;                         // [CB][nplane][8]
  const int c0 = blockIdx.x * CB, t = blockIdx.y;
  const int nc = min(CB, p.ncomp - c0);
  if ((int)threadIdx.x < nc) {
    const int i = threadIdx.x, c = c0 + i;
    const double x = p.pos[2 * c], y = p.pos[2 * c + 1];
    float px, py;
    const bool onGrid = pixel_of(p, x, y, px, py) && px >= 1.0f && px <= (float)p.nx && py >= 1.0f &&
                        py <= (float)p.ny;
    sFirst[i] = onGrid ? first_tap(py, p.ny, p.hwidth) * p.nx + first_tap(px, p.nx, p.hwidth) : -1;
    sPix[i][0] = px;
    sPix[i][1] = py;
    sAng[i] = sqrtf((float)(x * x + y * y));
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * 2 * iwid; e += kJonesThreads) {  // a thread per tap of an axis
    const int i = e / (2 * iwid), r = e - i * 2 * iwid, ax = r >= iwid, j = ax ? r - iwid : r;
    if (sFirst[i] >= 0) {
      const float pix = sPix[i][ax];
      sW[i][ax][j] = lagrange_weight(pix, first_tap(pix, ax ? p.ny : p.nx, p.hwidth), iwid, j);
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < nc && sFirst[threadIdx.x] >= 0) {
    const int i = threadIdx.x;
    float s = 0.f;
    for (int j = 0; j < iwid; j++)
      for (int k = 0; k < iwid; k++) s += sW[i][0][k] * sW[i][1][j];
    sSum[i] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * ntap; e += kJonesThreads) {
    const int i = e / ntap, k = e - i * ntap, j = k / iwid, m = k - j * iwid;
    if (sFirst[i] >= 0)
      sTap[e] = make_float2(__int_as_float(sFirst[i] + j * p.nx + m), sW[i][0][m] * sW[i][1][j]);
  }
  __syncthreads();
  // eight lanes per unit: lane group (image q, and a start within the component
  // and plane pairs), each lane taps l, l + 8, ...
  const int plane = p.ny * p.nx, l = threadIdx.x & 7, q = (threadIdx.x >> 3) & 7;
  const float* image = p.pixels + ((size_t)t * 8 + q) * p.nplane * plane;
  constexpr int kSide = kJonesThreads / 64;  // (component, plane) pairs side by side
  int i = 0, k = threadIdx.x >> 6;
  for (int ck0 = 0; ck0 < nc * p.nplane; ck0 += kSide, k += kSide) {
    while (k >= p.nplane) {
      k -= p.nplane;
      i++;
    }
    const bool have = i < nc && sFirst[min(i, kMaxCB - 1)] >= 0;
    float sum = 0.f, sumwt = 0.f;
    bool blank = false;
    if (have) {
      const float* d = image + (size_t)k * plane;
      const float2* tap = sTap + i * ntap;
      for (int e0 = l; e0 < ntap; e0 += 32) {  // four loads in flight per lane
        float val[4], w[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {  // (past the last tap: the first again, of no weight)
          const bool on = e0 + 8 * m < ntap;
          const float2 tw = tap[on ? e0 + 8 * m : l];
          w[m] = on ? tw.y : 0.f;
          val[m] = __ldg(d + __float_as_int(tw.x));
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const bool ok = val[m] != p.fblank;
          blank = blank || !ok;
          const float wt = ok ? w[m] : 0.f;
          sumwt += wt;
          sum += (ok ? val[m] : 0.f) * wt;
        }
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float wt = have ? sSum[i] : 1.f;
    if (__any_sync(0xffffffffu, blank)) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) sumwt += __shfl_xor_sync(0xffffffffu, sumwt, o);
      wt = sumwt;
    }
    if (have && l == 0) sV[(i * p.nplane + k) * 8 + q] = wt > 0.90f ? sum / wt : __int_as_float(kBlankBits);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nc * p.nplane; e += kJonesThreads) {
    const int i = e / p.nplane, k = e - i * p.nplane;
    float* J = p.jones + (((size_t)t * p.ncomp + c0 + i) * p.nplane + k) * 8;
    bool unit = sFirst[i] < 0;
    float v[8], g = 0.f;
    if (!unit) {
      g = inv_beam(p.refSizeFact, p.planeFreq[k], sAng[i]);
      for (int q = 0; q < 8; q++) {
        v[q] = sV[e * 8 + q];
        unit = unit || __float_as_int(v[q]) == kBlankBits;
      }
      unit = unit || !(g < 10.0f) || !(fabsf(g * v[0]) <= 1.3f) || !(fabsf(g * v[2]) <= 1.3f);
    }
    // cudaMatxSet2C order: P1, X1, X2, P2 (XX, XY, YX, YY)
    float4* J4 = reinterpret_cast<float4*>(J);
    J4[0] = unit ? make_float4(1.f, 0.f, 0.f, 0.f) : make_float4(g * v[0], g * v[1], g * v[4], g * v[5]);
    J4[1] = unit ? make_float4(0.f, 0.f, 1.f, 0.f) : make_float4(g * v[6], g * v[7], g * v[2], g * v[3]);
  }
}

}  // namespace
}  // namespace obit

extern "C" int obit_dft_beam_jones(const ObitDFTBeamImages* im, const float* pos, int ncomp, float parAng,
                                   float* jones, void* stream) {
  using namespace obit;
  set_last_error("");
  auto bad = [](int code, const char* msg) {
    set_last_error(msg);
    return code;
  };
  if (!im || !pos || !jones || !im->pixels || !im->planeFreq) return bad(OBIT_DFT_EBADARG, "NULL beam-image argument");
  if (ncomp < 0) return bad(OBIT_DFT_EBADARG, "negative component count");
  if (im->numAntType < 1 || im->nplane < 1) return bad(OBIT_DFT_EBADARG, "no antenna types or planes");
  if (im->nplane > kMaxPlanes) return bad(OBIT_DFT_EUNSUPPORTED, "more than 64 beam planes");
  if (im->hwidth < 1 || im->hwidth > 4) return bad(OBIT_DFT_EBADARG, "interpolation half-width must be 1..4");
  if (im->nx < 2 * im->hwidth + 1 || im->ny < 2 * im->hwidth + 1)
    return bad(OBIT_DFT_EBADARG, "beam images smaller than the interpolation kernel");
  if (im->projection < 0 || im->projection > 8) return bad(OBIT_DFT_EUNSUPPORTED, "projection must be 0..8");
  if (!(im->cdelt[0] != 0.0f) || !(im->cdelt[1] != 0.0f)) return bad(OBIT_DFT_EBADARG, "zero pixel increment");
  if (((uintptr_t)jones & 15u) != 0) return bad(OBIT_DFT_EBADARG, "Jones table not 16-byte aligned");
  if (ncomp == 0) return OBIT_DFT_OK;
  JonesParams p{};
  p.numAntType = im->numAntType;
  p.nx = im->nx;
  p.ny = im->ny;
  p.nplane = im->nplane;
  p.ncomp = ncomp;
  p.hwidth = im->hwidth;
  p.projection = im->projection;
  p.fblank = im->fblank;
  p.refSizeFact = im->refSizeFact;
  p.parAng = parAng;
  p.crval0 = im->crval[0];
  p.crval1 = im->crval[1];
  p.crpix0 = im->crpix[0];
  p.crpix1 = im->crpix[1];
  p.cdelt0 = im->cdelt[0];
  p.cdelt1 = im->cdelt[1];
  p.crota = im->crota;
  p.pixels = im->pixels;
  p.pos = pos;
  p.jones = jones;
  for (int k = 0; k < im->nplane; k++) p.planeFreq[k] = im->planeFreq[k];
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return bad(OBIT_DFT_ECUDA, cudaGetErrorString(ce));
  const int cb = jones_comps_per_cta(p.nplane), iwid = 2 * p.hwidth + 1;
  const dim3 grid((unsigned)((ncomp + cb - 1) / cb), (unsigned)im->numAntType);
  const size_t smem = sizeof(float) * ((size_t)2 * cb * iwid * iwid + (size_t)cb * p.nplane * 8);
  beam_jones_kernel<<<grid, kJonesThreads, smem, (cudaStream_t)stream>>>(p);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    set_last_error(std::string("beam Jones kernel launch: ") + cudaGetErrorString(ce));
    return OBIT_DFT_ECUDA;
  }
  return OBIT_DFT_OK;
}
