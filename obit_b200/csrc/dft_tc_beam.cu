// Tensor-core form of the beam-corrected DFT (the method is in dft_tc.cuh): the
// rows are 16 MA blocks of 8 channels, the columns the 8 channels of a block
// for each model correlation, so a component costs 16 MA + 8 phasors and 8 NJ
// complex products with its Jones coefficients for 128 MA channels and NJ
// correlations.  The coefficients are formed from the two antennas' Jones
// matrices once per (record, component, segment), by the lane that holds the
// component.  8,064 records x 1,024 channels x 4,000 points with an index, four
// correlations, three Jones planes: 17.7 ms against 30.7 of the form with a phasor
// per channel (dft_beam_mma.cu).
#include <algorithm>

#include "dft_tc.cuh"

namespace obit {

namespace {

template <int MA, int NJ, int EX, bool kCross, int kMix>
__global__ void __launch_bounds__(32, (MA * NJ > 4 ? 8 : 12))
    dft_tc_beam_kernel(const __grid_constant__ TcBeamParams bp) {
  extern __shared__ __align__(16) float smem[];
  const TcParams& p = bp.t;
  const BeamKParams& b = bp.b;
  float* sTab = smem;
  float2* sScale = reinterpret_cast<float2*>(sTab + tc_tab_floats(NJ, 1));
  float2* sL2 = sScale + 2;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const long long nItems = (long long)p.k.nvis * p.nteam;
  for (long long item = blockIdx.x; item < nItems; item += gridDim.x) {
    const int row = (int)(item / p.nteam);
    const TcTeamDesc& tm = p.teams[item - (long long)row * p.nteam];
    float* rec = p.k.vis + (size_t)(p.k.rowBase + row) * p.k.lrec;
    int a1, a2;
    beam_ants(b, rec, a1, a2);
    if (a1 < 0 || a1 >= b.numAnt || a2 < 0 || a2 >= b.numAnt) {
      if (lane == 0 && p.k.errFlag) atomicExch(p.k.errFlag, 3);
      continue;
    }
    const int ta = b.antType[a1], tc = b.antType[a2];
    const float u = rec[p.k.ilocu], v = rec[p.k.ilocv], w = rec[p.k.ilocw];
    TcSums<MA, NJ> S;
#pragma unroll
    for (int i = 0; i < MA * NJ * 4; i++) (&S.tot[0][0][0][0])[i] = 0ull;
    if constexpr (kMix != 0)
      tc_pass<MA, NJ, 1, kExSpec, (kMix == 2), true>(p, tm, p.k.compsPt, nullptr, p.k.ncompPt, 4, u, v, w, sTab, sScale,
                                                     sL2, S, &b, bp.perm, ta, tc);
    tc_pass<MA, NJ, 1, EX, kCross, true>(p, tm, p.k.comps, p.k.compsLo, p.k.ncomp, p.specField, u, v, w, sTab, sScale,
                                         sL2, S, &b, (kMix != 0) ? bp.perm + p.k.ncompPt : bp.perm, ta, tc);
    const TcSeg& seg = tm.seg[0];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      const int q = tc_corr(NJ, j);
      const int slot = (q == 0) ? 0 : (q == 1) ? 2 : (q == 2) ? 3 : 1;  // records hold XX, YY, XY, YX
      if (slot >= b.ncorr) continue;
      const float pf = b.polFact[slot];
#pragma unroll
      for (int mi = 0; mi < MA; mi++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int a = 16 * mi + g + 8 * (e >> 1), n = 2 * t + (e & 1);
          const int ch = seg.ch0 + tm.D * a + n;
          float x[2], y[2];
          up2(S.tot[mi][j][0][e >> 1], x[0], x[1]);
          up2(S.tot[mi][j][1][e >> 1], y[0], y[1]);
          float Mr = x[e & 1], Mi = y[e & 1];
          if (S.merged) {
            const int i0 = ((mi * NJ + j) * 2) * 4 + e;
            const float2 lr = sL2[i0 * 32 + threadIdx.x], li = sL2[(i0 + 4) * 32 + threadIdx.x];
            Mr = lr.x + (lr.y + Mr);
            Mi = li.x + (li.y + Mi);
          }
          if (ch >= seg.end) continue;
          Mr *= pf;
          Mi *= pf;
          float* o = rec + p.chanOff[ch] + slot * p.k.incs;
          if (o[2] <= 0.0f && p.k.op != kOpRepl) continue;
          if (p.k.op == kOpRepl) {
            o[0] = Mr;
            o[1] = Mi;
          } else if (p.k.op == kOpDiv) {
            const float m2 = Mr * Mr + Mi * Mi;
            const float Vr = o[0], Vi = o[1];
            o[0] = (Vr * Mr + Vi * Mi) / m2;
            o[1] = (Vi * Mr - Vr * Mi) / m2;
          } else {
            o[0] -= Mr;
            o[1] -= Mi;
          }
        }
    }
  }
}

using TcBeamFn = void (*)(const TcBeamParams);

template <int MA, int NJ>
TcBeamFn pick_shape(int kind, bool crossPt, int mixed) {
  switch (kind) {
    case kPoint: return dft_tc_beam_kernel<MA, NJ, kExNone, false, 0>;
    case kPointSpec:
      return crossPt ? dft_tc_beam_kernel<MA, NJ, kExSpec, true, 0> : dft_tc_beam_kernel<MA, NJ, kExSpec, false, 0>;
    case kGauss: return dft_tc_beam_kernel<MA, NJ, kExGauss, true, 0>;
    case kGaussSpec:
      if (mixed)
        return crossPt ? dft_tc_beam_kernel<MA, NJ, kExBoth, true, 2> : dft_tc_beam_kernel<MA, NJ, kExBoth, true, 1>;
      return dft_tc_beam_kernel<MA, NJ, kExBoth, true, 0>;
  }
  return nullptr;
}

TcBeamFn pick(const TcPlan& pl) {
  if (pl.MA == 2 && pl.NJ == 4) return pick_shape<2, 4>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 1 && pl.NJ == 4) return pick_shape<1, 4>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 2 && pl.NJ == 2) return pick_shape<2, 2>(pl.kind, pl.crossPt, pl.mixed);
  return nullptr;
}

}  // namespace

int tc_beam_prepare(const TcPlan& plan, int* gridCap, std::string* err) {
  TcBeamFn fn = pick(plan);
  if (!fn) {
    *err = "no tensor-core beam kernel for this shape";
    return 3;
  }
  return tc_resident((const void*)fn, 32, tc_smem_floats(plan.MA, plan.NJ, 1) * sizeof(float), gridCap, err);
}

int tc_beam_launch(const TcPlan& plan, const ModelDesc& model, const BeamKParams& beam, const int* perm,
                   const float* d_comps, cudaStream_t stream, std::string* err) {
  if (beam.k.nvis <= 0 || model.ncomp <= 0) return 0;
  TcBeamParams q;
  q.t = plan.kp;
  q.b = beam;
  q.perm = perm;
  q.t.k.vis = beam.k.vis;
  q.t.k.nvis = beam.k.nvis;
  q.t.k.rowBase = beam.k.rowBase;
  q.t.k.errFlag = beam.k.errFlag;
  q.t.k.ncomp = model.ncomp;
  q.t.k.comps = d_comps + (size_t)(plan.mixed ? model.ncompPt : 0) * q.t.k.cstride;
  q.t.k.compsPt = plan.mixed ? d_comps : nullptr;
  q.t.k.ncompPt = plan.mixed ? model.ncompPt : 0;
  const long long items = (long long)beam.k.nvis * q.t.nteam;
  const int grid = (int)std::min<long long>(items, (long long)plan.gridCap);
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    *err = std::string("error pending before the beam kernel launch: ") + cudaGetErrorString(ce);
    return 2;
  }
  pick(plan)<<<grid, 32, tc_smem_floats(plan.MA, plan.NJ, 1) * sizeof(float), stream>>>(q);
  if ((ce = cudaGetLastError()) != cudaSuccess) {
    *err = std::string("tensor-core beam kernel launch: ") + cudaGetErrorString(ce);
    return 2;
  }
  return 0;
}

}  // namespace obit
