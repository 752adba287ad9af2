// Tensor-core form of the DFT: the kernel over a plan's records (the method is
// in dft_tc.cuh), its choice and launch.
#include <algorithm>

#include "dft_tc.cuh"

namespace obit {

namespace {

// kMix: a Gaussian-family model whose untapered rows come first as points
// (p.k.compsPt, p.k.ncompPt).
template <int MA, int NJ, int T, int EX, bool kCross, int kMix>
__global__ void __launch_bounds__(32 * T, 12 / T)
    dft_tc_kernel(const __grid_constant__ TcParams p) {
  extern __shared__ __align__(16) float smem[];
  float* sTab = smem;
  float2* sScale = reinterpret_cast<float2*>(sTab + T * tc_tab_floats(NJ, T));
  float2* sL2 = sScale + 2 * T * T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const long long nItems = (long long)p.k.nvis * p.nteam;
  for (long long item = blockIdx.x; item < nItems; item += gridDim.x) {
    const int row = (int)(item / p.nteam);
    const TcTeamDesc& tm = p.teams[item - (long long)row * p.nteam];
    float* rec = p.k.vis + (size_t)(p.k.rowBase + row) * p.k.lrec;
    const float u = rec[p.k.ilocu], v = rec[p.k.ilocv], w = rec[p.k.ilocw];
    TcSums<MA, NJ> S;
#pragma unroll
    for (int i = 0; i < MA * NJ * 4; i++) (&S.tot[0][0][0][0])[i] = 0ull;
    if constexpr (kMix != 0)
      tc_pass<MA, NJ, T, kExSpec, (kMix == 2), false>(p, tm, p.k.compsPt, nullptr, p.k.ncompPt, 4, u, v, w, sTab, sScale,
                                               sL2, S);
    tc_pass<MA, NJ, T, EX, kCross, false>(p, tm, p.k.comps, p.k.compsLo, p.k.ncomp, p.specField, u, v, w, sTab, sScale, sL2,
                                   S);
    // every warp has read u, v, w and applies its own channels
    const TcSeg& seg = tm.seg[warp];
#pragma unroll
    for (int mi = 0; mi < MA; mi++)
#pragma unroll
      for (int j = 0; j < NJ; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int a = 16 * mi + g + 8 * (e >> 1), n = 8 * j + 2 * t + (e & 1);
          const int ch = seg.ch0 + tm.D * a + n;
          float sr, si;
          {
            float x[2], y[2];
            up2(S.tot[mi][j][0][e >> 1], x[0], x[1]);
            up2(S.tot[mi][j][1][e >> 1], y[0], y[1]);
            sr = x[e & 1];
            si = y[e & 1];
          }
          if (S.merged) {
            const int i0 = ((mi * NJ + j) * 2) * 4 + e;
            const float2 lr = sL2[i0 * (32 * T) + threadIdx.x], li = sL2[(i0 + 4) * (32 * T) + threadIdx.x];
            sr = lr.x + (lr.y + sr);
            si = li.x + (li.y + si);
          }
          if (ch < seg.end) apply_channel(p.k, rec + p.chanOff[ch], sr, si);
        }
  }
}

using TcFn = void (*)(const TcParams);

template <int MA, int NJ, int T>
TcFn tc_pick_shape(int kind, bool crossPt, int mixed) {
  switch (kind) {
    case kPoint: return dft_tc_kernel<MA, NJ, T, kExNone, false, 0>;
    case kPointSpec:
      return crossPt ? dft_tc_kernel<MA, NJ, T, kExSpec, true, 0> : dft_tc_kernel<MA, NJ, T, kExSpec, false, 0>;
    case kGauss: return dft_tc_kernel<MA, NJ, T, kExGauss, true, 0>;
    case kGaussSpec:
      if (mixed) return crossPt ? dft_tc_kernel<MA, NJ, T, kExBoth, true, 2> : dft_tc_kernel<MA, NJ, T, kExBoth, true, 1>;
      return dft_tc_kernel<MA, NJ, T, kExBoth, true, 0>;
  }
  return nullptr;
}

TcFn tc_pick(const TcPlan& pl) {
  if (pl.MA == 2 && pl.NJ == 2 && pl.T == 2) return tc_pick_shape<2, 2, 2>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 2 && pl.NJ == 2 && pl.T == 1) return tc_pick_shape<2, 2, 1>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 1 && pl.NJ == 2 && pl.T == 1) return tc_pick_shape<1, 2, 1>(pl.kind, pl.crossPt, pl.mixed);
  if (pl.MA == 1 && pl.NJ == 1 && pl.T == 1) return tc_pick_shape<1, 1, 1>(pl.kind, pl.crossPt, pl.mixed);
  return nullptr;
}

}  // namespace

int tc_finalize(TcPlan* plan, const KParams& base, std::string* err) {
  cudaError_t ce;
  if (plan->beam) {
    if (int rc = tc_beam_prepare(*plan, &plan->gridCap, err)) return rc;
  } else {
    TcFn fn = tc_pick(*plan);
    if (!fn) {
      *err = "no tensor-core kernel for this shape";
      return 3;
    }
    if (int rc = tc_resident((const void*)fn, 32 * plan->T, tc_smem_floats(plan->MA, plan->NJ, plan->T) * sizeof(float),
                             &plan->gridCap, err))
      return rc;
  }
  const size_t bt = sizeof(TcTeamDesc) * plan->teams.size(), bc = (sizeof(int) * plan->chanOff.size() + 15) & ~size_t(15),
               be = sizeof(float) * plan->expo.size();
  const size_t bt16 = (bt + 15) & ~size_t(15);
  if ((ce = cudaMalloc(&plan->d_mem, bt16 + bc + be + 16)) != cudaSuccess) {
    plan->d_mem = nullptr;
    *err = std::string("cudaMalloc tensor-core plan: ") + cudaGetErrorString(ce);
    return 2;
  }
  char* d = (char*)plan->d_mem;
  if ((ce = cudaMemcpy(d, plan->teams.data(), bt, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (ce = cudaMemcpy(d + bt16, plan->chanOff.data(), sizeof(int) * plan->chanOff.size(), cudaMemcpyHostToDevice)) !=
          cudaSuccess ||
      (be && (ce = cudaMemcpy(d + bt16 + bc, plan->expo.data(), be, cudaMemcpyHostToDevice)) != cudaSuccess)) {
    *err = std::string("tensor-core plan copy: ") + cudaGetErrorString(ce);
    return 2;
  }
  TcParams& q = plan->kp;
  q = TcParams{};
  q.k = base;
  q.teams = reinterpret_cast<const TcTeamDesc*>(d);
  q.nteam = (int)plan->teams.size();
  q.chanOff = reinterpret_cast<const int*>(d + bt16);
  q.expo = reinterpret_cast<const float*>(d + bt16 + bc);
  q.lay = tc_expo_layout(plan->MA, plan->NC);
  q.specField = (plan->kind == kGaussSpec) ? 7 : kSpecIndexField;
  return 0;
}

int tc_finalize_all(std::vector<TcPlan>* plan, const KParams& base, std::string* err) {
  for (TcPlan& p : *plan)
    if (int rc = tc_finalize(&p, base, err)) return rc;
  return 0;
}

void tc_free(std::vector<TcPlan>* plan) {
  for (TcPlan& p : *plan)
    if (p.d_mem) cudaFree(p.d_mem);
  plan->clear();
}

int tc_launch(const TcPlan& plan, const ModelDesc& model, float* d_vis, int nvis, const float* d_comps, int* d_err,
              cudaStream_t stream, std::string* err) {
  if (nvis <= 0 || model.ncomp <= 0) return 0;
  TcParams q = plan.kp;
  q.k.vis = d_vis;
  q.k.nvis = nvis;
  q.k.rowBase = 0;
  q.k.errFlag = d_err;
  q.k.ncomp = model.ncomp;
  q.k.comps = d_comps;
  q.k.compsPt = nullptr;
  q.k.ncompPt = 0;
  if (plan.mixed) {
    q.k.compsPt = d_comps;
    q.k.ncompPt = model.ncompPt;
    q.k.comps = d_comps + (size_t)model.ncompPt * q.k.cstride;
  }
  const long long items = (long long)nvis * q.nteam;
  const int grid = (int)std::min<long long>(items, (long long)plan.gridCap);
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    *err = std::string("error pending before the kernel launch: ") + cudaGetErrorString(ce);
    return 2;
  }
  const size_t smem = tc_smem_floats(plan.MA, plan.NJ, plan.T) * sizeof(float);
  tc_pick(plan)<<<grid, 32 * plan.T, smem, stream>>>(q);
  if ((ce = cudaGetLastError()) != cudaSuccess) {
    *err = std::string("tensor-core kernel launch: ") + cudaGetErrorString(ce);
    return 2;
  }
  return 0;
}

}  // namespace obit
