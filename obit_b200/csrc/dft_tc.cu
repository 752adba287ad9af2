// Tensor-core form of the DFT: the kernel over a plan's records (the method is
// in dft_tc.cuh), its choice and launch.
#include <algorithm>

#include "dft_tc.cuh"

namespace obit {

namespace {

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
  if (pl.kind == kPointTSpec || pl.kind == kGaussTSpec) return tc_pick_tab(pl);
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
  q.specField = (plan->kind == kGaussSpec || plan->kind == kGaussTSpec) ? 7 : kSpecIndexField;
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
