// Tensor-core form of the DFT model (dft_tc.cu): plan types shared by the host
// planner (dft_tc_plan.cpp, plain C++) and the kernel.
#pragma once
#include <functional>
#include <string>
#include <vector>

#include "dft_beam.h"
#include "dft_plan.h"

namespace obit {

constexpr int kTcChunk = 32;     // components per folded chunk
constexpr int kTcMaxTeam = 2;    // warps (segments) of one record sharing its (record, component) work
constexpr int kTcMinComps = 48;  // below this the recurrence kernels run (chunks would be mostly padding)

// One warp's share of a record: a grid of rows x columns of channels,
// channel(a, n) = ch0 + D a + n, valid below end.  Frequencies
// are ratios to the data's reference frequency divided by 2 pi, so that a
// product with X u + Y v + Z w is in turns.
struct TcSeg {
  float fa_hi, fa_lo;  // anchor: row 8 (MA - 1) + 4, column 4
  int ch0;             // channel-list index of row 0, column 0; column n is n channels on
  int end;             // first channel-list index past the segment (<= ch0: an empty segment)
  int jplane;          // Jones plane (beam models)
  int plane0, plane1;  // first and last coarse plane (tabulated spectra)
  int expo;            // float offset of the segment's exponent tables (TcExpo), spectra and tapers
  float lam0, xi0;        // log-frequency term and squared frequency ratio at the reference channel
};

// A team of up to kTcMaxTeam segments of one uniformly spaced run (same steps).
struct TcTeamDesc {
  float w_hi, w_lo;    // row step: D channel increments
  float w8_hi, w8_lo;  // eight rows
  float s_hi, s_lo;    // channel increment
  int D;
  TcSeg seg[kTcMaxTeam];
};

// Float offsets inside a segment's exponent tables: the log-frequency term is
// L(a, n) = lam0 + lamRow(a) + lamCol(n) + R(a, n), the squared frequency ratio
// xi0 + xiRow(a) + xiCol(n) + xf(a) y(n), and R(a, n) ~ xl(a) y(n).  (Tabulated
// spectra: the log frequency is to the row's plane, lam0 = 0, and the rows carry
// the planes' fluxes.)
struct TcExpo {
  int lamRow, xiRow, xl, xf, lamCol, xiCol, y, L, plane, total;
};
inline TcExpo tc_expo_layout(int MA, int NJ) {
  TcExpo e{};
  int o = 0;
  auto take = [&](int n) { const int at = o; o += (n + 3) & ~3; return at; };
  e.lamRow = take(16 * MA);
  e.xiRow = take(16 * MA);
  e.xl = take(16 * MA);
  e.xf = take(16 * MA);
  e.lamCol = take(8 * NJ);
  e.xiCol = take(8 * NJ);
  e.y = take(8 * NJ);
  e.L = take(128 * MA * NJ);  // L(a, n) - lam0, in the order the lanes hold their sums
  e.plane = take(16 * MA);        // coarse plane of each row (int bits)
  e.total = o;
  return e;
}

// Kernel parameters.  Record and application fields as in KParams.
struct TcParams {
  KParams k;                // vis, nvis, lrec, iloc*, incs, pol*, op, ..., comps, ncomp, cstride, compsLo
  const TcTeamDesc* teams;
  int nteam;
  const int* chanOff;       // record float offset of each selected channel's first polarization
  const float* expo;
  TcExpo lay;
  int specField;            // component field of the spectral index
};

// One launch: teams of one shape.  A model's plan is one of these per shape that
// its runs are cut into.
struct TcPlan {
  bool on = false;
  bool beam = false;
  int MA = 2, NJ = 2, T = 1;  // 16 MA rows x 8 NJ columns per warp, T warps per team
  int NC = 2;                 // column groups that are channels: NJ, or 1 for a beam (NJ correlations)
  int kind = kPoint;        // family of the (remaining) table
  int mixed = 0;            // a point sub-table precedes the Gaussian rows (as ModelDesc.ncompPt)
  bool crossPt = false;     // point rows with a spectral index need the cross product
  std::vector<TcTeamDesc> teams;
  std::vector<int> chanOff;
  std::vector<float> expo;
  // device copies (one allocation) and launch facts
  void* d_mem = nullptr;
  TcParams kp{};
  int gridCap = 0;
};

// Host part: whether the tensor-core form takes this layout and model, and its
// teams and tables.  fetch: host copy of the table the kernels read (asked for only
// when the layout can win; null: recurrence) (ncompPt
// point rows first when mixed), rows of comp_stride floats.  Leaves *plan
// empty when the recurrence kernels should run.
// jchan (beam models): Jones plane per frequency-table index, ncorr modelled
// correlations; runs never span a change of plane, and recurCost is what the
// other form costs in the shapes' units.
void tc_plan_layout(const LayoutDesc& L, const ModelDesc& M, const std::function<const float*()>& fetch,
                    double recurCost, std::vector<TcPlan>* plan, const int* jchan = nullptr, int ncorr = 0);
// Cost of the recurrence kernels for a plan of theirs.
double tc_recur_cost(const Plan& recur);

// Device side and launch.
int tc_finalize(TcPlan* plan, const KParams& base, std::string* err);  // plan->beam: the beam kernel
void tc_free(std::vector<TcPlan>* plan);
int tc_finalize_all(std::vector<TcPlan>* plan, const KParams& base, std::string* err);
// Kernels of the tabulated families (dft_tc_tab.cu).
using TcFn = void (*)(const TcParams);
TcFn tc_pick_tab(const TcPlan& pl);

struct TcBeamParams {
  TcParams t;
  BeamKParams b;    // antenna types, Jones table, application
  const int* perm;  // component's index in the Jones table, or null
};
// The beam form's kernel for the plan (dft_tc_beam.cu): resident CTAs, launch.
int tc_beam_prepare(const TcPlan& plan, int* gridCap, std::string* err);
int tc_beam_launch(const TcPlan& plan, const ModelDesc& model, const BeamKParams& beam, const int* perm,
                   const float* d_comps, cudaStream_t stream, std::string* err);

int tc_launch(const TcPlan& plan, const ModelDesc& model, float* d_vis, int nvis, const float* d_comps, int* d_err,
              cudaStream_t stream, std::string* err);

}  // namespace obit
