// loop.cuh — a whole constant-dt solve in one launch (loop.cu).
#pragma once
#include <cuda_runtime.h>

#include "dev.cuh"
#include "kernels.hpp"

namespace edus {

// What changes from step to step, laid out once per problem by the host with
// the run loop's own clock and fields.
struct alignas(16) LoopStep {
  double EF[3][2][3];   // pump, probe / 2 at t, t + dt/2, t + dt
  double EF_last[2][3]; // field of the last evaluation before this step (output record)
  double t;
  int e_non0;           // k-gradient on in this step
  int obs;              // an output instant precedes the step
  int startup;          // Adams-Bashforth: RK4 step of the start-up
  int pad;
};
static_assert(sizeof(LoopStep) == 224, "LoopStep is copied in 16-byte words");

struct LoopArgs {
  DevTables tb;
  const DevConsts* cst;
  const unsigned char* steps;  // per step: LoopStep, then its ngc gradient coefficients
  size_t stride;               // bytes per step, a multiple of 16
  int it0, res, nstartup;  // first step, output resolution, RK4 steps of the Adams-Bashforth start-up
  int nsteps, order, kt;   // order 0: RK4; kt: k points per block
  double2 *P0, *P1, *Pa, *Pb;
  double2* ring;           // Adams-Bashforth: derivatives before the first step, newest first, and after the last
  double dt, dt6, dt3, dt2, wx2;
  double coef[kMaxOrder];
  // stencil vectors with a k-gradient coefficient that can be nonzero in this
  // run, in b order; npc coefficients each (the pump's components in use)
  int nb_sel, npc, nbp, ngc;  // ngc: coefficients of a step [3][npc][nbp], nbp: nb_sel padded with zeros to 12 or a multiple of 6
  int bsel[kMaxNb];
  int ncomp, comp[3];      // field components in use
  // observables
  int want_current, want_tabs;
  double scaleJ, scaleTA;
  ObsRecord* log;
  int log_cap;
  double *ncond_dev, *pcmax_dev;
  double* part;            // [2][blocks][32]
  unsigned int* bar;       // arrivals, zeroed before the launch
};

// Shape of a solve's launch; blocks = 0 where the launch per stage stays
// (loop.cu gives the rule).
struct LoopPlan {
  int blocks = 0, threads = 0, kt = 0, small = 0, cluster = 0;
  size_t smem = 0;
  size_t part = 0;  // scratch doubles
};
LoopPlan loop_plan(const DevTables& tb, int nb, int ngc, int ncomp, int sms, bool ab);
cudaError_t launch_loop(const LoopArgs& a, const LoopPlan& p, cudaStream_t s);

}  // namespace edus
