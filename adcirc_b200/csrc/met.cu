// met.cu -- parametric-vortex met forcing on the device (NWS = 8).
//
// getMeteorologicalForcing (timestep.F:651) for NWS = 8 calls HollandGet
// (nws08.F90:562-717) and turns its 10 m wind and surface pressure into the
// GWCE/momentum forcing WSX2/WSY2/PR2 (wind.F:1172-1198).  In the step's first
// pass (k_step_begin) every block advances the track state for itself
// (GetHollandStormData, nws08.F90:827-878, whose module counter and WTRATIO
// persist across steps) and every node then evaluates the vortex
// independently (vortex_advance and node_vortex, step_bodies.cuh).  This file
// holds the track's set-up.  The step's TimeLoc and RampMete come
// from the device step table, so replayed step graphs need no host work.
//
// The mesh is Cartesian (ICS = 1): the storm centre is in mesh metres, the
// distance is Euclidean and theta = atan2(dy, dx) (thetaLatDep = .false.);
// the reference's DEG2RAD scaling and haversine distance apply to its
// spherical (ICS = 2) input only.  Transcendentals are CUDA's (sqrt, exp,
// pow, sin, cos, atan2).
#include "adc_internal.cuh"

#include <cmath>
#include <cstring>

namespace adc {

// NWS08INIT (nws08.F90:459-477): the first fix pair brackets the start time.
static int vortex_first_pair(const adc_vortex_t *v) {
  const double t = v->start_time;
  for (int i = 1; i < v->nfix; ++i)
    if (std::ceil(t) >= v->fix[i - 1].time && std::floor(t) < v->fix[i].time) return i;
  return -1;
}

}  // namespace adc

using namespace adc;

extern "C" int adc_set_vortex(adc_ctx *c, const adc_vortex_t *v) {
  if (!c || !v || !v->fix || v->nfix < 2) {
    set_error("adc_set_vortex: a track of at least two fixes is required");
    return ADC_ERR_ARG;
  }
  if (c->p.nws == 0) {
    set_error("adc_set_vortex: NWS = 0 in the bound parameters");
    return ADC_ERR_ARG;
  }
  for (int i = 1; i < v->nfix; ++i)
    if (!(v->fix[i].time > v->fix[i - 1].time)) {
      set_error("adc_set_vortex: fix times must increase (fix %d)", i + 1);
      return ADC_ERR_ARG;
    }
  if (!(v->bladj > 0.0) || !(v->rho_air > 0.0)) {
    set_error("adc_set_vortex: BLAdj and rhoAir must be positive");
    return ADC_ERR_ARG;
  }
  const int i0 = vortex_first_pair(v);
  if (i0 < 0) {
    set_error("adc_set_vortex: the track does not cover the start time %g s", v->start_time);
    return ADC_ERR_ARG;
  }
  if (c->vfix) {
    cudaFree(c->vfix);
    c->vfix = nullptr;
  }
  ADC_CUDA(cudaMalloc((void **)&c->vfix, v->nfix * sizeof(adc_vortex_fix_t)));
  ADC_CUDA(cudaMemcpy(c->vfix, v->fix, v->nfix * sizeof(adc_vortex_fix_t), cudaMemcpyHostToDevice));
  if (!c->vstate) ADC_CUDA(cudaMalloc((void **)&c->vstate, sizeof(VortexState)));
  VortexState st;
  memset(&st, 0, sizeof(st));
  st.counter = i0;
  st.wtratio = 1.0;   // module default, nws08.F90:68
  ADC_CUDA(cudaMemcpy(c->vstate, &st, sizeof(st), cudaMemcpyHostToDevice));
  c->vpar = *v;
  c->vpar.fix = nullptr;
  c->vortex_on = 1;
  drop_graphs(c);   // replayed steps must include the forcing
  return ADC_OK;
}
