// Runs of steps issued from native code: ppf_run calls the step entry point of
// a model once per pass, ping-ponging between two sets of field buffers. A
// step's own launch takes 2 to 3 us on the host, the interpreter's share of one
// step 9 us more (parameter and tiling structs, argument conversion), which
// bound short runs and runs on small grids.
#include "ppf_common.cuh"

namespace ppf {
namespace {

template <typename T>
struct Steps;
template <>
struct Steps<float> {
  static constexpr auto diffusion = ppf_diffusion_step_f32;
  static constexpr auto allen_cahn = ppf_allen_cahn_step_f32;
  static constexpr auto cahn_hilliard = ppf_cahn_hilliard_step_f32;
  static constexpr auto warren = ppf_warren1995_step_f32;
  static constexpr auto implicit = ppf_diffusion_implicit_step_f32;
  static constexpr auto phase = ppf_phase_implicit_step_f32;
  static constexpr auto ncgpu = ppf_ncgpu_step_f32;
  static constexpr auto warm = ppf_ncgpu_temperature_advance_f32;
};
template <>
struct Steps<double> {
  static constexpr auto diffusion = ppf_diffusion_step_f64;
  static constexpr auto allen_cahn = ppf_allen_cahn_step_f64;
  static constexpr auto cahn_hilliard = ppf_cahn_hilliard_step_f64;
  static constexpr auto warren = ppf_warren1995_step_f64;
  static constexpr auto implicit = ppf_diffusion_implicit_step_f64;
  static constexpr auto phase = ppf_phase_implicit_step_f64;
  static constexpr auto ncgpu = ppf_ncgpu_step_f64;
  static constexpr auto warm = ppf_ncgpu_temperature_advance_f64;
};

template <typename T>
int32_t one_pass(const PpfRun* r, T* const* in, T* const* out, const PpfTiling* t, int32_t done,
                 uint64_t step, int32_t* iterations, void* stream) {
  using S = Steps<T>;
  switch (r->model) {
    case PPF_RUN_DIFFUSION:
      return S::diffusion((const PpfDiffusionParams*)r->params, r->grid, r->boundary, in[0], out[0],
                          t, stream);
    case PPF_RUN_ALLEN_CAHN:
      return S::allen_cahn((const PpfAllenCahnParams*)r->params, r->grid, r->boundary, in[0],
                           out[0], t, stream);
    case PPF_RUN_CAHN_HILLIARD:
      return S::cahn_hilliard((const PpfCahnHilliardParams*)r->params, r->grid, r->boundary, in[0],
                              out[0], r->mass ? r->mass + done : nullptr, r->status, t, stream);
    case PPF_RUN_WARREN1995:
      return S::warren((const PpfWarren1995Params*)r->params, r->grid, r->boundary, in[0], in[1],
                       out[0], out[1], r->seed, step, r->step_base, t, stream);
    case PPF_RUN_DIFFUSION_IMPLICIT:
      return S::implicit((const PpfImplicitDiffusionParams*)r->params, r->grid, in[0], out[0],
                         (T*)r->tmp, r->scratch, r->scratch_bytes, iterations, stream);
    case PPF_RUN_PHASE_IMPLICIT:
      return S::phase((const PpfImplicitPhaseParams*)r->params, r->grid, in[0], out[0], (T*)r->tmp,
                      r->scratch, r->scratch_bytes, iterations, stream);
    case PPF_RUN_NCGPU: {
      const int32_t rc = S::ncgpu((const PpfNcgpuParams*)r->params, r->grid, r->boundary, in, out,
                                  (const T*)r->temperature, r->tables, (T*)r->tmp, r->seed, step,
                                  r->step_base, stream);
      // the step read T; then T rises
      if (rc || r->dT == 0.0) return rc;
      return S::warm(r->grid, (T*)r->temperature, r->dT, stream);
    }
  }
  return fail(PPF_ERR_INVALID, "run.model=%d unknown", r->model);
}

// passes the thread's last run issued without an error
thread_local int32_t g_passes = 0;

template <typename T>
int32_t run_passes(const PpfRun* r, const int32_t* depths, int32_t npasses, int32_t* iterations,
                   void* stream) {
  PpfTiling t{};
  if (r->tiling) t = *r->tiling;
  uint64_t step = r->step;
  int32_t done = 0;
  for (int32_t i = 0; i < npasses; ++i) {
    t.depth = depths[i];
    T* const* in = (T* const*)(i & 1 ? r->b : r->a);
    T* const* out = (T* const*)(i & 1 ? r->a : r->b);
    const int32_t rc = one_pass<T>(r, in, out, &t, done, step, iterations, stream);
    if (rc) return rc;
    g_passes = i + 1;
    done += depths[i];
    step += (uint64_t)depths[i];
  }
  return PPF_OK;
}

}  // namespace
}  // namespace ppf

using namespace ppf;

extern "C" {

int32_t ppf_run(const PpfRun* run, const int32_t* depths, int32_t npasses, int32_t* iterations,
                void* stream) {
  clear_error();
  g_passes = 0;
  if (!run || !run->params || !run->grid) return fail(PPF_ERR_INVALID, "run is NULL");
  if (npasses < 0 || (npasses > 0 && !depths)) return fail(PPF_ERR_INVALID, "bad pass list");
  const bool deep = run->model == PPF_RUN_DIFFUSION || run->model == PPF_RUN_ALLEN_CAHN;
  for (int32_t i = 0; i < npasses; ++i) {
    if (depths[i] < 1) return fail(PPF_ERR_INVALID, "depth=%d < 1", depths[i]);
    if (depths[i] > 1 && !deep)
      return fail(PPF_ERR_UNSUPPORTED, "run.model=%d advances one step per pass (depth=%d)",
                  run->model, depths[i]);
  }
  if (run->elem_bytes == 4) return run_passes<float>(run, depths, npasses, iterations, stream);
  if (run->elem_bytes == 8) return run_passes<double>(run, depths, npasses, iterations, stream);
  return fail(PPF_ERR_INVALID, "elem_bytes must be 4 or 8");
}

int32_t ppf_run_passes(int32_t* passes) {
  if (!passes) return fail(PPF_ERR_INVALID, "passes is NULL");
  *passes = g_passes;
  return PPF_OK;
}

}  // extern "C"
