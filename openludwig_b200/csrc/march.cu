// A batch of coarse time steps of one simulation in one call: the recursion of
// solver_control.jl:6-218 over caller-owned levels, each level sub-step through
// the same entry points a caller would use one by one (ol_stream_collide,
// ol_bouzidi_apply_links, ol_thermal, ol_restrict; timestep.jl:1-159).
//
// A small level's sub-step is 10-20 us of GPU time in three launches.  Driving
// them from an interpreted host costs about 21 us a step, so the GPU waited for
// the host; here a launch costs the host 1-2 us.
#include <algorithm>

#include "common.cuh"
#include "lattice.cuh"

namespace ol {
namespace {

struct March {
  const ol_march_level *lv;
  int n_levels;
  ol_step_params sp;
  ol_thermal_params tp;
  int ddf, restriction;
  int nx, ny, nz;
  cudaStream_t s;
};

// The state a parent step leaves for its children.
struct ParentState {
  float *f_new, *vel_new, *g_new;
  const float *f_old, *vel_old, *g_old;
};

template <class VIEW>
void ghost_views(VIEW &v, const ol_march_level &l, float *ghost, float *ghost2, int mode) {
  if (!ghost || !ghost2) mode = OL_GHOST_UNPAIRED;
  v.ghost_mode = mode;
  v.ghost = mode == OL_GHOST_PAIR_SECOND ? ghost2 : ghost;
  v.ghost_next = mode == OL_GHOST_PAIR_FIRST ? ghost2 : nullptr;
  const bool edge = mode == OL_GHOST_PAIR_SECOND;
  const int32_t *blocks = edge ? l.edge_blocks : l.view.ghost_blocks;
  v.ghost_blocks = ghost ? blocks : nullptr;
  v.n_ghost_blocks = ghost && blocks ? (edge ? l.n_edge_blocks : l.view.n_ghost_blocks) : 0;
}

int sub_step(const March &M, int i, int64_t t_sub, const ParentState *par, float tw, int mode,
             const float *f_in, float *f_out, const float *vel_in, float *vel_out,
             const float *g_in, float *g_out) {
  const ol_march_level &l = M.lv[i];
  const int n = l.view.n_blocks;
  if (n == 0) return OL_OK;
  const ol_march_level *p = par ? &M.lv[i - 1] : nullptr;
  ol_step_params sp = M.sp;
  sp.tau_molecular = l.tau;
  sp.tau_parent = p ? p->tau : 0.5f;
  sp.is_level_1 = par == nullptr;
  sp.nx_global = M.nx << i; sp.ny_global = M.ny << i; sp.nz_global = M.nz << i;
  sp.time_step_seed = (int32_t)(t_sub % 1000000);
  sp.store_post_collision = 0;
  sp.temporal_weight = tw;
  ol_level_view v = l.view;
  v.f_in = f_in; v.f_out = f_out; v.f_post = nullptr;
  v.vel_in = vel_in; v.vel_out = vel_out;
  ghost_views(v, l, l.view.ghost, l.view.ghost_next, mode);
  ol_parent_view pv = {};
  if (par) {
    pv.f = par->f_new; pv.rho = p->view.rho; pv.vel = par->vel_new;
    pv.f_old = par->f_old; pv.rho_old = p->rho_old; pv.vel_old = par->vel_old;
    pv.block_ptr = p->block_ptr;
    pv.dim_x = p->dim_x; pv.dim_y = p->dim_y; pv.dim_z = p->dim_z;
    pv.n_blocks = p->view.n_blocks;
  }
  int rc = ol_stream_collide(&v, &pv, &sp, M.s);
  if (rc) return rc;
  if (l.n_links > 0 &&
      (rc = ol_bouzidi_apply_links(f_out, l.links, l.n_links, n, l.link_scratch, M.s)))
    return rc;
  if (!M.ddf || !g_out) return OL_OK;
  ol_thermal_params tp = M.tp;
  tp.tau_g = l.tau_g;
  tp.tau_g_parent = p ? p->tau_g : 0.5f;
  tp.is_level_1 = sp.is_level_1;
  tp.nx_global = sp.nx_global; tp.ny_global = sp.ny_global; tp.nz_global = sp.nz_global;
  tp.store_post_collision = 0;
  tp.temporal_weight = tw;
  ol_thermal_view tv = {};
  tv.g_out = g_out; tv.g_in = g_in;
  tv.temperature = l.temperature; tv.vel = vel_out;
  tv.obstacle = l.view.obstacle; tv.sponge = l.view.sponge;
  tv.neighbor_table = l.view.neighbor_table;
  tv.map_x = l.view.map_x; tv.map_y = l.view.map_y; tv.map_z = l.view.map_z;
  tv.n_blocks = n;
  ghost_views(tv, l, l.ghost_g, l.ghost_g2, mode);
  if (par) {
    tv.pg = par->g_new; tv.pT = p->temperature; tv.pvel = par->vel_new;
    tv.pg_old = par->g_old; tv.pT_old = p->temperature_old; tv.pvel_old = par->vel_old;
    tv.p_block_ptr = p->block_ptr;
    tv.p_dim_x = p->dim_x; tv.p_dim_y = p->dim_y; tv.p_dim_z = p->dim_z;
    tv.p_n_blocks = p->view.n_blocks;
  }
  if ((rc = ol_thermal(&tv, &tp, M.s))) return rc;
  if (l.n_links > 0) return ol_bouzidi_apply_links(g_out, l.links, l.n_links, n, l.link_scratch, M.s);
  return OL_OK;
}

int copy_field(float *dst, const float *src, int n_blocks, cudaStream_t s) {
  if (n_blocks > 0)
    OL_CUDA(cudaMemcpyAsync(dst, src, sizeof(float) * BCELLS * (size_t)n_blocks,
                            cudaMemcpyDeviceToDevice, s));
  return OL_OK;
}

int recurse(const March &M, int i, int64_t t_sub, const ParentState *par, float tw, int mode) {
  if (i >= M.n_levels) return OL_OK;
  const ol_march_level &l = M.lv[i];
  const bool even = t_sub % 2 == 0;
  // view.f_in / f_out are the buffers read and written on even sub-steps
  float *const fa = const_cast<float *>(l.view.f_in), *const fb = l.view.f_out;
  float *const va = const_cast<float *>(l.view.vel_in), *const vb = l.view.vel_out;
  const float *f_in = even ? fa : fb, *vel_in = even ? va : vb, *g_in = even ? l.g : l.g_temp;
  float *f_out = even ? fb : fa, *vel_out = even ? vb : va, *g_out = even ? l.g_temp : l.g;
  const bool children = i + 1 < M.n_levels;
  const bool temporal = M.sp.use_temporal_interp != 0;
  int rc;
  if (children && temporal) {
    // copy_to_old! (blocks.jl:241-252): f, vel and g alias the untouched pull
    // sources; rho and T are overwritten in place
    if ((rc = copy_field(l.rho_old, l.view.rho, l.view.n_blocks, M.s))) return rc;
    if (M.ddf && l.g && (rc = copy_field(l.temperature_old, l.temperature, l.view.n_blocks, M.s)))
      return rc;
  }
  if ((rc = sub_step(M, i, t_sub, par, tw, mode, f_in, f_out, vel_in, vel_out,
                     M.ddf ? g_in : nullptr, M.ddf ? g_out : nullptr)))
    return rc;
  if (!children) return OL_OK;
  const ParentState me = {f_out, vel_out, M.ddf ? g_out : nullptr, temporal ? f_in : nullptr,
                          temporal ? vel_in : nullptr, temporal && M.ddf ? g_in : nullptr};
  if ((rc = recurse(M, i + 1, 2 * t_sub, &me, 0.0f, OL_GHOST_PAIR_FIRST))) return rc;
  if ((rc = recurse(M, i + 1, 2 * t_sub + 1, &me, 0.5f, OL_GHOST_PAIR_SECOND))) return rc;
  if (!M.restriction) return OL_OK;
  const ol_march_level &c = M.lv[i + 1];
  ol_restrict_view r = {};
  r.f_fine = c.view.f_in;  // the child's second sub-step is odd: it wrote this buffer
  r.obstacle_fine = c.view.obstacle;
  r.map_x = c.view.map_x; r.map_y = c.view.map_y; r.map_z = c.view.map_z;
  r.n_fine = c.view.n_blocks;
  r.f_coarse = f_out; r.rho_coarse = l.view.rho; r.vel_coarse = vel_out;
  r.obstacle_coarse = l.view.obstacle;
  r.block_ptr = l.block_ptr;
  r.dim_x = l.dim_x; r.dim_y = l.dim_y; r.dim_z = l.dim_z;
  r.n_coarse = l.view.n_blocks;
  r.tau_fine = c.tau; r.tau_coarse = l.tau;
  r.compressible = M.sp.compressible_corr;
  return ol_restrict(&r, M.s);
}

}  // namespace
}  // namespace ol

using namespace ol;

extern "C" int ol_march(const ol_march_level *levels, int32_t n_levels, const ol_step_params *sp,
                        const ol_thermal_params *tp, int32_t restriction, int32_t nx, int32_t ny,
                        int32_t nz, int64_t t_start, int32_t n_steps, void *stream) {
  OL_CHECK_ARG(levels && sp, "ol_march: null argument");
  OL_CHECK_ARG(n_levels >= 1 && n_levels <= 16 && n_steps >= 0 && t_start >= 0,
               "ol_march: bad sizes");
  for (int i = 0; i < n_levels; ++i) {
    const ol_march_level &l = levels[i];
    OL_CHECK_ARG(!tp || (l.g && l.g_temp && l.temperature),
                 "ol_march: level %d has no thermal buffers", i + 1);
    OL_CHECK_ARG(i + 1 == n_levels || sp->use_temporal_interp == 0 ||
                     (l.rho_old && (!tp || l.temperature_old)),
                 "ol_march: level %d needs rho_old (and temperature_old) for its children", i + 1);
  }
  March M = {levels, n_levels, *sp, {}, tp != nullptr, restriction, nx, ny, nz,
             (cudaStream_t)stream};
  if (tp) M.tp = *tp;
  for (int32_t k = 0; k < n_steps; ++k) {
    const int rc = recurse(M, 0, t_start + k, nullptr, 0.0f, OL_GHOST_UNPAIRED);
    if (rc) return rc;
  }
  return OL_OK;
}
