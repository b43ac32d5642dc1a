// mpm_ops.cuh -- launch wrappers that bind the kernels of one arithmetic form
// into a StepOps table (included once per form).
#pragma once

#include "mpm_kernels.cuh"

namespace mpm {

// Launch shape of the one-thread-per-item kernels: blocks of 256, halved down
// to one warp while there would be fewer than two blocks per SM. These kernels
// are bound by the FP64 pipe of the SMs they run on (2 lanes per SM and clock),
// so a small scene has to reach every SM: 5.8 k particles in blocks of 256
// keep 23 of 152 SMs busy.
struct Shape {
  unsigned grid, block;
  explicit Shape(long long n) : block(kBlock) {
    while (block > 32 && (n + block - 1) / block < 304) block >>= 1;
    grid = (unsigned)((n + block - 1) / block);
  }
};
// a pair_walk kernel over n nodes or cells: a block per group of nodes, no more
// than there can be groups with pairs and blocks of nodes without
template <int PAIRS, class... P, class... A>
inline void launch_walk(void (*kernel)(P...), long long n, const Geometry& g, cudaStream_t st, A... args) {
  constexpr int T = kWalkNodes * PAIRS;
  const long long all = (n + kWalkNodes - 1) / kWalkNodes;
  const long long some = (g.np * g.K + kWalkNodes - 1) / kWalkNodes + (n + T - 1) / T;
  launch_chained(kernel, (unsigned)(all < some ? all : some), T, st, args...);
}

template <class P>
struct Ops {
  static St<P>& S(void* st) { return *reinterpret_cast<St<P>*>(st); }

  static void begin_step(void* st, const Geometry&, cudaStream_t s) {
    prof_begin(K_BEGIN, s);
    launch_chained(k_begin_step, 1, 1, s, S(st).sc);
    prof_end(K_BEGIN, s);
  }
  template <bool LISTED>
  static void gimp_slots(void* st, const Geometry& g, int with_comp, cudaStream_t s) {
    launch_chained(k_gimp_slots<P, LISTED>, (unsigned)((g.np + 31) / 32), 32 * kGimpWarps, s, S(st), g, with_comp);
  }
  static void locate(void* st, const Geometry& g, cudaStream_t s) {
    const Shape h(g.np);
    prof_begin(K_LOCATE, s);
    switch (g.shape) {
      case 0: launch_chained(k_locate<P, 0>, h.grid, h.block, s, S(st), g); break;
      case 1:
        launch_chained(k_locate<P, 1>, h.grid, h.block, s, S(st), g);
        gimp_slots<true>(st, g, 1, s);
        break;
      case 2: launch_chained(k_locate<P, 2>, h.grid, h.block, s, S(st), g); break;
      default: launch_chained(k_locate<P, 3>, h.grid, h.block, s, S(st), g);
    }
    prof_end(K_LOCATE, s);
  }
  static void p2g_mass(void* st, const Geometry& g, int bc, int vel, cudaStream_t s) {
    prof_begin(K_P2G_MASS, s);
    if (g.shape == 3) {
      launch_walk<kWalkFew>(k_sg_cell_mass<P>, g.ncell, g, s, S(st), g);
      launch_chained(k_sg_node_mass<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g, bc, vel);
    } else {
      launch_walk<kWalkFew>(k_p2g_mass<P>, g.nnt, g, s, S(st), g, bc, vel);
    }
    prof_end(K_P2G_MASS, s);
  }
  static void node_velocity(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_NODE_VEL, s);
    launch_chained(k_node_velocity<P>, Shape(g.nnt).grid, Shape(g.nnt).block, s, S(st), g);
    prof_end(K_NODE_VEL, s);
  }
  static void apply_bc(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_BC, s);
    launch_chained(k_apply_bc<P>, Shape(g.nnt).grid, Shape(g.nnt).block, s, S(st), g);
    prof_end(K_BC, s);
  }
  // the stress update's instantiation for the deck's one material type; scenes
  // with fewer than a warp of particles per scheduler share a particle's gather
  // among three warps (k_stress; registers do not matter there)
  static constexpr long long kAxesMost = 304 * 32;
  template <int UV>
  static void stress_of(void* st, const Geometry& g, cudaStream_t s) {
    const Shape h(g.np);
    if (g.np <= kAxesMost) {
      launch_chained(k_stress<P, 0, UV, true>, (unsigned)((g.np + 31) / 32), kAxesBlock, s, S(st), g);
      return;
    }
    switch (stress_has(S(st).mat_type) ? S(st).mat_type : 0) {
      case 1: launch_chained(k_stress<P, 1, UV, false>, h.grid, h.block, s, S(st), g); break;
      case 7: launch_chained(k_stress<P, 7, UV, false>, h.grid, h.block, s, S(st), g); break;
      case 9: launch_chained(k_stress<P, 9, UV, false>, h.grid, h.block, s, S(st), g); break;
      case 10: launch_chained(k_stress<P, 10, UV, false>, h.grid, h.block, s, S(st), g); break;
      case 11: launch_chained(k_stress<P, 11, UV, false>, h.grid, h.block, s, S(st), g); break;
      default: launch_chained(k_stress<P, 0, UV, false>, h.grid, h.block, s, S(st), g);
    }
  }
  static void stress(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_STRESS, s);
    if (g.shape == 3) launch_chained(k_sg_cell_gradient<P>, Shape(g.ncell).grid, Shape(g.ncell).block, s, S(st), g);
    if (g.uvfp) stress_of<1>(st, g, s);
    else stress_of<0>(st, g, s);
    prof_end(K_STRESS, s);
  }
  static void depeff_apply(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_DEPEFF, s);
    launch_chained(k_depeff_apply<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
    launch_chained(k_depeff_carry<P>, 1, 1, s, S(st), g);
    prof_end(K_DEPEFF, s);
  }
  static void force_prep(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_FORCE_PREP, s);
    launch_chained(k_force_prep<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
    prof_end(K_FORCE_PREP, s);
  }
  static void p2g_force(void* st, const Geometry& g, int integ, cudaStream_t s) {
    prof_begin(K_P2G_FORCE, s);
    if (g.shape == 3) {
      launch_walk<kWalkMany>(k_sg_cell_force<P>, g.ncell, g, s, S(st), g);
      launch_chained(k_sg_node_force<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g, integ);
    } else {
      if (g.contact) launch_walk<kWalkMany>(k_p2g_force<P, true>, g.nnt, g, s, S(st), g, integ);
      else launch_walk<kWalkMany>(k_p2g_force<P, false>, g.nnt, g, s, S(st), g, integ);
    }
    prof_end(K_P2G_FORCE, s);
  }
  static void integrate(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_INTEGRATE, s);
    launch_chained(k_integrate<P>, Shape(g.nnt).grid, Shape(g.nnt).block, s, S(st), g);
    prof_end(K_INTEGRATE, s);
  }
  static void position(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_POSITION, s);
    if (g.shape == 3) launch_chained(k_sg_cell_velocity<P>, Shape(g.ncell).grid, Shape(g.ncell).block, s, S(st), g);
    const Shape h(g.np);
    launch_chained(k_position<P>, dim3(h.grid, 3), h.block, s, S(st), g);
    prof_end(K_POSITION, s);
  }
  static void p2g_momentum(void* st, const Geometry& g, int vel, cudaStream_t s) {
    prof_begin(K_P2G_MOM, s);
    if (g.shape == 3) {
      launch_walk<kWalkFew>(k_sg_cell_momentum<P>, g.ncell, g, s, S(st), g);
      launch_chained(k_sg_node_momentum<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g, vel);
    } else {
      launch_walk<kWalkFew>(k_p2g_momentum<P>, g.nnt, g, s, S(st), g, vel);
    }
    prof_end(K_P2G_MOM, s);
  }
  static void reduce(void* st, const Geometry& g, int mode, int nblocks, cudaStream_t s) {
    prof_begin(K_REDUCE, s);
    launch_chained(k_reduce<P>, nblocks, kBlock, s, S(st), g, mode);
    prof_end(K_REDUCE, s);
  }
  static void dr_damping(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_DR, s);
    launch_chained(k_dr_damping<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
    launch_chained(k_dr_finish, 1, 1, s, S(st).sc);
    prof_end(K_DR, s);
  }

  static void fixed_locate(void* st, const Geometry& g, int with_comp, cudaStream_t s) {
    prof_begin(K_LOCATE, s);
    const Shape h(g.np);
    switch (g.shape) {
      case 0: launch_chained(k_fixed_locate<P, 0>, h.grid, h.block, s, S(st), g, with_comp); break;
      case 1: gimp_slots<false>(st, g, with_comp, s); break;
      case 2: launch_chained(k_fixed_locate<P, 2>, h.grid, h.block, s, S(st), g, with_comp); break;
      default: launch_chained(k_fixed_locate<P, 3>, h.grid, h.block, s, S(st), g, with_comp);
    }
    prof_end(K_LOCATE, s);
  }
  static void tl_initial(void* st, const Geometry& g, cudaStream_t s) {
    launch_chained(k_tl_initial<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
  }
  static void tl_momentum(void* st, const Geometry& g, int vel, cudaStream_t s) {
    prof_begin(K_P2G_MASS, s);
    if (g.shape == 3) {
      launch_walk<kWalkFew>(k_sg_cell_momentum<P>, g.ncell, g, s, S(st), g);
      launch_chained(k_tl_sg_node_momentum<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g, vel);
    } else {
      launch_walk<kWalkFew>(k_p2g_momentum<P>, g.nnt, g, s, S(st), g, vel);
    }
    prof_end(K_P2G_MASS, s);
  }
  static void tl_stress(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_STRESS, s);
    if (g.shape == 3) launch_chained(k_sg_cell_gradient<P>, Shape(g.ncell).grid, Shape(g.ncell).block, s, S(st), g);
    launch_chained(k_tl_stress<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
    prof_end(K_STRESS, s);
  }
  static void tl_force(void* st, const Geometry& g, int integ, cudaStream_t s) {
    prof_begin(K_P2G_FORCE, s);
    if (g.shape == 3) {
      launch_chained(k_tl_sg_cell_force<P>, Shape(g.ncell).grid, Shape(g.ncell).block, s, S(st), g);
      launch_chained(k_tl_sg_node_force<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g, integ);
    } else {
      launch_chained(k_tl_p2g_force<P>, Shape(g.nnt).grid, Shape(g.nnt).block, s, S(st), g, integ);
    }
    prof_end(K_P2G_FORCE, s);
  }
  static void smooth(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_SMOOTH, s);
    if (g.shape == 3) {
      launch_walk<kWalkFew>(k_smooth_cell<P>, g.ncell, g, s, S(st), g);
      launch_chained(k_smooth_sg_node<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g);
      launch_chained(k_smooth_sg_back<P>, Shape(g.ncell).grid, Shape(g.ncell).block, s, S(st), g);
    } else {
      launch_walk<kWalkFew>(k_smooth_node<P>, g.nnt, g, s, S(st), g);
    }
    launch_chained(k_smooth_g2p<P>, Shape(g.np).grid, Shape(g.np).block, s, S(st), g);
    prof_end(K_SMOOTH, s);
  }

  static void contact(void* st, const Geometry& g, cudaStream_t s) {
    prof_begin(K_CONTACT, s);
    launch_chained(k_contact<P>, Shape(g.nn).grid, Shape(g.nn).block, s, S(st), g);
    launch_chained(k_contact_sum<P>, 1, kBlock, s, S(st), g);
    prof_end(K_CONTACT, s);
  }

  static StepOps table(const char* name) {
    StepOps o;
    o.name = name;
    o.bulk_size = sizeof(typename P::B);
    o.real_size = sizeof(typename P::R);
    o.begin_step = begin_step;
    o.locate = locate;
    o.p2g_mass = p2g_mass;
    o.node_velocity = node_velocity;
    o.apply_bc = apply_bc;
    o.stress = stress;
    o.depeff_apply = depeff_apply;
    o.force_prep = force_prep;
    o.p2g_force = p2g_force;
    o.integrate = integrate;
    o.position = position;
    o.p2g_momentum = p2g_momentum;
    o.reduce = reduce;
    o.dr_damping = dr_damping;
    o.fixed_locate = fixed_locate;
    o.tl_initial = tl_initial;
    o.tl_momentum = tl_momentum;
    o.tl_stress = tl_stress;
    o.tl_force = tl_force;
    o.smooth = smooth;
    o.contact = contact;
    return o;
  }
};

}  // namespace mpm
