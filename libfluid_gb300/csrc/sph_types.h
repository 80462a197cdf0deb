// Plain-old-data types shared by host code and sm_103a kernels.
//
// One scene = one independent fluid system (a FluidSystem in the reference,
// libfluid/include/fluidsystem.h:16-126).  The reference keeps one parameter
// block per process in __constant__ memory (fluidparams.cu:6); here every
// scene has its own DevParams in global memory so that many scenes can be
// advanced by one launch per pass.
#pragma once
#include <stdint.h>

#define SPH_NULL_HASH 0xFFFFFFFFu   // fluiddefines.h:12 (UINT_MAX)
#define SPH_OKEY_NULL 0xFFFFFFFFu   // packed cell of a particle outside the grid
#define SPH_OKEY_MOVED 0x80000000u  // packed-cell flag: the particle has changed cell since
#define SPH_OKEY_MAX_DIM 1024u      // grids up to this many cells per axis can defer XSPH
#define SPH_FLAG_DEFER_XSPH 0x2u    // DevParams.flags: XSPH applied by the next density pass
#define SPH_FLAG_SPHERE 0x4u        // DevParams.flags: sphere boundary instead of the box

// Derived per-scene parameters (the FluidParamData of fluidparams.cuh:16-69,
// generalised to a rectangular box [0,L]^3 with cell size h).
struct DevParams {
    // grid: cell = floor(p * inv_cell) per axis, linearised x fastest
    uint32_t gx, gy, gz, gxy;     // grid dims and gx*gy
    uint32_t ncells;              // gx*gy*gz; the scene's NULL bucket is cell ncells
    float inv_cell;               // float(res) for the unit cube
    // box signed distance: d = |p - c| - b (fluidutil.cu:85-102)
    float box_cx, box_cy, box_cz, box_bx, box_by, box_bz;
    // smoothing length and kernel constants (fluidparams.cu:51-89)
    float h, halfh, h2, h4, h6, h8, h9, invh9;
    float poly6, grad_poly6, grad_spiky, cohesion;
    float visc_eps;               // 0.01*h^2 (fluidphysics.cu:279), rounded to float once
    // fluid
    float rest_density, inv_rest_density, gas_constant, gamma, eos_k;  // eos_k = B*rho0/gamma
    float mass, two_mass, particle_size, inv_particle_size;
    float dt, dtdt;
    float xsph, surface_tension, viscosity, adhesion, vdamp;
    float vel_limit, acc_limit, vel_limit2, acc_limit2;
    float grav_x, grav_y, grav_z;
    float eps;                    // FLT_MIN (fluidparams.cu:48)
    uint32_t flags;               // bit0: surface tension active (normals pass needed);
                                  // bit1: the scene defers XSPH (SPH_FLAG_DEFER_XSPH);
                                  // bit2: sphere boundary (SPH_FLAG_SPHERE)
    float skin2;                  // ((1 + skin) h)^2: radius of the neighbour masks
    float inv_h2;                 // 1/h^2, normalises displacements for the XSPH mask check
    float xsph_disp_limit2;       // (skin/2)^2 * 0.98: largest (displacement/h)^2 XSPH may accept
    float sphere_r;               // sphere boundary (flags bit2): radius about the box centre
    float near2;                  // threshold of the half-precision candidate test (HalfScan), in cells squared
    uint32_t pad_;
};

// The skin words are built with radius (1 + skin) h (default skin below).
// XSPH, which runs on positions moved by the integrator, may use them only
// while every particle moved less than skin*h/2 in the substep (checked on
// the device; otherwise XSPH walks all candidates).
#define SPH_SKIN_DEFAULT 0.1f

// Neighbour words per slot (row m of slot k at mask[m * stride + k]): the
// neighbour list's header, its words (four neighbours each), and the skin-radius
// words, used only when some scene runs a per-substep XSPH pass.
#define SPH_NBR_LIST       1u    // first list row; row 0 is the header
#define SPH_NBR_LIST_WORDS 17u   // (odd: the threads' lists in shared memory start in different banks)
#define SPH_MASK_SKIN      18u   // 9 rows: candidates within the skin radius (rows of <= 32)
#define SPH_DENSE_ROWS     18u   // 4 rows: position and density again, for the normal pass (one thread per particle)
#define SPH_AXIS_ROWS      24u   // 3 rows: the per-axis positions of the candidate scan, of which the
                                 // half-precision ones (one thread per particle) take 2
#define SPH_AXIS_ROWS_SKIN 15u   // with a skin pass, whose words take those
#define SPH_MASK_ROWS      27u
#define SPH_NBR_CAP        68u   // listed neighbours: four to a word
#define SPH_NBR_CAP_SKIN   56u   // with a skin pass: the words before SPH_AXIS_ROWS_SKIN
#define SPH_NBR_CAP_WIDE   92u   // several lanes per particle: all words before SPH_AXIS_ROWS
#define SPH_NBR_NEW_ROW    128u  // added to a row's first neighbour
#define SPH_NBR_MAX_ROW    128u  // longest row whose offsets fit below that
#define SPH_NBR_ROWS       10u   // row starts kept per thread: nine and one that is read ahead
#define SPH_NBR_SMEM_WORDS (SPH_NBR_ROWS + SPH_NBR_LIST_WORDS)

// Kernel variants (bits of the execution config's `variant`). All variants
// visit neighbours in the same order and give identical results; they differ
// only in how the walk is scheduled.
#define SPH_VARIANT_DENSITY_ROWS  0x1u   // no effect: one candidate scan is left
#define SPH_VARIANT_XSPH_ROWS     0x2u   // XSPH: one loop per cell row instead of one flattened walk
#define SPH_VARIANT_FORCE_OCC     0x4u   // force: 64-register build (more resident warps)
#define SPH_VARIANT_FORCE_TABLE   0x8u   // no effect: the force and normal passes walk the neighbour list
#define SPH_VARIANT_NORMALS_TABLE 0x10u  // no effect
#define SPH_VARIANT_DENSITY_SPLIT 0x20u  // neighbour passes: several lanes per particle in small launches
                                         // (at most SPH_DENSITY_SPLIT_MAX threads of tiles, more where crowded)
#define SPH_VARIANT_MASK          0x3fu
#define SPH_VARIANT_DEFAULT       0x3fu

// Largest launches (threads of all tiles) that run eight and four lanes per
// particle in the neighbour passes.  Measured on cubes of fluid at rest density
// (33 neighbours), substep in us with eight lanes, four, one: 13,824 particles
// 34.9, 36.7, 52.5; 21,952 45.9, 40.0, 52.2; 32,768 55.4, 46.1, 53.3; 35,937
// with surface tension 75.0, 70.6, 67.2; 46,656 68.0, 60.9, 58.2.  A crowded
// particle's walk is longer and the lanes shorten it by more: two collapsing
// columns of (neighbours on average) 38,266 particles (200) 323, 389, 897;
// 59,048 (158) 403, 459, 757; 59,048 (91) 170, 164, 351; 119,168 (116) 561,
// 574, 559.  Crowded: at least SPH_CROWDED_NBRS neighbours on average, from h,
// the rest density and the mass.
#ifndef SPH_WIDE8_MAX
#define SPH_WIDE8_MAX         14336u
#endif
#ifndef SPH_DENSITY_SPLIT_MAX
#define SPH_DENSITY_SPLIT_MAX 34816u
#endif
// Threads that an SM holds at once with 80 registers each (six blocks of 128; 152 SMs
// 116,736): a launch of one thread per particle that is no larger gains nothing from
// smaller register budgets, and runs builds that have more loads in flight instead.  Density, normals, force of 82,484 particles 32.5, 14.3, 27.5 -> 30.6,
// 13.8, 24.6 us, of 97,336 (no normals) 33.3, -, 24.4 -> 31.5, -, 20.6; a launch
// that takes a second wave is slower with them (125,000 particles 37.6, -, 26.6
// -> 42.8, -, 30.6).
#define SPH_ONE_WAVE_THREADS  768u
#define SPH_CROWDED_NBRS      80u
#define SPH_CROWDED8_MAX      61440u

// Scene placement in the engine's arenas.
struct DevScene {
    uint32_t part_base;   // first particle slot of the scene
    uint32_t n;           // particle count
    uint32_t cell_base;   // first cell of the scene in the packed cell arena
    uint32_t ncells;      // real cells; the NULL bucket follows at cell_base+ncells
};

// A tile: up to SPH_TILE consecutive particle slots of one scene.
// x = scene, y = first slot, z = count, w = 0.
#define SPH_TILE 256

// Status bits raised by kernels (read back after a step).
#define SPH_STATUS_CELL_OVERFLOW 0x1u   // a cell held more particles than the rank pass supports
#define SPH_STATUS_NONFINITE     0x2u   // a non-finite position appeared
#define SPH_STATUS_SCAN_TIMEOUT  0x4u   // a wait of the cell scan's look-back ran out

// Maximum particles one cell (or a scene's NULL bucket) may hold.  The
// reference cannot launch more than 1024 threads per cell block
// (fluidsystem.cu:322); this build supports 8x that.
#define SPH_MAX_CELL_OCC 8192u

// Lattice block generator (a dam-break fluid block with seeded jitter).
struct LatticeSpec {
    float lo[3];          // block corner
    float spacing;        // lattice spacing
    uint32_t nx, ny, nz;  // lattice sites per axis (x outermost, z innermost)
    float jitter;         // uniform jitter amplitude (+/-)
    float vel[3];         // initial velocity
    uint32_t pad_;
    uint64_t seed;
};
