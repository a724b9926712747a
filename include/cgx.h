/*
 * cgx.h -- B200 (sm_100a) compressible-LES right-hand side and RK3 step for
 * periodic Voronoi meshes: the C ABI that a host solver calls in place of the
 * reference's IdealGasSolver hot path.
 *
 * Reference interface replaced (paths relative to the reference source tree):
 *   IdealGasSolver::calcRhs                 src/charles/ideal_gas/IdealGasSolver.hpp:697-705
 *     -> calcRhsBase                        src/charles/ideal_gas/IdealGasSolver.cpp:257-535
 *   IdealGasSolver::rk3Step                 src/charles/ideal_gas/IdealGasSolver.hpp:692,
 *                                           IdealGasSolver.cpp:840-872
 *   updateConservativeAndPrimitiveData      src/charles/ideal_gas/IdealGasSolver.hpp:732-759
 *   calcSgsAndMaterialProperties            src/charles/ideal_gas/IdealGasSolver.cpp:182-255
 *     (computeSgsVreman IdealGasSolverSgs.cpp:207-296, setFgrCvs IdealGasSolver.cpp:894-984)
 *   calcCfl                                 src/charles/ideal_gas/IdealGasSolver.cpp:1048-1095
 *   setDt (TIMESTEP DT|CFL|CFL_DT)          src/charles/FlowSolver.hpp:2274-2328
 *   advanceSolution                         src/charles/ideal_gas/IdealGasSolver.hpp:414-594
 *   checkForNans / storeData / restoreData  src/charles/ideal_gas/IdealGasSolver.hpp:303-405,596-611
 *   report() conservation totals            src/charles/ideal_gas/IdealGasSolver.hpp:825-838
 *
 * Conventions
 *   - Every function returns CGX_OK (0) or a negative CGX_E_* code and never
 *     throws; cgx_last_error() gives the text of the last failure on the
 *     calling thread.
 *   - Host arrays are in the caller's (reference) cell numbering and layout:
 *     rho[ncv], u[ncv][3], rhoE[ncv], rhs[ncv][5] = {rho, rhou[3], rhoE}.
 *     The library renumbers cells internally by recursive bisection and
 *     keeps the permutation.
 *   - The library owns all device memory.  A solver handle is not
 *     thread-safe; all of its work is ordered on one CUDA stream.
 *   - Ghost cells are translated copies of owned cells (periodic boxes); the
 *     library resolves them to their owners and stores no ghost data.
 */
#ifndef CGX_H
#define CGX_H

#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

#define CGX_OK          0
#define CGX_E_ARG      -1   /* invalid argument or inconsistent mesh */
#define CGX_E_OOM      -2   /* host or device allocation failed */
#define CGX_E_CUDA     -3   /* a CUDA call failed */
#define CGX_E_NAN      -4   /* NaN detected; state restored (advanceSolution -1) */
#define CGX_E_TIMEOUT  -5   /* a bounded device wait gave up */
#define CGX_E_STATE    -6   /* call out of order (e.g. step before set_state) */

typedef enum cgx_precision {
  CGX_FP64  = 0,   /* all arithmetic in FP64 */
  CGX_MIXED = 1    /* FP32 flux/gradient/SGS arithmetic, FP64 face sums,
                      FP64 state, pressure recovery, dt and reductions */
} cgx_precision;

/* TIMESTEP modes (FlowSolver.hpp:2274-2328) */
#define CGX_DT_CONST   0   /* TIMESTEP DT <dt>              */
#define CGX_DT_CFL     1   /* TIMESTEP CFL <cfl>            */
#define CGX_DT_CFL_DT  2   /* TIMESTEP CFL_DT <cfl> <dtmax> */

/* SGS_MODEL */
#define CGX_SGS_NONE    0
#define CGX_SGS_VREMAN  1

/* NO_DISS / ALL_DISS switches of setFgrCvs */
#define CGX_DISS_SENSOR 0
#define CGX_DISS_NONE   1
#define CGX_DISS_ALL    2

/* Solver parameters; names follow the reference's input-file keys. */
typedef struct cgx_params {
  double gamma;            /* GAMMA 1.4 */
  double p_ref;            /* P_REF */
  double rho_ref;          /* RHO_REF */
  double T_ref;            /* T_REF */
  double mu_ref;           /* MU_REF */
  double mu_power_law;     /* MU_POWER_LAW 0.75 */
  double Pr_lam;           /* PR_LAM 0.7 */
  int    sgs_model;        /* SGS_MODEL (CGX_SGS_*) */
  double vreman_coeff;     /* VREMAN_COEFF 0.07 */
  double a_sgs_coeff;      /* A_SGS_COEFF 0.05 */
  double a_sgs_coeff2;     /* A_SGS_COEFF2 0.0015 */
  double lambda_dil_coeff; /* LAMBDA_DIL_COEFF 0 */
  double Pr_t;             /* PR_T 0.9 */
  double coeff_p;          /* COEFF_P 0.5 */
  double coeff_h;          /* COEFF_H 0.1 */
  double gr_nrm;           /* GR_NRM 0.03 */
  int    diss_mode;        /* CGX_DISS_* */
  int    dt_mode;          /* CGX_DT_* */
  double dt_data[2];       /* DT: {dt}; CFL: {cfl}; CFL_DT: {cfl, dt_max} */
  int    check_interval;   /* CHECK_INTERVAL (NaN store cadence) */
  int    limit_asgs;       /* LIMIT_ASGS: cap a_sgs at 1/(4 dt fax sos^2), fax = 1/(gamma-1) +
                              |u|^2/(2 sos^2), once dt > 0 (limitAsgs,
                              IdealGasSolverSgs.cpp:4-48); 0 = off, the default */
} cgx_params;

/* Fill with the reference's defaults (P_REF, RHO_REF, T_REF, MU_REF = 1). */
void cgx_params_default(cgx_params* p);

/*
 * Mesh in the reference's single-rank layout (StaticSolver.hpp:416-481):
 * owned cells [0,ncv), ghosts [ncv,ncv_g2) with icv_owner_g[ig-ncv] their
 * owners; compact faces cvofa/n_fa/area_over_delta_fa (a face whose second
 * cell is a ghost updates only its first cell); compact CSR cvocv_i/v (the
 * diagonal first) with cvocv_grad_coeff; extended faces cvoef/n_ef/c_ef with
 * c_ef NOT halved (as StaticSolver stores it); dcmag_hat_cv and
 * sa_to_vol_ratio as FlowSolver::init() computes them.  x_cv[ncv][3] is
 * optional: when given, cells are renumbered by recursive bisection of x_cv.
 */
typedef struct cgx_mesh_desc {
  int ncv, ncv_g2;
  int nfa, nef;
  const int*    cvofa;              /* [nfa][2] */
  const double* n_fa;               /* [nfa][3] */
  const double* area_over_delta_fa; /* [nfa] */
  const double* vol_cv;             /* [ncv] */
  const int*    cvocv_i;            /* [ncv+1] */
  const int*    cvocv_v;            /* [cvocv_i[ncv]] */
  const double* cvocv_grad_coeff;   /* [cvocv_i[ncv]][3] */
  const int*    cvoef;              /* [nef][2] */
  const double* n_ef;               /* [nef][3] */
  const double* c_ef;               /* [nef][3] */
  const double* dcmag_hat_cv;       /* [ncv] */
  const double* sa_to_vol_ratio;    /* [ncv] */
  const int*    icv_owner_g;        /* [ncv_g2-ncv] */
  const double* x_cv;               /* [ncv][3] or NULL */
  /* Boundary faces (nbf = 0 for a periodic box), as StaticSolver holds them
   * (cvobf, n_bf outward, area_over_delta_bf), with each face's boundary
   * zone in [0, nbf_zones); every zone needs a boundary condition
   * (cgx_set_bc) before cgx_init_complete.  The gradient coefficients given
   * above must include the faces' Gij_bf term, as calcCvGradCoeff forms them
   * (StaticSolver.cpp:5642-5650). */
  int nbf, nbf_zones;
  const int*    cvobf;              /* [nbf] owned cell */
  const double* n_bf;               /* [nbf][3] */
  const double* area_over_delta_bf; /* [nbf] */
  const int*    zone_bf;            /* [nbf] */
} cgx_mesh_desc;

typedef struct cgx_mesh cgx_mesh;
typedef struct cgx_solver cgx_solver;

typedef struct cgx_mesh_stats {
  int    ncv;
  long long n_ef_dir;      /* directed extended-face entries (2 per internal face) */
  long long n_cf_dir;      /* directed compact-face entries */
  double e_per_cell;       /* extended faces per cell, each face once */
  double f_per_cell;       /* compact faces per cell, each face once */
  size_t device_bytes;     /* device memory held by the mesh */
} cgx_mesh_stats;

/* Copy the mesh to device `device`, renumber it and build the CSR layouts. */
int cgx_mesh_create(const cgx_mesh_desc* desc, int device, cgx_mesh** out);
int cgx_mesh_stats_get(const cgx_mesh* m, cgx_mesh_stats* out);
int cgx_mesh_destroy(cgx_mesh* m);

int cgx_solver_create(cgx_mesh* m, const cgx_params* p, cgx_precision prec,
                      cgx_solver** out);
int cgx_solver_destroy(cgx_solver* s);

/* Conserved state in reference order (host arrays).  Host arrays may be
 * page-locked (copied directly) or pageable, such as a host solver's new[]
 * arrays: pageable arrays of 4 MiB or more are staged through two pinned 64
 * MiB chunks (allocated at first use and kept for later calls and meshes: as many
 * such pairs as solvers of a device have needed at once, two when they are gone),
 * which is several times faster than a pageable copy.  The same holds for every
 * call below that takes or fills a host array of cells. */
int cgx_set_state(cgx_solver* s, const double* rho, const double* u, const double* rhoE);
/* rho, u, p; rhoE = p/(gamma-1) + 0.5 rho |u|^2 (IdealGasSolver.hpp:275-301). */
int cgx_set_state_primitive(cgx_solver* s, const double* rho, const double* u,
                            const double* p);
int cgx_get_state(cgx_solver* s, double* rho, double* u, double* rhoE);

/* Passive transport scalars: nsc (0..8) scalars per cell in
 * the reference's order sc[icv*nsc + isc] (transport_scalar_vec,
 * IdealGasSolver.hpp).  Once set, calcRhs also forms rhs_sc as
 * calcRhsScalars does (IdealGasSolver.cpp:537-693: convective flux
 * 0.5 (sc0 + sc1) mf on every extended face with mf its mass flux, minus the
 * unity-Lewis diffusion on compact faces) and every rk3Step advances them as
 * advanceScalars does (IdealGasSolver.cpp:874-892).  nsc = 0 removes them.
 * Scalars, their face sums and their update are FP64 in both precisions; a
 * mixed-precision solver supplies mass fluxes from its FP32 flux arithmetic.
 * Like the reference's storeData, NaN recovery does not restore scalars. */
int cgx_set_scalars(cgx_solver* s, int nsc, const double* sc);
int cgx_get_scalars(cgx_solver* s, double* sc);
/* rhs_sc of stage rk_stage (1..3) as the last calcRhs/step left it,
 * [ncv][nsc] in reference order (unscaled face sums). */
int cgx_get_rhs_sc(cgx_solver* s, int rk_stage, double* rhs_sc);

/*
 * Source terms: the counterpart of the user hook addSourceHook(rhs, time,
 * rk_stage) (IdealGasSolver.hpp:713), which calcRhs calls after calcRhsBase
 * and calcRhsScalars (IdealGasSolver.hpp:697-705) to add to the stage's rhs.
 * Two forms, which may be combined; both apply to single-case solvers (not
 * to batch cases), in every stage of cgx_calc_rhs, cgx_advance_solution and
 * cgx_step.
 *
 * cgx_set_source: evaluated on the device inside the step graph.
 *   force: per cell f = vol rho (A u + g) (unscaled, like every rhs term)
 *          added as rhs.rhou += f, rhs.rhoE += f.u.  g alone is a body force
 *          (gravity), A = -1/tau with g = u_target/tau the relaxation force
 *          of the reference's example hooks (quiver/charles/charles.sphere.cpp
 *          :166-173), A alone linear forcing of isotropic turbulence.
 *   field: optional host array [ncv][5] (reference order and rhs layout),
 *          copied once and added as is to every stage's rhs.
 * A NULL source, or one with A = 0, g = 0 and field = NULL, removes it.
 */
typedef struct cgx_source {
  double A;             /* 1/time: coefficient of u in the force */
  double g[3];          /* acceleration */
  const double* field;  /* [ncv][5] or NULL */
} cgx_source;
int cgx_set_source(cgx_solver* s, const cgx_source* src);

/*
 * cgx_set_source_hook: a host callback with the reference hook's contract,
 * for sources that need host code.  In each stage, after the face sums, the
 * library copies the stage's conserved state to page-locked host memory and
 * calls
 *   fn(user, ncv, rho, u, rhoE, rhs, time, rk_stage)
 * with rho[ncv], u[ncv][3], rhoE[ncv] in reference order, rhs[ncv][5] zero
 * on entry, time the stage's time (t, t + dt, t + dt/2 for stages 1, 2, 3,
 * IdealGasSolver.hpp:488,528,569; the caller's time for cgx_calc_rhs), and
 * rk_stage 1..3.  What fn leaves in rhs is added to the stage's rhs.  fn runs
 * on a CUDA-owned host thread, as a host node of the step graph: it must not
 * call CUDA (or this library), and must not block on the thread that called
 * cgx_step.  The copies cost 80 bytes per cell per stage over PCIe, so this
 * form is for sources the device form cannot express.  fn = NULL removes it.
 */
typedef void (*cgx_source_hook)(void* user, int ncv, const double* rho, const double* u,
                                const double* rhoE, double* rhs, double time, int rk_stage);
int cgx_set_source_hook(cgx_solver* s, cgx_source_hook fn, void* user);

/*
 * cgx_set_frame_rotation: ROTATING_REFERENCE_FRAME wx wy wz (revolutions per
 * unit time; IdealGasSolver.hpp:126-142 turns them into radians, as here).
 * Each stage's rhs then takes addRotationSourceTerms (IdealGasSolver.cpp:
 * 695-733), after the source terms: the centrifugal -rho vol w x (w x x_cv)
 * and the Coriolis -2 rho vol w x u into rhs.rhou, and their dot product
 * with u into rhs.rhoE.  x_cv[ncv][3] are the cell centroids in reference
 * order.  A zero rate removes it.
 */
int cgx_set_frame_rotation(cgx_solver* s, const double rev_per_time[3], const double* x_cv);

/*
 * Boundary conditions of a mesh's boundary zones (registerBoundaryConditions,
 * IdealGasSolver.hpp:170-231).  Their fluxes enter each stage's rhs as
 * addBoundaryFlux does (IdealGasSolver.cpp:261-262) and their faces enter
 * calcCfl (IdealGasSolver.cpp:1068-1074):
 *   CGX_BC_SLIP            SLIP / SYMMETRY: rhs.rhou -= p n_bf
 *                          (SlipWallBc::addBoundaryFlux, IdealGasSolverBcs.cpp:14-23)
 *   CGX_BC_WALL_ADIABATIC  WALL_ADIABATIC [TRANSLATE u_wall]: tau = mu_lam
 *                          area_over_delta_bf (u - u_wall), rhs.rhou -= p n_bf +
 *                          tau, rhs.rhoE -= u_wall.tau
 *                          (WallAdiabatic::addBoundaryFlux, IdealGasSolverBcs.cpp:25-48;
 *                          u_wall = 0 by default, IdealGasSolverBcs.cpp:450-475)
 * u_wall may be NULL (zero).  Single-case solvers only: a batch refuses
 * meshes with boundary faces.
 */
#define CGX_BC_SLIP            1
#define CGX_BC_WALL_ADIABATIC  2
int cgx_set_bc(cgx_solver* s, int zone, int kind, const double u_wall[3]);

/*
 * Boundary conditions that take the reference's zone parameters, in the
 * order its input line gives them after the type name (params may be NULL
 * when nparams is 0):
 *   CGX_BC_SLIP             -
 *   CGX_BC_WALL_ADIABATIC   [u0 u1 u2]   (the TRANSLATE velocity)
 *   CGX_BC_WALL_ISOTHERMAL  T            WALL_ISOTHERMAL: tau = mu_lam
 *                           area_over_delta_bf u, q = loc_lam
 *                           area_over_delta_bf cp (T - T_bc); rhs.rhou -= p n_bf +
 *                           tau, rhs.rhoE -= q (WallIsothermal, IdealGasSolverBcs.cpp:1480-1510)
 *   CGX_BC_CBC_UPT          u0 u1 u2 p T (CbcUpt::initData, IdealGasSolverBcs.cpp:3182-3207)
 *   CGX_BC_CBC_RUNP         rho un p     inflow speed un against n_bf (CbcRunp::initData, :3242-3266)
 *   CGX_BC_CBC_MPT          mdot p T     mass flow rate into the zone over its whole area
 *                           (CbcMpt::initData, :3209-3240)
 * The CBC zones add the HLLC Riemann flux between the cell's state and the
 * zone's boundary state (Cbc::addBoundaryFlux, IdealGasSolverBcs.cpp:2960-2976;
 * calcRiemannFlux, IdealGasSolverFlux.hpp:218-306).  CBC zones carry no
 * transport scalars: cgx_init_complete refuses a solver that has both.
 * Returns CGX_E_ARG for an unknown kind, a zone out of range or a wrong
 * parameter count.
 */
#define CGX_BC_WALL_ISOTHERMAL 3
#define CGX_BC_CBC_UPT         4
#define CGX_BC_CBC_RUNP        5
#define CGX_BC_CBC_MPT         6
/* Characteristic zones whose boundary state follows the flow, updated in
 * each step as the reference's rk3Step of the zone does (before the stage's
 * RK update) and set after cgx_init_complete as initialHookBcs does:
 *   CGX_BC_CBC_EXTRAPOLATE  -             the boundary state is the cell's,
 *                           renewed every stage (CbcExtrapolate,
 *                           IdealGasSolverBcs.cpp:3436-3445, 3504-3576)
 *   CGX_BC_CBC_TOTAL_PT     p_total T_total t_relax: each face's normal
 *                           speed relaxes toward its cell's once per step
 *                           (eps = 1/(t_relax/dt + 1)), the rest from the
 *                           isentropic relations (CbcTotalPt,
 *                           IdealGasSolverBcs.cpp:3372-3434, 3447-3564; the
 *                           USE_AVG and STATIONARY_FRAME options are not built) */
#define CGX_BC_CBC_EXTRAPOLATE 7
#define CGX_BC_CBC_TOTAL_PT    8
/* Navier-Stokes characteristic zones: each face carries its own rho, p, u,
 * advanced by the zone's characteristic equations with the solver's RK3
 * weights (Nscbc::rk3Step, IdealGasSolverBcs.cpp:3651-3660), and stored and
 * restored with the state on a NaN (Nscbc::storeData/restoreData, :3578-3606):
 *   CGX_BC_NSCBC_MT        mdot T       subsonic inflow at a fixed mass flow
 *                          rate and static temperature (NscbcMt, :3722-3844;
 *                          the T_TOTAL form is not built)
 *   CGX_BC_NSCBC_OUTLET_P  p_ref sigma L_ref   partially reflecting pressure
 *                          outlet (NscbcOutletP, :3846-4092; sigma < 0: constant
 *                          pressure; the MDOT form is not built) */
#define CGX_BC_NSCBC_MT        9
#define CGX_BC_NSCBC_OUTLET_P  10
/*   CGX_BC_NSCBC_OUTLET_MDOT  mdot t_relax  outlet driving the zone's mean mass
 *                          flux toward mdot / area (NscbcOutletP, NSCBC_OUTLET_MDOT:
 *                          calcRhsMdot, IdealGasSolverBcs.cpp:3934-4007)
 * Zone-wide forms: CBC_TOTAL_PT takes an optional fourth parameter, 1 for
 * USE_AVG (one normal speed for the whole zone, relaxed toward its
 * density-weighted mean); NSCBC_MT with T < 0 takes -T as the total
 * temperature (T_TOTAL: the static temperature from the zone's mean Mach
 * number each stage).  Zone means are summed in a fixed order. */
#define CGX_BC_NSCBC_OUTLET_MDOT 11
/*   CGX_BC_CBC_RUP          rho u0 u1 u2 p  a fixed boundary state (CbcRup::initData,
 *                           IdealGasSolverBcs.cpp:3268-3333, without STATIONARY_FRAME)
 *   CGX_BC_WALL_CONDUCTIVE  T_end [L_1 k_1 L_2 k_2 ...]  a wall at rest behind
 *                           layers of thickness L_i and conductivity k_i ending at
 *                           T_end: q = (T - T_end) / (sum L_i/k_i / A + delta /
 *                           (loc_lam cp A)) / A (WallConductive, :2699-2743) */
#define CGX_BC_CBC_RUP         12
#define CGX_BC_WALL_CONDUCTIVE 13
/*   CGX_BC_SPONGE  type strength t_relax length p_sponge L_max
 *     a sponge layer (Sponge, IdealGasSolverBcs.cpp:4094-4363): each cell
 *     keeps a sponge state (T_sponge, u_sponge) that relaxes toward its own
 *     once per step (eps = 1/(t_relax/dt + 1)) and starts from it after
 *     cgx_init_complete; the zone's faces take the HLLC flux against their
 *     cell's sponge state at p_sponge, and the cells whose distance s along
 *     the layer's direction exceeds L_max - length are pulled toward it with
 *     strength ((s - L_max + length) / length)^2 per unit volume.  type: 0, 1,
 *     2 for x, y, z; 3 for the radius about the x axis, 4 about the z axis.
 *     L_max is the domain's largest extent in that direction (the reference
 *     takes it from the mesh nodes).  The sponge state is stored and restored
 *     with the flow state.  One sponge zone per solver; the mesh needs x_cv. */
#define CGX_BC_SPONGE          14
/*   CGX_BC_WM_ALG_ADIABATIC   [u_wall0 u_wall1 u_wall2]   (WM_ALG_ADIABATIC
 *     [TRANSLATE u]) and
 *   CGX_BC_WM_ALG_ISOTHERMAL  T_wall                       (WM_ALG_ISOTHERMAL T)
 *     the algebraic wall model (WmAdiabatic, WmIsothermal,
 *     IdealGasSolverBcs.cpp:996-1478, 2054-2262): once per step, at the
 *     first stage, each face's wall stress tau_wall comes from the law of the
 *     wall at the cell's distance y1 = |n_bf| / area_over_delta_bf and its
 *     speed along the wall (AlgebraicWM.hpp), from the last step's tau_wall as
 *     the first guess; the isothermal form adds the wall heat flux of the
 *     same model.  The wall force is tau_wall |n_bf| along the cell's wall-
 *     parallel velocity.  tau_wall starts from the laminar estimate after
 *     cgx_init_complete and is stored and restored with the state.  RELAX,
 *     Y_PLUS0 and TOL belong to the equilibrium (WM_EQ_*) forms, not built. */
#define CGX_BC_WM_ALG_ADIABATIC  15
#define CGX_BC_WM_ALG_ISOTHERMAL 16
/*   CGX_BC_WM_ALG_CONDUCTIVE  T_end [L_1 k_1 [L_2 k_2 ...]]   (WM_ALG_CONDUCTIVE
 *     T_end L_1 k_1 ... END) the algebraic wall model behind conducting
 *     layers (WmAlgConductive, IdealGasSolverBcs.cpp:2411-2560): tau_wall as
 *     WM_ALG_ISOTHERMAL, and the wall heat flux through the model's near-wall
 *     resistance (AlgebraicWM::compute_R_approx) in series with the layers'
 *     sum of L_i / k_i, toward T_end; no heat flux until the first step. */
#define CGX_BC_WM_ALG_CONDUCTIVE 17
/*   CGX_BC_CBC_PROFILE  (set with cgx_set_bc_profile)  CBC_PROFILE and
 *     CBC_PROFILE_SIMPLE (CbcProfile, CbcProfileSimple, IdealGasSolverBcs.cpp:
 *     3024-3180, 5339-5375): a characteristic zone whose boundary state is
 *     given face by face; the HLLC Riemann flux as the other CBC zones. */
#define CGX_BC_CBC_PROFILE       18
/*   CGX_BC_WM_EQ_ADIABATIC   [u_wall0 u_wall1 u_wall2 [relax y_plus0 tol]]
 *   CGX_BC_WM_EQ_ISOTHERMAL  T_wall [relax y_plus0 tol]
 *     the equilibrium wall model (WM_EQ_ADIABATIC, WM_EQ_ISOTHERMAL;
 *     EquilibriumWM::solve_qt, src/charles/wm/EquilibriumWM.hpp:36-204): once
 *     per step, at the first stage, the wall-layer momentum and energy
 *     equations are marched from the wall to the cell's distance y1 with a
 *     damped mixing-length eddy viscosity, and tau_wall (with the adiabatic
 *     wall temperature, or the isothermal wall's heat flux) is corrected
 *     until the march meets the cell's speed and temperature within tol.
 *     relax, y_plus0 and tol default to 0.7, 1 and 1e-4 (RELAX, Y_PLUS0,
 *     TOL).  The adiabatic form stores and restores tau_wall and its wall
 *     temperature with the state; the isothermal form keeps its own, as the
 *     reference does.  A march is cut off after 200000 steps in all (the
 *     reference has no bound; a face that needs more is degenerate). */
#define CGX_BC_WM_EQ_ADIABATIC   19
#define CGX_BC_WM_EQ_ISOTHERMAL  20
/*   CGX_BC_HOOK  (no parameters)  HOOK (initHookBc, IdealGasSolver.hpp:221,
 *     251): a zone whose condition is the caller's own code.  Its faces add
 *     nothing on the device; the caller's addBoundaryFlux (and calcRhs,
 *     rk3Step) run in the host hook of cgx_set_source_hook, which adds to the
 *     stage's rhs of the zone's cells.  Transport scalars are refused with
 *     it, as with the CBC zones. */
#define CGX_BC_HOOK              21
/*   CGX_BC_WM_EXCHANGE_ADIABATIC   [del_exch_ratio]
 *   CGX_BC_WM_EXCHANGE_ISOTHERMAL  T_wall [del_exch_ratio]
 *     the algebraic wall model fed from off the wall (WmExchange,
 *     IdealGasSolverBcs.cpp:500-990): once per step, at the first stage, each
 *     face's velocity comes from its exchange point x_ex = x_bf - ratio
 *     delta n_hat (ratio 3 by default), reconstructed in the cell that holds
 *     it as u + dudx (x_ex - x_cv), and the model is solved at distance ratio
 *     delta; a face whose point was not located uses its own cell at delta.
 *     The exchange points' cells and positions are set with
 *     cgx_set_bc_exchange before cgx_init_complete. */
#define CGX_BC_WM_EXCHANGE_ADIABATIC  22
#define CGX_BC_WM_EXCHANGE_ISOTHERMAL 23
int cgx_set_bc_params(cgx_solver* s, int zone, int kind, const double* params, int nparams);

/* A CBC_PROFILE zone from the boundary states of its faces: bf_state
 * [nbf_zone][6] = u[0], u[1], u[2], sp_vol, p, h of each face (the members of
 * the reference's IdealGasState that Cbc::addBoundaryFlux reads), the zone's
 * faces in the order the mesh description lists them.  The reference reads a
 * profile file and interpolates it to the faces in CbcProfile::initData; the
 * caller passes the interpolated states.
 * nbf_zone must be the zone's face count. */
int cgx_set_bc_profile(cgx_solver* s, int zone, const double* bf_state, int nbf_zone);

/* A velocity face by face, u_bf[nbf_zone][3], the zone's faces in the order
 * the mesh description lists them (CBC_RUP: the STATIONARY_FRAME velocity
 * u_fr; its u_bc then turns with the frame, CbcRup::calcBfState, :3335-3348;
 * NSCBC zones: the frame velocity u_fr =
 * -w x x_bf that the reference forms in a rotating frame, NscbcMt::initData,
 * :3752-3770: its part along the face joins NSCBC_MT's u_bc, and the
 * outlets' centrifugal term is w x u_fr; the outlets' Coriolis term needs no
 * per-face data):
 *   WALL_ADIABATIC, WM_ALG_ADIABATIC, WM_EQ_ADIABATIC: the wall's velocity,
 *     the zones' u_bc after their initData (IdealGasSolverBcs.cpp:450-497,
 *     996-1041): TRANSLATE gives every face the same velocity,
 *     STATIONARY_FRAME in a rotating frame gives each face -w x x_bf;
 *   CBC_TOTAL_PT: the frame velocity u_fr of STATIONARY_FRAME (-w x x_bf,
 *     CbcTotalPt::initData, :3372-3405), whose part along the face enters
 *     the boundary state beside the relaxed normal speed (calcBfState,
 *     :3413-3434).
 * Set the zone's kind first (cgx_set_bc_params); setting the kind again
 * returns the zone to its one velocity (or to no frame velocity). */
int cgx_set_bc_face_velocity(cgx_solver* s, int zone, const double* u_bf, int nbf_zone);

/* The exchange points of a WM_EXCHANGE zone's faces (WmExchange::initData and
 * its DataExchanger, IdealGasSolverBcs.cpp:500-575): cv_ex[nbf_zone] the cell
 * (reference numbering) that holds each face's point, or -1 where the point
 * was not located, and x_ex[nbf_zone][3] the points, the zone's faces in the
 * order the mesh description lists them.  The mesh needs x_cv. */
int cgx_set_bc_exchange(cgx_solver* s, int zone, const int* cv_ex, const double* x_ex, int nbf_zone);

/* initComplete: updateConservativeAndPrimitiveData + calcSgsAndMaterialProperties,
 * then stores the state for NaN recovery (initialHookBcs -> storeData). */
int cgx_init_complete(cgx_solver* s);
int cgx_update_primitive(cgx_solver* s);
int cgx_calc_sgs_props(cgx_solver* s);

/* calcRhs into the solver's rhs buffer of rk_stage (1..3), which is zeroed
 * first; if rhs_out != NULL the result is also copied out in reference order
 * as [ncv][5] (unscaled face sums, as the reference stores them). */
int cgx_calc_rhs(cgx_solver* s, double* rhs_out, double time, int rk_stage);
/* rk3Step with weights w over the rhs buffers of stages 1..rk_stage. */
int cgx_rk3_step(cgx_solver* s, const double w[3], double dt, int rk_stage);
/* calcCfl(cfl, dt): rank-local max; cfl[ncv] optional (reference order). */
int cgx_calc_cfl(cgx_solver* s, double dt, double* cfl_max, double* cfl);

/* One advanceSolution with the current dt (setDt not included).  Returns
 * CGX_E_NAN after restoring the stored state and scaling dt_data[0] by 0.8. */
int cgx_advance_solution(cgx_solver* s);
/* nsteps of {setDt; advanceSolution}, dt and time kept on the device, the
 * step replayed from a CUDA graph.  NaNs are checked whenever the global step
 * count reaches a multiple of check_interval and after the last step, and the
 * restore point is stored at multiples of 20 check_intervals
 * (IdealGasSolver.hpp:807-811; CGX_E_NAN as above). */
int cgx_step(cgx_solver* s, int nsteps);
/* cgx_step, then the state in the caller's host arrays (cgx_get_state's
 * layout), for a host solver that keeps its arrays on the host.  The copy of
 * the last step's state starts as soon as its last RK update is done and runs
 * beside the step's remaining kernels (the gradient and the once-per-step
 * properties, which do not change the state); pageable arrays go through the
 * library's pinned chunks on that copy.  On CGX_E_NAN the arrays hold the
 * restored state. */
int cgx_step_out(cgx_solver* s, int nsteps, double* rho, double* u, double* rhoE);

/* time, dt of the last completed step (0 before the first) and step count */
int cgx_get_time(cgx_solver* s, double* time, double* dt, int* step);
/* Restart: set the solver's time and step count, as a host solver does after
 * reading them from a restart file.  After cgx_init_complete the current
 * state becomes the restore point. */
int cgx_set_time(cgx_solver* s, double time, int step);
/* report(): {sum rho V, sum rho u V (3), sum rhoE V}, fixed-order reduction. */
int cgx_totals(cgx_solver* s, double out[5]);

/* Diagnostics in reference order: p, T, sos [ncv]; dudx [ncv][3][3];
 * aux [ncv][6] = {mu_total, loc_total, a_sgs, fgr, symh_fax, symp_fax}. */
int cgx_get_primitive(cgx_solver* s, double* p, double* T, double* sos);
int cgx_get_grad(cgx_solver* s, double* dudx);
int cgx_get_aux(cgx_solver* s, double* aux);

int cgx_synchronize(cgx_solver* s);

/* Timing hooks (no counterpart in the reference, which prints wall time per
 * step, FlowSolver.hpp:2596-2605): run nsteps as cgx_step does and return
 * their device time from CUDA events on the solver's stream. */
int cgx_step_timed(cgx_solver* s, int nsteps, float* device_ms);
/* As cgx_step_timed, with the two face-flux kernels of calcRhs timed inside
 * the steps by CUDA events recorded in the step graph around them:
 * face_ms = {average launch time of the pair (extended faces + compact
 * closures), of the extended-face kernel, of the compact-closure kernel}
 * over the 3 x nsteps stages.  The host waits for each step before the next
 * one (the marks are reused), which device_ms includes. */
int cgx_step_profiled(cgx_solver* s, int nsteps, float* device_ms, double face_ms[3]);
/* Average device time of one launch of each step kernel, measured with CUDA
 * events over `reps` back-to-back launches: ms[0] face fluxes (calcRhs, both
 * kernels), ms[1] rk3Step + packed state (3 weights, dt = 0 so the state is
 * kept), ms[2] gradient, ms[3] once-per-step SGS/properties/sensor/CFL,
 * ms[4] the extended-face flux kernel alone, ms[5] the compact-closure kernel
 * alone.  Overwrites the stage-0 rhs. */
int cgx_kernel_times(cgx_solver* s, int reps, double ms[6]);
/* Lanes per cell chosen by the autotuner that cgx_init_complete runs (timed
 * candidates per kernel, cached per mesh-size bucket and precision):
 * out = {face fluxes, compact closures, gradient, once-per-step kernel}. */
int cgx_get_tuning(const cgx_solver* s, int out[4]);
/* Number of this library's kernels launched by the handle so far. */
long long cgx_launch_count(const cgx_solver* s);
/* Self-test of the device reciprocal that the flux kernels use for the face
 * density 2/(v0+v1) and the face Mach number |u_n|/c (no counterpart in the
 * reference, which divides in IEEE FP64): out[i] = that reciprocal of x[i]
 * for n host values, evaluated on `device`. */
int cgx_selftest_rcp(int device, const double* x, double* out, int n);
/* Host threads that the calling thread's later calls run their parallel
 * host phases on (cgx_mesh_create, cgx_operators_build's host side, the
 * host generator): n > 0 sets the count, n <= 0 restores all cores.  Other
 * threads are not affected, so a thread that admits new meshes while others
 * step can leave cores to them. */
int cgx_set_host_threads(int n);

/*
 * Batched and served form (no single reference counterpart: the reference
 * runs one case per process, FlowSolver::run, FlowSolver.hpp:2445-2678).
 * A batch holds many resident cases of uneven size on one device and
 * advances them together: each step is one replay of a CUDA graph whose
 * kernels walk a packed work list of cell blocks across all active cases.
 * Cases join and leave between steps (continuous batching); their state
 * stays on the device.  Every case keeps its own parameters, dt (its own
 * CFL reduction), time, step count and NaN recovery.
 */
typedef struct cgx_batch cgx_batch;

/* max_cases resident at once; hbm_budget_bytes bounds the device memory the
 * batch's cases may hold (their meshes counted once each). */
int cgx_batch_create(int device, cgx_precision prec, int max_cases, size_t hbm_budget_bytes,
                     cgx_batch** out);
int cgx_batch_destroy(cgx_batch* b);
/* Admit a case on a device mesh (shared with other cases, not owned): state
 * from rho, u, p as cgx_set_state_primitive, then initComplete.  The case
 * advances with the batch until it has taken nsteps steps.  Returns
 * CGX_E_OOM, allocating nothing, when the case would exceed the budget. */
int cgx_batch_add(cgx_batch* b, cgx_mesh* mesh, const cgx_params* p, const double* rho,
                  const double* u, const double* pres, int nsteps, int* case_id);
/* cgx_batch_add in two parts, so that a server can build new cases while the
 * batch steps.  cgx_batch_prepare creates the case's solver on its own
 * stream, sets its state and runs initComplete (with the batch's lane counts:
 * no tuning); it reads only the batch's device and precision, so another
 * host thread may call it while cgx_batch_step runs.  cgx_batch_admit joins a
 * prepared case between steps (a slot, its descriptor, the budget check:
 * CGX_E_OOM leaves the case prepared, to be admitted later or released) and
 * takes ownership of it on success.  The mesh must outlive the case. */
typedef struct cgx_batch_case cgx_batch_case;
int cgx_batch_prepare(cgx_batch* b, cgx_mesh* mesh, const cgx_params* p, const double* rho,
                      const double* u, const double* pres, int nsteps, cgx_batch_case** out);
int cgx_batch_admit(cgx_batch* b, cgx_batch_case* c, int* case_id);
int cgx_batch_case_release(cgx_batch_case* c);
/* Advance every active case by up to nsteps steps (a case stops at its own
 * step count); *n_done = cases that have finished and not been removed. */
int cgx_batch_step(cgx_batch* b, int nsteps, int* n_done);
/* Ids of finished cases not yet removed (up to max). */
int cgx_batch_done(cgx_batch* b, int* ids, int max, int* n);
int cgx_batch_get_state(cgx_batch* b, int case_id, double* rho, double* u, double* rhoE);
int cgx_batch_get_time(cgx_batch* b, int case_id, double* time, double* dt, int* step);
int cgx_batch_remove(cgx_batch* b, int case_id);
/* Device bytes held by resident cases (meshes once each) and the budget. */
int cgx_batch_bytes(const cgx_batch* b, size_t* used, size_t* budget);
long long cgx_batch_launch_count(const cgx_batch* b);

/*
 * report() totals that allocate nothing (no counterpart in the reference).
 * For host solvers that cannot call cudaMalloc -- for instance because their
 * device memory comes from another allocator or is fixed at start-up -- this
 * computes {sum rho V, sum rho u V (3), sum rhoE V} over caller-owned device
 * arrays rho[n], u[n][3] (the reference's interleaved layout), rhoE[n],
 * vol[n] into the caller's device array out5[5], on `stream` (a
 * cudaStream_t; NULL for the legacy default stream), without allocating.
 * The reduction's scratch is a file-scope device array of 8192 x 5 doubles
 * (320 KiB, held by every GPU that loads this library until the process
 * exits); n is limited to 16,777,216 cells (8192 blocks of 2048) and larger
 * n is rejected with CGX_E_ARG.  The first call on a device looks up the
 * array's device address and keeps it for the life of the process; make that
 * first call before any stream capture.  cudaDeviceReset (or any other
 * teardown of the device's primary context) reloads the module and leaves
 * the kept address stale: do not call this entry point on a device after
 * resetting it.
 * All calls share the array: calls that overlap on the GPU (other streams,
 * other host threads) race, so serialise them.  Returns without waiting for
 * the GPU.
 */
int cgx_totals_noalloc(long long n, const double* rho, const double* u, const double* rhoE,
                       const double* vol, double* out5, void* stream);

const char* cgx_last_error(void);

#ifdef __cplusplus
}
#endif
#endif
