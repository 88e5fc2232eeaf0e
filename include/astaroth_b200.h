/*
 * astaroth_b200 -- C ABI of the B200 (sm_100a) single-GPU MHD integrator.
 *
 * A drop-in for the device layer of Astaroth (include/astaroth_device.h and
 * src/core/device.cc in the reference): same function names, argument meaning,
 * buffer semantics (in/out per field, swap after every substep) and AcResult
 * return codes, for the 8-field compressible non-ideal MHD module (lnrho, uu,
 * aa, entropy; 6th-order central differences, periodic box, 2N RK3).
 *
 * Every declaration below names the reference interface it replaces as
 * file:line in the reference tree.  Types are plain C: pointers, sizes,
 * enums and small structs; no CUDA or torch header is needed (the one CUDA
 * stream handle, of acDeviceFinishReduceRealStream, is an opaque struct
 * pointer).
 */
#pragma once

#include <stdbool.h>
#include <stddef.h>

#ifdef __cplusplus
#define AC_BEGIN_C_DECLARATIONS extern "C" {
#define AC_END_C_DECLARATIONS }
#else
#define AC_BEGIN_C_DECLARATIONS
#define AC_END_C_DECLARATIONS
#endif

/* ---------------------------------------------------------------------------
 * Basic types
 * (acc-runtime/api/acreal.h:3-4, include/host_datatypes.h:10,
 *  acc-runtime/acc/implementation.c:3-5)
 * ------------------------------------------------------------------------- */
typedef double AcReal; /* FP64 build of the reference (AC_DOUBLE_PRECISION=1) */
#define AC_REAL_EPSILON (2.2204460492503131e-16)

typedef enum { AC_SUCCESS = 0, AC_FAILURE = 1, AC_NOT_ALLOCATED = 2 } AcResult;

typedef struct {
    size_t x, y, z;
} Volume;

#ifndef INT3_DEFINED
#ifndef __CUDACC__
typedef struct {
    int x, y, z;
} int3;
#endif
#define INT3_DEFINED
#endif

typedef struct {
    AcReal x, y, z;
} AcReal3;

/* Field handles in declaration order of
 * acc-runtime/samples/mhd_modular/mhdsolver.ac:125,136,140 (LENTROPY=1,
 * LMAGNETIC=1, LBFIELD=0). */
typedef enum {
    VTXBUF_LNRHO = 0,
    VTXBUF_UUX,
    VTXBUF_UUY,
    VTXBUF_UUZ,
    VTXBUF_AX,
    VTXBUF_AY,
    VTXBUF_AZ,
    VTXBUF_ENTROPY,
    NUM_VTXBUF_HANDLES
} VertexBufferHandle;
typedef VertexBufferHandle Field;
#define NUM_FIELDS (NUM_VTXBUF_HANDLES)
#define STENCIL_ORDER (6)
#define NGHOST (STENCIL_ORDER / 2)

/* Streams: include/astaroth_base.h:49-86 (32 streams and STREAM_ALL). */
typedef enum {
    STREAM_0, STREAM_1, STREAM_2, STREAM_3, STREAM_4, STREAM_5, STREAM_6, STREAM_7,
    STREAM_8, STREAM_9, STREAM_10, STREAM_11, STREAM_12, STREAM_13, STREAM_14, STREAM_15,
    STREAM_16, STREAM_17, STREAM_18, STREAM_19, STREAM_20, STREAM_21, STREAM_22, STREAM_23,
    STREAM_24, STREAM_25, STREAM_26, STREAM_27, STREAM_28, STREAM_29, STREAM_30, STREAM_31,
    STREAM_ALL
} Stream;
#define NUM_STREAMS (32)
static const Stream STREAM_DEFAULT = STREAM_0;

/* ---------------------------------------------------------------------------
 * Mesh configuration.  The reference's AcMeshInfo is generated by its DSL
 * compiler (acc-runtime/api/acc_runtime.h:157-175), so binary layout
 * compatibility is impossible; this struct keeps the same parameter names and
 * the same access forms (info.real_params[AC_x] in C, info[AC_x] in C++).
 * ------------------------------------------------------------------------- */
typedef enum {
    /* Storage and arithmetic of the device fields: 0 = FP64 (the reference),
     * 1 = FP32 fields with a compensated FP32 hi/lo RK3 accumulator. */
    AC_precision = 0,
    /* calc_timestep variant (mhdsolver.ac:551-583): 0 = max reductions,
     * 1 = additive (min over cells of the local dt). */
    AC_additive_timestep,
    /* Selects the solve kernel (for tests and timing): 0 = the default (the
     * split-stage kernel where it takes the mesh, but for small FP64 meshes with
     * an odd x side, else the per-plane tap kernel, else the plain one), 1 = the plain (untiled) kernel, 2 = the tiled kernel
     * that reads every stencil tap of plane z from shared memory, 3 (and 4) =
     * the split-stage kernel for every mesh that it takes. */
    AC_debug_plain_kernel,
    /* Upwinding terms of the continuity and momentum equations when nonzero:
     * the reference's LUPWD build option (mhdsolver.ac:101,336-338,357-359;
     * model src/utils/modelsolver.cc:424-506,776-779,837-841). */
    AC_upwind,
    /* Helical forcing in substep 2 when nonzero (the reference's LFORCING,
     * mhdsolver.ac:524-549 `AC_lforcing`). */
    AC_lforcing,
    /* The auxiliary field B = curl A of the input of substep 2, kept for
     * acDeviceStoreBfield when nonzero (the reference's LBFIELD,
     * mhdsolver.ac:103,147-151,546-548,605-608). */
    AC_lbfield,
    NUM_INT_PARAMS
} AcIntParam;

typedef enum {
    AC_ngrid = 0,       /* global interior size */
    AC_nlocal,          /* interior size held by this device (= AC_ngrid on one GPU) */
    AC_nmin,            /* first interior index, (3,3,3) */
    AC_nlocal_max,      /* AC_nmin + AC_nlocal */
    AC_ngrid_max,       /* AC_nmin + AC_ngrid */
    AC_mlocal,          /* AC_nlocal + 2*NGHOST: allocated size per axis */
    AC_mgrid,           /* AC_ngrid + 2*NGHOST */
    AC_multigpu_offset, /* (0,0,0) on one GPU */
    NUM_INT3_PARAMS
} AcInt3Param;

typedef enum {
    AC_nu_visc = 0,
    AC_eta,
    AC_cs_sound,
    AC_gamma,
    AC_cp_sound,
    AC_lnrho0,
    AC_lnT0,
    AC_mu0,
    AC_zeta,
    AC_K_heatcond,
    AC_cdt,          /* Courant factor for advection (config/astaroth.conf:45) */
    AC_cdtv,         /* Courant factor for diffusion (config/astaroth.conf:46) */
    AC_chi,          /* thermal diffusivity used by the timestep bound */
    AC_current_time,
    AC_cs2_sound,    /* derived: cs_sound^2 */
    AC_dsmin,        /* derived: min(ds) */
    /* Helical forcing (the reference's LFORCING option, mhdsolver.ac:286-331,
     * model src/utils/modelsolver.cc:1003-1076; parameters
     * src/utils/astaroth_forcing.cc:229-283, config/astaroth.conf:58-61).
     * Applied in substep 2 when AC_lforcing is set and AC_current_time >
     * AC_switch_forcing. */
    AC_forcing_magnitude,
    AC_forcing_phase,
    AC_k_forcex,
    AC_k_forcey,
    AC_k_forcez,
    AC_ff_hel_rex,
    AC_ff_hel_rey,
    AC_ff_hel_rez,
    AC_ff_hel_imx,
    AC_ff_hel_imy,
    AC_ff_hel_imz,
    AC_kaver,
    AC_switch_forcing,
    AC_relhel,       /* relative helicity, input of acHostForcingParams */
    AC_kmin,         /* forcing wave-number shell, input of acHostGenerateForcingParams */
    AC_kmax,
    NUM_REAL_PARAMS
} AcRealParam;

typedef enum {
    AC_ds = 0,   /* grid spacing */
    AC_inv_ds,   /* derived: 1/ds */
    AC_inv_ds_2, /* derived: 1/ds^2 */
    AC_len,      /* derived: ds * ngrid */
    NUM_REAL3_PARAMS
} AcReal3Param;

typedef struct AcMeshInfo {
    int int_params[NUM_INT_PARAMS];
    int3 int3_params[NUM_INT3_PARAMS];
    AcReal real_params[NUM_REAL_PARAMS];
    AcReal3 real3_params[NUM_REAL3_PARAMS];
#ifdef __cplusplus
    int& operator[](const AcIntParam p) { return int_params[p]; }
    int operator[](const AcIntParam p) const { return int_params[p]; }
    int3& operator[](const AcInt3Param p) { return int3_params[p]; }
    int3 operator[](const AcInt3Param p) const { return int3_params[p]; }
    AcReal& operator[](const AcRealParam p) { return real_params[p]; }
    AcReal operator[](const AcRealParam p) const { return real_params[p]; }
    AcReal3& operator[](const AcReal3Param p) { return real3_params[p]; }
    AcReal3 operator[](const AcReal3Param p) const { return real3_params[p]; }
#endif
} AcMeshInfo;

/* Host mesh: include/astaroth_base.h:35-39. */
typedef struct {
    AcReal* vertex_buffer[NUM_VTXBUF_HANDLES];
    AcMeshInfo info;
} AcMesh;

/* ---------------------------------------------------------------------------
 * Reductions: the AcReduction record of acc-runtime/api/acc_runtime.h:78-86
 * and the reduction types of stdlib/reduction.h:1-8.
 * ------------------------------------------------------------------------- */
typedef enum AcReduceOp {
    AC_REDUCE_OP_NO_REDUCE,
    AC_REDUCE_OP_MIN,
    AC_REDUCE_OP_MAX,
    AC_REDUCE_OP_SUM,
} AcReduceOp;
typedef enum { AC_NO_REDUCE_POST_PROCESSING = 0, AC_RMS = 1 } AcReductionPostProcessingOp;
/* Map kernels of acc-runtime/stdlib/map.h:29-150 used by the reductions. */
typedef enum {
    AC_NULL_KERNEL = 0,
    AC_MAP_VTXBUF,
    AC_MAP_VTXBUF_SQUARE,
    AC_MAP_VTXBUF_EXP_SQUARE,
    AC_MAP_VTXBUF3_NORM,
    AC_MAP_VTXBUF3_SQUARE,
    AC_MAP_VTXBUF3_EXP_SQUARE,
    AC_MAP_VTXBUF4_ALFVEN_NORM,
    AC_MAP_VTXBUF4_ALFVEN_SQUARE,
    NUM_MAP_KERNELS,
    /* the kernels whose launches reduce the CFL outputs below: the substep
     * kernel (its substep 2) and the stand-alone calc_timestep
     * (acc-runtime/samples/mhd_modular/mhdsolver.ac:551-583,611) */
    AC_KERNEL_SOLVE = NUM_MAP_KERNELS,
    AC_KERNEL_CALC_TIMESTEP,
    NUM_KERNELS
} AcKernel;

/* The real outputs that calc_timestep reduces (mhdsolver.ac:570,574-575):
 * max |u|, max Alfven speed |curl A| / sqrt(exp(lnrho)), and for
 * AC_additive_timestep = 1 the minimum over cells of min(visc_dt, advec_dt). */
typedef enum {
    UU_MAX_ADVEC,
    ALFVEN_SPEED_MAX,
    AC_dt_min,
    NUM_REAL_OUTPUTS
} AcRealOutputParam;
typedef struct {
    AcReduceOp reduce_op;
    AcReductionPostProcessingOp post_processing_op;
    AcKernel map_vtxbuf_single;
    AcKernel map_vtxbuf_vec;
    AcKernel map_vtxbuf_vec_scal;
    const char* name;
} AcReduction;

static const AcReduction RTYPE_MAX = {AC_REDUCE_OP_MAX, AC_NO_REDUCE_POST_PROCESSING,
                                      AC_MAP_VTXBUF, AC_MAP_VTXBUF3_NORM, AC_NULL_KERNEL,
                                      "RTYPE_MAX"};
static const AcReduction RTYPE_MIN = {AC_REDUCE_OP_MIN, AC_NO_REDUCE_POST_PROCESSING,
                                      AC_MAP_VTXBUF, AC_MAP_VTXBUF3_NORM, AC_NULL_KERNEL,
                                      "RTYPE_MIN"};
static const AcReduction RTYPE_SUM = {AC_REDUCE_OP_SUM, AC_NO_REDUCE_POST_PROCESSING,
                                      AC_MAP_VTXBUF, AC_MAP_VTXBUF3_NORM, AC_NULL_KERNEL,
                                      "RTYPE_SUM"};
static const AcReduction RTYPE_RMS = {AC_REDUCE_OP_SUM, AC_RMS, AC_MAP_VTXBUF_SQUARE,
                                      AC_MAP_VTXBUF3_SQUARE, AC_NULL_KERNEL, "RTYPE_RMS"};
static const AcReduction RTYPE_RMS_EXP = {AC_REDUCE_OP_SUM, AC_RMS, AC_MAP_VTXBUF_EXP_SQUARE,
                                          AC_MAP_VTXBUF3_EXP_SQUARE, AC_NULL_KERNEL,
                                          "RTYPE_RMS_EXP"};
static const AcReduction RTYPE_ALFVEN_MAX = {AC_REDUCE_OP_MAX, AC_NO_REDUCE_POST_PROCESSING,
                                             AC_NULL_KERNEL, AC_NULL_KERNEL,
                                             AC_MAP_VTXBUF4_ALFVEN_NORM, "RTYPE_ALFVEN_MAX"};
static const AcReduction RTYPE_ALFVEN_MIN = {AC_REDUCE_OP_MIN, AC_NO_REDUCE_POST_PROCESSING,
                                             AC_NULL_KERNEL, AC_NULL_KERNEL,
                                             AC_MAP_VTXBUF4_ALFVEN_NORM, "RTYPE_ALFVEN_MIN"};
static const AcReduction RTYPE_ALFVEN_RMS = {AC_REDUCE_OP_SUM, AC_RMS, AC_NULL_KERNEL,
                                             AC_NULL_KERNEL, AC_MAP_VTXBUF4_ALFVEN_SQUARE,
                                             "RTYPE_ALFVEN_RMS"};

/* Opaque device handle: include/astaroth_base.h:135. */
typedef struct device_s* Device;
struct CUstream_st; /* a CUDA stream handle (cudaStream_t) */

AC_BEGIN_C_DECLARATIONS

/* ---------------------------------------------------------------------------
 * Host helpers (src/core/astaroth.cc, src/core/update_params/update_params.cc)
 * ------------------------------------------------------------------------- */

/* Fills the derived params (nlocal, nmin, mlocal, inv_ds, cs2_sound, ...).
 * Replaces acHostUpdateParams, include/astaroth_helpers.h:291. */
AcResult acHostUpdateParams(AcMeshInfo* info);

/* Sets the defaults of config/astaroth.conf for this module and the given
 * cubic size n with ds = 2*pi/n; the caller may override any field after.
 * Plays the role of acLoadConfig(AC_DEFAULT_CONFIG, ...), include/astaroth.h. */
AcResult acHostMeshInfoDefault(const int nx, const int ny, const int nz, AcMeshInfo* info);

/* Reads `key = value` lines (the reference's .conf syntax) into info.
 * Replaces acLoadConfig, src/utils/config_loader.cc. Unknown keys are ignored. */
AcResult acLoadConfig(const char* path, AcMeshInfo* info);

/* Allocates (zeroed) host field arrays of the full size incl. halos.
 * Replaces acHostMeshCreate / acHostMeshDestroy, include/astaroth_helpers.h:301,318. */
AcResult acHostMeshCreate(const AcMeshInfo info, AcMesh* mesh);
AcResult acHostMeshDestroy(AcMesh* mesh);

/* Helical forcing parameters (src/utils/astaroth_forcing.cc:137-256,
 * generateForcingParams and helpers).  acHostForcingParams takes the three
 * random draws of the reference -- the wave vector k_force (an integer vector
 * of the shell AC_kmin <= |k| <= AC_kmax), the angle phi of the helical basis
 * vector about k, and the phase -- and sets AC_k_force*, AC_ff_hel_re*,
 * AC_ff_hel_im* (with AC_relhel), AC_forcing_phase and AC_kaver =
 * (AC_kmax - AC_kmin) / 2 as the reference computes them.
 * acHostGenerateForcingParams draws them from a counter-based generator of
 * (seed, step): reproducible, but not the reference's random sequence. */
AcResult acHostForcingParams(const AcReal3 k_force, const AcReal phi, const AcReal phase,
                             AcMeshInfo* info);
AcResult acHostGenerateForcingParams(const unsigned long long seed, const unsigned long long step,
                                     AcMeshInfo* info);

/* Host snapshots in the reference's format (src/utils/memory.cc:182-247,
 * declared in include/astaroth_utils.h:79-81): data-format.csv
 * ("use_double, mx, my, mz" and their values) and <VTXBUF name>-<id, 5 digits>.dat
 * per field with every cell incl. halos, in the current directory.  Read
 * checks the header against mesh->info and fails on any mismatch or short file. */
AcResult acHostMeshWriteToFile(const AcMesh mesh, const size_t id);
AcResult acHostMeshReadFromFile(const size_t id, AcMesh* mesh);

/* Seeded initial conditions (no counterpart in the reference, which only has
 * rand()/RAND_MAX, src/core/astaroth.cc:391-401).  Counter-based splitmix64
 * indexed by (seed, field, i, j, k): lnrho, entropy ~ U(-amp_s, amp_s);
 * uu ~ N(0, sigma_u^2); aa ~ N(0, sigma_a^2); every cell incl. halos.
 * Fields whose vertex_buffer is NULL are skipped (each field's values do not
 * depend on the others, so a mesh can be generated one field at a time). */
AcResult acHostMeshRandomizeSeeded(AcMesh* mesh, const unsigned long long seed,
                                   const AcReal amp_scalar, const AcReal sigma_uu,
                                   const AcReal sigma_aa);

/* Replaces uu by a solenoidal superposition of nmodes random Fourier modes
 * with integer wave vectors |k| <= kmax, normalised so that max|u| over the
 * modes' amplitudes is `amplitude` (u = sum a_m (k_m x e_m) sin(k_m.x + phi_m)).
 * Interior and halos are written (periodic by construction).  The three uu
 * buffers must be allocated. */
AcResult acHostMeshSolenoidalModes(AcMesh* mesh, const unsigned long long seed,
                                   const int nmodes, const int kmax, const AcReal amplitude);

/* CFL timestep of samples/standalone_mpi/main.cc:396-441 from the two device
 * maxima (max |u| and max Alfven speed). */
AcReal acHostTimestepFromMaxima(const AcMeshInfo info, const AcReal uu_max,
                                const AcReal alfven_max);

/* ---------------------------------------------------------------------------
 * Device interface: include/astaroth_device.h
 * ------------------------------------------------------------------------- */

/* include/astaroth_device.h:13 -- allocates and zero-fills 2 x 8 field buffers. */
AcResult acDeviceCreate(const int id, const AcMeshInfo device_config, Device* device);
/* include/astaroth_device.h:15 -- frees everything and sets *device = NULL. */
AcResult acDeviceDestroy(Device* device);
/* include/astaroth_device.h:18 -- zero-fills both buffers of every field. */
AcResult acDeviceResetMesh(const Device device, const Stream stream);
/* include/astaroth_device.h:20 */
AcResult acDevicePrintInfo(const Device device);
/* include/astaroth_device.h:24 */
AcResult acDeviceSynchronizeStream(const Device device, const Stream stream);
/* include/astaroth_device.h:26,28 -- pointer swaps of in/out. */
AcResult acDeviceSwapBuffer(const Device device, const VertexBufferHandle handle);
AcResult acDeviceSwapBuffers(const Device device);
/* include/astaroth_device.h:32 */
AcResult acDeviceLoadScalarUniform(const Device device, const Stream stream,
                                   const AcRealParam param, const AcReal value);
/* include/astaroth_device.h:47 */
AcResult acDeviceLoadVectorUniform(const Device device, const Stream stream,
                                   const AcReal3Param param, const AcReal3 value);
/* include/astaroth_device.h:50 */
AcResult acDeviceLoadIntUniform(const Device device, const Stream stream,
                                const AcIntParam param, const int value);
/* include/astaroth_device.h:58 */
AcResult acDeviceStoreScalarUniform(const Device device, const Stream stream,
                                    const AcRealParam param, AcReal* value);
/* include/astaroth_device.h:61 (vector) and the generated
 * device_load_uniform_decl.h / device_store_uniform_decl.h included at
 * include/astaroth_device.h:86,91 (int, int3).  Loading an int3 parameter
 * goes through the same checks as acDeviceLoadMeshInfo: the mesh dimensions
 * cannot change after acDeviceCreate. */
AcResult acDeviceStoreVectorUniform(const Device device, const Stream stream,
                                    const AcReal3Param param, AcReal3* value);
AcResult acDeviceStoreIntUniform(const Device device, const Stream stream,
                                 const AcIntParam param, int* value);
AcResult acDeviceStoreInt3Uniform(const Device device, const Stream stream,
                                  const AcInt3Param param, int3* value);
AcResult acDeviceLoadInt3Uniform(const Device device, const Stream stream,
                                 const AcInt3Param param, const int3 value);
/* include/astaroth_device.h:64 -- sizes must match the created device. */
AcResult acDeviceLoadMeshInfo(const Device device, const AcMeshInfo device_config);
/* include/astaroth_device.h:103 */
AcMeshInfo acDeviceGetConfig(const Device device);
/* include/astaroth_device.h:77,80 -- H2D of the in buffer incl. halos. */
AcResult acDeviceLoadVertexBuffer(const Device device, const Stream stream,
                                  const AcMesh host_mesh, const VertexBufferHandle vtxbuf_handle);
AcResult acDeviceLoadMesh(const Device device, const Stream stream, const AcMesh host_mesh);
/* include/astaroth_device.h:94 -- sets every cell of the in buffer. */
AcResult acDeviceSetVertexBuffer(const Device device, const Stream stream,
                                 const VertexBufferHandle handle, const AcReal value);
/* include/astaroth_device.h:97 -- zero-fills the out buffers. */
AcResult acDeviceFlushOutputBuffers(const Device device, const Stream stream);
/* include/astaroth_device.h:112,115 -- D2H of the in buffer incl. halos. */
AcResult acDeviceStoreVertexBuffer(const Device device, const Stream stream,
                                   const VertexBufferHandle vtxbuf_handle, AcMesh* host_mesh);
AcResult acDeviceStoreMesh(const Device device, const Stream stream, AcMesh* host_mesh);

/* Linear ranges: include/astaroth_device.h:67,73,99,109 (host <-> device) and
 * :118,124,128,131 (device -> device; src/core/device.cc:666-698 and the
 * store/transfer counterparts).  num_vertices consecutive values in host-layout
 * linear order (x fastest, rows of mx incl. halos) move from position src of
 * the source mesh to position dst of the target, into or out of the in-buffer;
 * a range that does not fit either mesh is AC_FAILURE, a NULL host field
 * AC_NOT_ALLOCATED.  Store calls return with the host range written.
 * Transfers run on the source device's stream (a peer copy between GPUs) and
 * need both devices in the same precision; the non-offset forms move whole
 * fields between devices of equal dims. */
AcResult acDeviceLoadVertexBufferWithOffset(const Device device, const Stream stream,
                                            const AcMesh host_mesh,
                                            const VertexBufferHandle vtxbuf_handle,
                                            const int3 src, const int3 dst,
                                            const int num_vertices);
AcResult acDeviceLoadMeshWithOffset(const Device device, const Stream stream,
                                    const AcMesh host_mesh, const int3 src, const int3 dst,
                                    const int num_vertices);
AcResult acDeviceStoreVertexBufferWithOffset(const Device device, const Stream stream,
                                             const VertexBufferHandle vtxbuf_handle,
                                             const int3 src, const int3 dst,
                                             const int num_vertices, AcMesh* host_mesh);
AcResult acDeviceStoreMeshWithOffset(const Device device, const Stream stream, const int3 src,
                                     const int3 dst, const int num_vertices, AcMesh* host_mesh);
AcResult acDeviceTransferVertexBufferWithOffset(const Device src_device, const Stream stream,
                                                const VertexBufferHandle vtxbuf_handle,
                                                const int3 src, const int3 dst,
                                                const int num_vertices, Device dst_device);
AcResult acDeviceTransferMeshWithOffset(const Device src_device, const Stream stream,
                                        const int3 src, const int3 dst, const int num_vertices,
                                        Device dst_device);
AcResult acDeviceTransferVertexBuffer(const Device src_device, const Stream stream,
                                      const VertexBufferHandle vtxbuf_handle, Device dst_device);
AcResult acDeviceTransferMesh(const Device src_device, const Stream stream, Device dst_device);

/* Pipelined whole-mesh loads (no counterpart in the reference, whose
 * acDeviceLoadMesh, include/astaroth_device.h:80, writes the in-buffer
 * directly).  acDeviceLoadMeshStaged copies a host mesh into a device-side
 * stage on `stream` and returns at once (the host buffers must stay valid
 * until the copy is done, and be page-locked for it to be asynchronous);
 * acDeviceCommitStagedMesh makes `stream` wait for that copy and moves the
 * stage into the in-buffer.  Staging the next input on one stream while the
 * device integrates on another overlaps the host transfer with the compute;
 * a staged load waits for the previous commit to have read the stage (two
 * staged loads with no commit between them must use the same stream). */
AcResult acDeviceLoadMeshStaged(const Device device, const Stream stream, const AcMesh host_mesh);
AcResult acDeviceCommitStagedMesh(const Device device, const Stream stream);

/* include/astaroth_device.h:217,246 -- acDeviceLoadMeshInfo and
 * acDeviceGetConfig under their other names. */
AcResult acDeviceUpdate(Device device, const AcMeshInfo info);
AcMeshInfo acDeviceGetLocalConfig(const Device device);

/* include/astaroth_device.h:235 (acc-runtime/api/common_kernels.cc:143-155):
 * copies the box min(in_volume, out_volume) of FP64 device arrays laid out x
 * fastest with their volume's dims, from in at in_offset to out at out_offset,
 * on the device's stream.  A box reaching past either array is AC_FAILURE. */
AcResult acDeviceVolumeCopy(const Device device, const Stream stream, const AcReal* in,
                            const Volume in_offset, const Volume in_volume, AcReal* out,
                            const Volume out_offset, const Volume out_volume);

/* include/astaroth_device.h:133 -- one RK3 substep (step_number 0..2) over
 * [start, end): the whole interior [nmin, nmin + nlocal), or a box of whole
 * interior x-y planes (start.xy = nmin.xy, end.xy = nmin.xy + nlocal.xy,
 * nmin.z <= start.z < end.z <= nmin.z + nlocal.z); other boxes are AC_FAILURE.
 * A substep solved as z boxes (the interior planes while the z halos travel,
 * then the planes at each end, as the reference's task graph splits it,
 * src/core/task.cc:1933-1993) gives the bits of the whole-interior call; its
 * boxes cover the interior once, in any order, each after the halo fill of
 * the planes it reads.  In substep 2 the first box called clears the CFL
 * maxima that the others add to, so boxes on other streams must be ordered
 * after it.  Reads `in` (stencils) and `out` (previous
 * substep state), writes `out`; the caller swaps the buffers afterwards, as
 * with the reference. */
AcResult acDeviceIntegrateSubstep(const Device device, const Stream stream,
                                  const int step_number, const Volume start, const Volume end,
                                  const AcReal dt);
/* include/astaroth_device.h:135,139 -- periodic halo fill of the in buffer
 * over [start, end) (interior cells are not written). */
AcResult acDevicePeriodicBoundcondStep(const Device device, const Stream stream,
                                       const VertexBufferHandle vtxbuf_handle,
                                       const Volume start, const Volume end);
AcResult acDevicePeriodicBoundconds(const Device device, const Stream stream,
                                    const Volume start, const Volume end);

/* include/astaroth_device.h:149-175 -- synchronous reductions over the
 * interior of the in buffer; the result is written to *result on the host. */
AcResult acDeviceReduceScalNoPostProcessing(const Device device, const Stream stream,
                                            const AcReduction reduction,
                                            const VertexBufferHandle vtxbuf_handle,
                                            AcReal* result);
AcResult acDeviceReduceScal(const Device device, const Stream stream,
                            const AcReduction reduction, const VertexBufferHandle vtxbuf_handle,
                            AcReal* result);
AcResult acDeviceReduceVecNoPostProcessing(const Device device, const Stream stream,
                                           const AcReduction reduction,
                                           const VertexBufferHandle vtxbuf0,
                                           const VertexBufferHandle vtxbuf1,
                                           const VertexBufferHandle vtxbuf2, AcReal* result);
AcResult acDeviceReduceVec(const Device device, const Stream stream,
                           const AcReduction reduction, const VertexBufferHandle vtxbuf0,
                           const VertexBufferHandle vtxbuf1, const VertexBufferHandle vtxbuf2,
                           AcReal* result);
AcResult acDeviceReduceVecScalNoPostProcessing(const Device device, const Stream stream,
                                               const AcReduction reduction,
                                               const VertexBufferHandle vtxbuf0,
                                               const VertexBufferHandle vtxbuf1,
                                               const VertexBufferHandle vtxbuf2,
                                               const VertexBufferHandle vtxbuf3,
                                               AcReal* result);
AcResult acDeviceReduceVecScal(const Device device, const Stream stream,
                               const AcReduction reduction, const VertexBufferHandle vtxbuf0,
                               const VertexBufferHandle vtxbuf1,
                               const VertexBufferHandle vtxbuf2,
                               const VertexBufferHandle vtxbuf3, AcReal* result);

/* No reference counterpart (the reference checks NaN and infinity on the host,
 * src/utils/modelsolver.cc:966-988, and aborts on CUDA errors): after any
 * acDeviceReduce* call, *nonfinite is 1 if one of the values that call reduced
 * (after its map) was NaN or infinite, else 0.  A maximum or minimum drops NaN,
 * so its result alone does not show one; the flag is formed in the same pass
 * over the fields. */
AcResult acDeviceGetReduceNonFinite(const Device device, int* nonfinite);

/* include/astaroth_device.h:248 -- raw device pointers of one field (FP64
 * devices only; the layout is the host layout, x fastest, halos included). */
AcResult acDeviceGetVertexBufferPtrs(Device device, const VertexBufferHandle vtxbuf,
                                     AcReal** in, AcReal** out);
/* include/astaroth_device.h:249 */
AcResult acDeviceMemGetInfo(const Device device, size_t* free_mem, size_t* total_mem);

/* ---------------------------------------------------------------------------
 * Additions beside the drop-in (no counterpart signature in the reference)
 * ------------------------------------------------------------------------- */

/* One full RK3 step: for s in 0..2 { periodic boundconds; substep s; swap }.
 * The sequence is captured once per (device, stream) into a CUDA graph and
 * replayed.  Equivalent to the reference's loop in samples/devicetest/main.cc:94-100. */
AcResult acDeviceIntegrateStep(const Device device, const Stream stream, const AcReal dt);

/* Computes the CFL maxima below from the current in-buffer (halos filled), for
 * the first step of an adaptive run; the reference launches calc_timestep as
 * its own kernel for this (samples/standalone_mpi/main.cc:396-441 calling the
 * AC_calc_timestep task graph).  Asynchronous on `stream`. */
AcResult acDeviceCalcTimestep(const Device device, const Stream stream);

/* The maxima the last substep 2 (or acDeviceCalcTimestep) computed: max |u| and max
 * Alfven speed |curl A| / sqrt(exp(lnrho)).  Replaces acDeviceGetOutput(UU_MAX_ADVEC)
 * and acDeviceGetOutput(ALFVEN_SPEED_MAX) of the reference
 * (include/astaroth_device.h device_get_output_decls.h; computed by calc_timestep,
 * acc-runtime/samples/mhd_modular/mhdsolver.ac:551-583,611).  Waits for the device. */
AcResult acDeviceGetTimestepMaxima(const Device device, AcReal* uu_max, AcReal* alfven_max);

/* CFL timestep from those maxima: samples/standalone_mpi/main.cc:396-441
 * (AC_additive_timestep = 0) or the additive form of mhdsolver.ac:558-569 (= 1). */
AcResult acDeviceGetTimestep(const Device device, AcReal* dt);

/* The output interface of the reference for these reductions
 * (include/astaroth_device.h:203,209 acDeviceFinishReduceReal[Stream];
 * device_get_output_decls.h acDeviceGetOutput / acDeviceSetOutput, as
 * src/core/grid.cc:3004-3024 uses them around its MPI allreduce).
 *
 * acDeviceFinishReduceReal waits for `stream` and returns in *result the
 * output that the last launch of `kernel` (AC_KERNEL_SOLVE at substep 2, or
 * AC_KERNEL_CALC_TIMESTEP) reduced on the device; `reduce_op` must be the
 * output's own (AC_REDUCE_OP_MAX for UU_MAX_ADVEC and ALFVEN_SPEED_MAX,
 * AC_REDUCE_OP_MIN for AC_dt_min), else AC_FAILURE.  The Stream variant takes
 * a CUDA stream handle instead of one of the device's streams.
 *
 * acDeviceGetOutput returns the output (waiting for the device), or the value
 * that acDeviceSetOutput stored since the last launch reducing it; NaN for an
 * invalid device or param.  acDeviceSetOutput stores a value, typically the
 * result of combining all ranks' outputs, that acDeviceGetOutput and
 * acDeviceGetTimestep use until the next substep 2 or acDeviceCalcTimestep. */
AcResult acDeviceFinishReduceReal(Device device, const Stream stream, AcReal* result,
                                  const AcKernel kernel, const AcReduceOp reduce_op,
                                  const AcRealOutputParam output);
AcResult acDeviceFinishReduceRealStream(Device device, struct CUstream_st* stream,
                                        AcReal* result, const AcKernel kernel,
                                        const AcReduceOp reduce_op,
                                        const AcRealOutputParam output);
AcReal acDeviceGetOutput(const Device device, const AcRealOutputParam param);
AcResult acDeviceSetOutput(const Device device, const AcRealOutputParam param,
                           const AcReal value);

/* Device-to-device transfers of the in-buffer from/to caller-owned FP64
 * arrays (8 device pointers, host layout with halos); FP32-compensated devices
 * split/join on the fly.  No counterpart signature in the reference (its
 * acDeviceLoadMesh/StoreMesh, include/astaroth_device.h:80,115, take host meshes). */
AcResult acDeviceLoadMeshDevice(const Device device, const Stream stream,
                                const AcReal* const* src);
AcResult acDeviceStoreMeshDevice(const Device device, const Stream stream, AcReal* const* dst);

/* Discrete adjoint (no counterpart in the reference; the entry point named by
 * the design of this library).  FP64 devices only.
 *
 * acDeviceLoadAdjoint sets the adjoint of the state, lf, from 8 device arrays
 * (NULL: zero), and zeroes the adjoint of the RK3 register w and the parameter
 * adjoints.  acDeviceIntegrateSubstepAdjoint(step_number = s) then maps the
 * adjoints (lf, lw) of (f_{s+1}, w_s) to those of (f_s, w_{s-1}) for the 2N RK3
 * substep w_s = alpha_s w_{s-1} + dt R(f_s), f_{s+1} = f_s + beta_s w_s
 * (acc-runtime/stdlib/integrators.h:11-29), reading f_s from the in-buffer
 * (halos must be filled, i.e. acDevicePeriodicBoundconds first) and adding
 * d(dt lw . R)/d(nu, eta) to the parameter adjoints.  Run s = 2, 1, 0 per RK3
 * step, backwards in time; acDeviceStoreAdjoint returns lf (interior values;
 * halo entries are not updated), acDeviceGetParamAdjoints the parameter ones. */
AcResult acDeviceLoadAdjoint(const Device device, const Stream stream,
                             const AcReal* const* lam_f);
AcResult acDeviceIntegrateSubstepAdjoint(const Device device, const Stream stream,
                                         const int step_number, const Volume start,
                                         const Volume end, const AcReal dt);
AcResult acDeviceStoreAdjoint(const Device device, const Stream stream, AcReal* const* lam_f);
AcResult acDeviceGetParamAdjoints(const Device device, AcReal* nu_bar, AcReal* eta_bar);

/* Checkpointed reverse sweeps without a call per substep (no counterpart in the
 * reference).  acDeviceAdjointTapeForward integrates `steps` RK3 steps from the
 * in-buffers exactly as acDeviceIntegrateStep (halo fill, substep, swap, three
 * times per step) and keeps every substep's input state, halos filled, on a
 * device tape of 3 * steps states owned by the Device (grown on demand; FP64
 * only).  acDeviceAdjointTapeBackward then applies
 * acDeviceIntegrateSubstepAdjoint about the taped states: s = 2, 1, 0 of the
 * last taped step first, down to the first; the in- and out-buffers are not
 * read.  A checkpointed backward pass is, per segment from the last: load the
 * segment's checkpoint, TapeForward(k), TapeBackward(k). */
AcResult acDeviceAdjointTapeForward(const Device device, const Stream stream, const int steps,
                                    const AcReal dt);
AcResult acDeviceAdjointTapeBackward(const Device device, const Stream stream, const int steps,
                                     const AcReal dt);

/* The auxiliary field BFIELD (AC_lbfield): B = curl A of the input of the
 * last substep 2, into three host arrays of (nx+6)(ny+6)(nz+6) AcReal each
 * (host layout; halo entries 0).  Synchronous.  AC_FAILURE without AC_lbfield. */
AcResult acDeviceStoreBfield(const Device device, const Stream stream, AcReal* bx, AcReal* by,
                             AcReal* bz);

/* Whole-plane copies for a decomposition along z (no counterpart with this
 * signature in the reference; they take the place of its halo packing,
 * src/core/kernels/packing.cuh:59-470, for z slabs).  Pack copies the xy planes
 * [z0, z0 + nplanes) of every field's in-buffer (mesh plane index, 0 = first
 * ghost plane, halo rows and columns included) into `buffer`; unpack copies them
 * back.  `buffer` is device memory of nplanes * acDevicePlaneBytes(device)
 * bytes, laid out array by array (the 8 fields; FP32-compensated meshes then
 * the 8 compensation arrays).  Asynchronous on `stream`. */
size_t acDevicePlaneBytes(const Device device);
AcResult acDevicePackPlanes(const Device device, const Stream stream, const int z0,
                            const int nplanes, void* buffer);
AcResult acDeviceUnpackPlanes(const Device device, const Stream stream, const int z0,
                              const int nplanes, const void* buffer);

/* Box copies for a decomposition in x, y and z (the reference's
 * kernel_pack_data / kernel_unpack_data and acKernelPackData /
 * acKernelUnpackData, src/core/kernels/packing.cuh:59-90,133-160,491-520, with
 * the box given as start and dims).  Pack copies the box [start, start + dims)
 * (padded mesh indices, 0 = first ghost cell) of every field's in-buffer into
 * `buffer`; unpack copies it back.  `buffer` is device memory of
 * acDeviceBoxBytes(device, dims) bytes, laid out array by array (the 8 fields;
 * FP32-compensated meshes then the 8 compensation arrays), then z, y, x (x
 * fastest).  A box that leaves the padded mesh is AC_FAILURE; acDeviceBoxBytes
 * is 0 for an empty box.  Asynchronous on `stream`. */
size_t acDeviceBoxBytes(const Device device, const int3 dims);
AcResult acDevicePackBox(const Device device, const Stream stream, const int3 start,
                         const int3 dims, void* buffer);
AcResult acDeviceUnpackBox(const Device device, const Stream stream, const int3 start,
                           const int3 dims, const void* buffer);

/* Snapshots of the computational domain (the single-process case of
 * acGridWriteMeshToDiskLaunch / acGridReadVarfileToMesh, src/core/grid.cc:3792-3935):
 * one raw file of nx*ny*nz AcReal values (x fastest) per field,
 * <dir>/<VTXBUF name>-<label>.mesh, or with segmented != 0
 * <dir>/<VTXBUF name>-segment-<ox>-<oy>-<oz>-<label>.mesh with (ox, oy, oz) =
 * AC_multigpu_offset, the distributed-I/O name.  Write creates `dir` (one
 * level) and reads the in-buffers; read loads the in-buffers, fills the halos
 * periodically and returns when done.  Both are synchronous. */
AcResult acDeviceWriteMeshToDisk(const Device device, const char* dir, const char* label,
                                 const int segmented);
AcResult acDeviceReadMeshFromDisk(const Device device, const char* dir, const char* label,
                                  const int segmented);

/* Raw CUDA stream handle behind `stream` (as void*), for callers that order
 * their own work (e.g. events) against the library's launches. */
void* acDeviceGetStreamHandle(const Device device, const Stream stream);

/* Number of kernel launches this device issued since creation (for audits). */
unsigned long long acDeviceGetLaunchCount(const Device device);

/* Library version string. */
const char* acB200Version(void);

/* The energy functional of the differentiable integration and its gradient;
 * no counterpart in the reference (whose reductions are RMS and exp^2 maps).
 *   J = sum over the interior of ((1/2) exp(lnrho) |u|^2 + |curl A|^2 / (2 mu0)) dV
 * with the solver's 6th-order first derivatives on the periodic interior
 * (wrapped indices: the halos of `fields` are not read).
 * fields:  8 device arrays in the host layout (mx*my*mz doubles, halos included)
 *          of the mesh described by info (AC_nlocal, AC_ds, AC_mu0).
 * J:       device pointer to one double (deterministic double-double sum).
 * grad:    NULL, or 8 device arrays (same layout) receiving dJ/dfields on the
 *          interior; their halo cells are not written.
 * scratch: device memory of acEnergyFunctionalScratchBytes(info) bytes.
 * stream:  a cudaStream_t (NULL for the default stream); asynchronous on it. */
AcResult acEnergyFunctional(const AcMeshInfo info, const AcReal* const* fields, AcReal* J,
                            AcReal* const* grad, AcReal* scratch, void* stream);
size_t acEnergyFunctionalScratchBytes(const AcMeshInfo info);

/* Test switch of the failure path of the tiled solve kernels (no counterpart in
 * the reference, whose errors abort): while enabled (nonzero), every block of a
 * tiled substep skips the shared-memory load of the last plane of its z chunk,
 * gives up waiting for it after a short bound, waits (bounded) until the loads
 * it did issue have landed, and completes.  The substep's results are invalid
 * and the next acDeviceSynchronizeStream reports AC_FAILURE (once); the device
 * stays usable.  Off (0) at acDeviceCreate; for tests only. */
AcResult acDeviceDebugSkipPlaneLoad(Device device, int enable);

/* Maximum number of thread blocks acReduceNoAlloc accepts: its scratch is a
 * fixed-size array inside the library (2 doubles per block, 33 KB per GPU). */
#define AC_REDUCE_NOALLOC_MAX_BLOCKS 2048

/* Reduction of caller-owned device fields that allocates no memory.  This
 * entry point has no counterpart in the reference.
 *
 * For callers that cannot allocate device memory: applications whose memory is
 * owned by their own pool or arena (a cudaMalloc outside it can fail once the
 * pool holds the memory, and cudaFree synchronizes the device), or coupled codes
 * held to a fixed memory budget.  No Device handle is needed.
 *
 * fields:  nfields device pointers (1 = scalar, 3 = vector, 4 = vector + scalar)
 *          to FP64 arrays in the host layout with 3-cell halos, (nx+6)(ny+6)(nz+6)
 *          values, x fastest; the interior is reduced.
 * reduction: one of the RTYPE_* records; its map must fit nfields.
 * result:  device pointer to one AcReal, written with the value before
 *          post-processing (as acDeviceReduce*NoPostProcessing; for RTYPE_RMS*
 *          apply sqrt(value / (nx*ny*nz)) yourself).
 * blocks:  0 for the default grid, else the grid size, at most
 *          AC_REDUCE_NOALLOC_MAX_BLOCKS (larger or negative requests return
 *          AC_FAILURE).
 * stream:  a cudaStream_t (NULL for the default stream); the call is
 *          asynchronous on it.
 *
 * The block partials and the completion counter live in one static device
 * array per GPU, shared by every call on that GPU and keeping the last call's
 * contents; the counter is cleared at the start of each call.  Calls that
 * overlap on the GPU race on the array and must be ordered by the caller.
 * The first call on a device looks up the array's device address for that
 * device (cudaGetSymbolAddress) and keeps it for the life of the process, so
 * make that first call before any stream capture.  A cudaDeviceReset (or any
 * destruction of the device's primary context) reloads the library's device
 * code, which can move the array: do not call this entry point on a device
 * after resetting it. */
AcResult acReduceNoAlloc(const AcReal* const* fields, const int nfields, const int nx,
                         const int ny, const int nz, const AcReduction reduction,
                         AcReal* result, const int blocks, void* stream);

/* ---- Ensembles of independent meshes -------------------------------------
 *
 * These entry points have no counterpart in the reference (its device layer
 * integrates one mesh per Device; an ensemble there is a loop of Devices or
 * of acDeviceIntegrateSubstep calls, src/core/device.cc:941-997).
 *
 * An Ensemble holds n members of possibly different sizes and physics
 * parameters on one GPU, all of one precision (AC_precision of the first
 * config).  Every member has an in-buffer and an out-buffer as a Device; one
 * step advances all members by one RK3 step with 3 x [one periodic halo fill
 * launch over all members + one persistent solve launch over a tile work-list
 * of all members], captured once as a CUDA graph.  Each member's cells follow
 * the same arithmetic as a Device of that member without tiling
 * (AC_debug_plain_kernel = 1), so the results agree bit for bit.  Members
 * with AC_upwind or AC_lforcing are refused. */
typedef struct ensemble_s* Ensemble;

/* How a step runs.  mode 0: the persistent solve over the work list: tx * ty
 * threads per block (one cell per thread and plane), zb planes per work item,
 * blocks_per_sm resident blocks per SM (0 = the occupancy limit), or, with
 * blocks_per_sm = AC_ENSEMBLE_MEMBER_LAUNCHES, one launch per member and substep
 * of the tap kernel, which has the same bits, as concurrent branches of the
 * step graph.  mode 1: one launch per member and substep of the kernel a
 * single-mesh Device of that member uses (the split-stage kernel, or the tap or
 * plain one for meshes it does not fit), as such branches (tx, ty, zb,
 * blocks_per_sm unused).  Each member gets the bits of a single-mesh Device of
 * that member (mode 0: of its plain kernel; mode 1: of its default kernel). */
#define AC_ENSEMBLE_MEMBER_LAUNCHES 1048576
typedef struct {
    int tx, ty, zb, blocks_per_sm;
    int mode;
} AcEnsembleTiles;

/* member_infos: n member configurations (AC_nlocal, AC_ds, physics parameters, AC_precision).
 * The dt of every member starts at 0; set it with acEnsembleSetTimesteps. */
AcResult acEnsembleCreate(const int device_id, const int n, const AcMeshInfo* member_infos,
                          Ensemble* ensemble);
AcResult acEnsembleDestroy(Ensemble* ensemble);
/* Host mesh <-> the member's in-buffer (whole mesh with halos, FP64 host
 * layout).  Synchronous. */
AcResult acEnsembleLoadMember(const Ensemble ensemble, const int member, const AcMesh host_mesh);
AcResult acEnsembleStoreMember(const Ensemble ensemble, const int member, AcMesh* host_mesh);
/* n timesteps, one per member, kept in device memory (read by every later step). */
AcResult acEnsembleSetTimesteps(const Ensemble ensemble, const AcReal* dts);
/* One RK3 step of every member through the captured graph (asynchronous). */
AcResult acEnsembleIntegrateStep(const Ensemble ensemble);
/* The same step as one halo-fill launch and one plain solve launch per member
 * and substep, issued one member after another (the comparison path). */
AcResult acEnsembleIntegrateStepSequential(const Ensemble ensemble);
AcResult acEnsembleSetTiles(const Ensemble ensemble, const AcEnsembleTiles tiles);
AcResult acEnsembleGetTiles(const Ensemble ensemble, AcEnsembleTiles* tiles);
/* Times the solve of substep 0 (which leaves the in-buffers unchanged) for
 * the persistent launch over a fixed candidate set of tiles, then for the
 * launches per member of mode 0 and, where some member is larger than about
 * 96^3, of mode 1, keeps the fastest and returns it with its time per substep in
 * milliseconds.  (Ensembles of small members so keep the bits of their
 * sequential launches; mode 1 is faster and can be set where these are not
 * needed.) */
AcResult acEnsembleAutotune(const Ensemble ensemble, AcEnsembleTiles* best, double* best_ms);
/* Reduction of one member's in-buffer, as acDeviceReduceScal / acDeviceReduceVec. */
AcResult acEnsembleReduceScal(const Ensemble ensemble, const int member, const AcReduction reduction,
                              const VertexBufferHandle vtxbuf, AcReal* result);
AcResult acEnsembleReduceVec(const Ensemble ensemble, const int member, const AcReduction reduction,
                             const VertexBufferHandle a, const VertexBufferHandle b,
                             const VertexBufferHandle c, AcReal* result);
AcResult acEnsembleSynchronize(const Ensemble ensemble);
void* acEnsembleGetStreamHandle(const Ensemble ensemble);
unsigned long long acEnsembleGetLaunchCount(const Ensemble ensemble);
/* Interior cells of all members (the unit of the ensemble's cell-updates/s). */
long long acEnsembleCellCount(const Ensemble ensemble);

AC_END_C_DECLARATIONS
