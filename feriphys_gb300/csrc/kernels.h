// Host-visible launch wrappers of the device kernels (no CUDA types beyond
// cudaStream_t/cudaError_t in the signatures).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "step_consts.h"

namespace fgb {

// CSR incidence lists of the general gather (see step_general.cu).
struct GeneralTopo {
  const int* strut_off;
  const int2* strut_inc;
  const float4* strut_kcl;
  const int* face_off;
  const int* face_inc;
  const int4* face_vtx;
  // the compact form (mesh_build.h: CompactTopo): form 1 with 32-bit strut
  // words, 2 with 16-bit ones; form 0 reads the lists above instead
  int form = 0;
  const int* own_off = nullptr;
  const float* sk = nullptr;
  const float* sc = nullptr;
  const float* sl = nullptr;
  const uint32_t* strut_word = nullptr;
  const uint16_t* strut_word16 = nullptr;
  const uint16_t* face_word = nullptr;
  // FP64 scratch: 6 doubles a strut (spring, damper) and a face (force, three
  // corner weights); null: the step evaluates them vertex by vertex
  double* strut_term = nullptr;
  double* face_term = nullptr;
  const uint32_t* strut_ab = nullptr;  // with them: the struts' first points, then their second ones
  int n_struts = 0, n_faces = 0;
};

// Grid (Cloth::new topology) description for the stencil kernel (see
// step_grid.cu).  params holds the strut constants (grid_order.h: param_rec).
struct GridTopo {
  int rows, cols;
  const float* params;
  int variant;  // 0: shared-memory tiles, 1: one thread per vertex reading global memory
};

// Chained to the launch before it in the stream (chain_launch.cuh).
template <class T>
cudaError_t launch_step_general(int n, const void* pos, const void* vel, const void* force_in, void* pos_out,
                                void* vel_out, const GeneralTopo& t, const StepConsts& c, cudaStream_t s);
template <class T>
cudaError_t launch_accumulate(int n, const void* pos, const void* vel, void* force, const GeneralTopo& t,
                              const StepConsts& c, cudaStream_t s);
template <class T>
cudaError_t launch_integrate(int n, int integration, float h, const void* pos, const void* vel, const void* force,
                             void* spos, void* svel, void* sforce, cudaStream_t s);
template <class T>
cudaError_t launch_update(int n, void* pos, void* vel, void* force, const void* spos, const void* svel,
                          const void* sforce, const StepConsts& c, cudaStream_t s);
template <class T>
cudaError_t launch_zero4(int n, void* a, cudaStream_t s);

// chained: the launch may overlap the end of the one before it in the stream
// (chain_launch.cuh); false where that one writes what a step reads besides
// the state (cloth tables, work items).
cudaError_t launch_step_grid(const GridTopo& g, const float4* pos, const float4* vel, const float4* force_in,
                             float4* pos_out, float4* vel_out, const StepConsts& c, cudaStream_t s, bool chained);

// One cloth of a batch (Cloth::new topology); buffers [parity] are read and
// [parity ^ 1] written by a step.
struct ClothDesc {
  const float* params;  // strut constants (grid_order.h: param_rec)
  float4* pos[2];
  float4* vel[2];
  const float4* force_in;  // accumulated force carried into the step, or null
  unsigned* flags;         // non-finite flag of this cloth
  int rows, cols;
  float wind[3];
  int skip;  // nonzero: the batched step leaves this cloth untouched (masked fallback steps)
};

// Batch tiles are 32 wide and kDefaultTileH (or another height the
// autotuner picks, batch_tile_height_ok) tall.
constexpr int kDefaultTileH = 8;
constexpr int kBatchTileHeights[3] = {4, 8, 12};
bool batch_tile_height_ok(int th);

// Tiles of one cloth for the batch work list: {cloth, tile x, tile y, interior}.
void batch_tiles(int cloth, int rows, int cols, int th, int* out4 /* may be null */, int* n_ring, int* n_interior);

// The single-cloth tiled kernel's grid: the CTA count for an R x C cloth and
// 32 x th tiles, and (out3 non-null) each CTA's {tile x, tile y, interior}
// in blockIdx order, by the kernel's own mapping.
int grid_tiles(int rows, int cols, int th, int* out3 /* may be null */);

// One CTA per work item.  n_work_dev: null, or the item count in device memory
// (n_work is then its upper bound, which sizes the grid).
// th: the tile height the work list was made for.
cudaError_t launch_step_batched(const ClothDesc* cloths, const int4* work, int n_work, int parity,
                                const StepConsts& c, cudaStream_t s, bool chained, const int* n_work_dev = nullptr,
                                int th = kDefaultTileH);
// Sets the launch attributes of the tiled and batched step kernels (done by
// their launchers on first use; call it before a stream capture).
cudaError_t prime_step_kernels();
int batched_ctas_per_sm(int th = kDefaultTileH);

}  // namespace fgb
