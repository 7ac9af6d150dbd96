// Several explicit steps per launch: the host's plan of tiles with halos (block.cu).
#pragma once
#include <vector>

#include "nrt_internal.h"

namespace nrt {

// A tile: `cnt` consecutive elements from `s` that its CTA owns, and `nh` halo elements, the
// ones within `depth` steps of dependence.  Local indices: the owned elements, then the halo
// (nearest first).
struct __align__(16) BlockTile {
  int32_t s, cnt, nh, h0;  // h0: its first entry of BlockView::halo
  int32_t nx, x0;          // its entries of BlockView::spec
  int32_t p0, p1;          // its probes: entries [p0, p1) of BlockView::probe
};

struct BlockView {
  const BlockTile *tile;
  const int4 *halo;      // {global element, mother | DR << 16, DL | distance << 16, 0}, local indices
  const ushort4 *spec;   // owned elements whose neighbours are not l - 1 and l + 1: {l, mother, DR, DL}
  const int2 *probe;     // {local element, slot of the recording}, per tile; or null
  const int32_t *scls;   // strain class + 1 per element (0: unstrained), or null
  int ntiles;
  int depth;             // steps per launch at most
  int cap;               // local elements at most
  int rows;              // strain: the classes' rows of a launch are staged in shared memory
  int max_probes;        // probes of a tile at most
  int lanes;             // FP64: threads per local element
};

// The plan on the host.
struct BlockPlan {
  std::vector<BlockTile> tile;
  std::vector<int4> halo;
  std::vector<ushort4> spec;
  int depth = 0, cap = 0;
  int lanes = 1;
};

// The plan expected to be fastest; false when one launch per step is.
bool choose_block_plan(const HostPack &host, const PackView &pv, bool mixed, BlockPlan &plan);

// Whether `steps` steps save more than making a plan takes.
bool block_plan_pays(const HostPack &host, const PackView &pv, bool mixed, int64_t steps);

struct StrainView;
// nk (<= depth) steps from loop index base + k0: V and its FP32 shadow from Vin to Vout / Fout,
// gates from gin to gout.  r.nprobe > 0: the tiles' probes record after every step.  s.n > 0:
// strained elements take row k0 + k of the chunk table at step k (mixed
// precision only).  Gates are FP32 or FP64 with the precision.
int launch_explicit_block(const PackView &pv, const BlockView &bv, int precision, int k0, int nk,
                          const double *Vin, double *Vout, float *Fout, const void *gin, void *gout,
                          const RecView &r, const StrainView &s, cudaStream_t st);
}  // namespace nrt
