// Host side of the uniform levels (kern_uni.cuh): which hierarchies have
// them, and the plan of a cluster's V-cycle over the coarse ones.
#pragma once
#include "hier.h"

namespace bsamg {

// Levels minlevel .. 0 are each one patch covering its parent, one ghost
// layer, every dimension periodic (even extents) or between physical faces;
// then SetGhost on them is the image copy of kern_uni.cuh.  The plugin's
// stencils reach face neighbours only.
bool uni_eligible(const Hier& H);
// the boundary conditions of those levels
UniBC uni_bc(const Hier& H);
// host table entries of the patch of level l <= 0
inline int uni_patch(const Hier& H, int level) { return H.L(level).patches[0]; }
// whether an operation on `level` takes the uniform form (schedules being
// recorded as tail or solve programs keep the general operations)
inline bool uni_level(const Hier& H, int level) { return H.uni && !H.rec && level <= 0; }
// The highest level <= `level` from which the V-cycle down to minlevel runs
// in one cluster launch, and its plan; null when it does not (disabled by
// tail_cells 0, or nothing fits).
const Hier::UniPlan* uni_plan(Hier& H, const PluginUni& U, int level, int minlevel, int nsmooth);
// FillDown of the fields (bit 0: q, bit 1: f) from `level` <= 0 to minlevel
int uni_enq_fill(Hier& H, const PluginUni& U, int fields, int level, int minlevel);

}  // namespace bsamg
