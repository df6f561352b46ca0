// Schedule of one scene's strain sweeps in shared memory (host side of
// k_strain_sweeps in cc_strain.cu).
#pragma once

#include <vector>

#include "cc_launch.h"

namespace ccg {

// The schedules of all scenes of a solver, one after the other.
struct SweepArrays {
    std::vector<SweepElem> elems;  // by scene, then level
    std::vector<int> lev;          // per scene: first element of each level, and the end
    std::vector<int4> epoch;       // per scene and epoch: copy-ins [x, y) and write-backs [z, w)
    std::vector<int> need;         // per scene and epoch: epochs the sweep before must have written back
    std::vector<int2> load, wb;    // (point, slot)
};

// Appends one scene's schedule. `elems` are the scene's strain elements in
// the reference's order with batch point ids (slots unset); points are
// [v0, v0 + nv). Fills the scene's sw_* fields and returns the points it
// touches.
//
// Level of an element = 1 + the level of the last earlier element at any of
// its points: the elements of a level share no point, and one thread takes
// an element's edges in their order, so level by level is the reference's
// sequential sweep. `sw_k` levels make an epoch. A point holds a slot from
// the step (epoch number) two before its first epoch, when its copy-in is
// issued, to the step after its last one, when it is written back.
int append_sweep_plan(const std::vector<SweepElem>& elems, int v0, int nv, SweepArrays& out, SceneDev& sd);

}  // namespace ccg
