// Choices of the decode attention, plain C++ so that they can be checked without a GPU.
#pragma once

#include "ring.h"

namespace b200q {

// What a warp of a cluster CTA appends of the new token: the last warp its V row, the one before it its K row, so that every byte has
// one writer.  With sixteen warps neither has a query row to rotate.
enum AppendRole { kAppendNothing, kAppendK, kAppendV };
B200Q_HD AppendRole append_role(int warp, int warps) { return warp == warps - 1 ? kAppendV : warp == warps - 2 ? kAppendK : kAppendNothing; }

}  // namespace b200q
