// prt_sah.cuh - binned-SAH construction of the binary tree (prt_sah.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "prt_build.cuh"

namespace prt {

// What `gate` says (0: the trees are complete).
constexpr uint32_t kGateError = 1, kGateLevels = 2;

// Device scratch the SAH build of n triangles in S scenes needs (ws.sah).
size_t sah_scratch_bytes(uint32_t n, uint32_t S);

// Queues the build of the plan's scenes' binary trees, top-down with binned SAH, which writes
// what the collapse reads: ws.vals (position -> triangle), ws.lbox (by position), ws.left,
// ws.right, ws.rfirst, ws.rlast, ws.ibox (node ids up to n_int + S), ws.splits and ws.roots
// (scene s -> its root node).  d_toff: the device triangle offsets; scene_of: the scene of
// each triangle (several scenes) or null; x_faces (log 0: none) is cleared and filled.  Nothing is waited for: `gate` (device memory)
// becomes 0 when the trees are complete, kGateError when a check failed, kGateLevels when
// the trees need more levels than were queued (`level` of them; sah_build_more queues the
// rest).  The stages after it do nothing unless the gate is 0.
int sah_build_enqueue(const float *d_tris, const BuildPlan &plan, BuildScratch &ws,
                      const uint32_t *d_toff, const uint32_t *scene_of, XFaces x_faces,
                      cudaStream_t st, uint32_t *d_err, uint32_t *gate, int &level,
                      std::string &msg);

// The levels after `level` (synchronises `st` every few of them) and the rest of the trees.
int sah_build_more(const BuildPlan &plan, BuildScratch &ws, cudaStream_t st, uint32_t *d_err,
                   uint32_t *gate, int &level, std::string &msg);

} // namespace prt
