// A stand-in for the CUDA runtime calls and kernel launches of the host
// sources (sgl_api.cpp, sgl_lane.cpp, sgl_scene.cpp, sgl_serve.cpp), so that
// their ordering and their use of page-locked staging are checked without a
// GPU.  Streams execute nothing until something waits for them.  What it
// records:
//  - unordered: work enqueued on a stream that the work enqueued just before
//    it on another stream does not precede (no event wait, no host wait);
//  - overwritten: page-locked memory that changed between an asynchronous copy
//    from it and that copy's execution;
//  - live / peak: device bytes allocated;
//  - device_calls: allocations, copies, fills and launches.
#pragma once
#include <cstddef>
#include <string>

namespace fake {
extern long unordered, overwritten, device_calls;
extern size_t live, peak;
extern bool auto_progress;  // cudaEventQuery completes what it asks about
extern std::string fail_on; // the named call or launch fails while set
extern long streams_destroyed_twice, foreign_streams_destroyed;
void drain_all();
} // namespace fake
