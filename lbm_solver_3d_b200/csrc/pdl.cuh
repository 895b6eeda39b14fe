// ============================================================================
//  pdl.cuh -- programmatic dependent launches: waiting for the predecessor, and
//  ordering what is read before that wait.
// ============================================================================
#pragma once

namespace lbmgpu {

// Programmatic dependent launch. A kernel launched with programmatic stream
// serialisation may start before its predecessor in the stream has finished;
// pdl_wait() blocks until that predecessor has completed and its writes are
// visible, so it comes before the first read of anything the predecessor
// writes. pdl_launch_dependents() lets the successor start early. Both are
// no-ops for an ordinary launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What a kernel that waits for its predecessor is shown, a kernel behind it that
// has not waited yet is not: pdl_wait makes earlier writes visible to the grid
// that calls it. A thread behind its own pdl_wait therefore publishes this
// step's tag (release), and a thread of the later kernel that reads that tag
// (acquire) sees all that was visible there. One that does not find it waits
// itself, so neither ever spins.
__device__ __forceinline__ void order_publish(int* word, int tag) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(word), "r"(tag) : "memory");
}
__device__ __forceinline__ void order_acquire(const int* word, int tag) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    if (v != tag) pdl_wait();
}

}  // namespace lbmgpu
