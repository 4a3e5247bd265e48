// Programmatic dependent launch.
#pragma once

namespace b200 {

// wait: block until every grid this one depends on has completed and its memory is visible.
// launch_dependents: allow the next kernel in the stream to start launching (it still waits
// at its own griddepcontrol.wait for our completion before touching dependent data).
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Dependency point of every non-GEMM kernel of the Llama path: wait for the producer, THEN let the consumer launch.  GEMMs
// release their consumer at entry (before their own wait).  Consequence used by the kernels' pre-wait prologues: code that
// runs before griddep_enter() in kernel K_n may read per-step inputs uploaded before the step's first kernel, static tables
// (weights, cos/sin, segment tables), and of what the step's kernels write only
//   * the output of K_{n-2} or earlier when K_{n-1} is a non-GEMM kernel (it was released after K_{n-2} had completed),
//   * with g GEMMs directly in front, the output of K_{n-g-2} or earlier: the last non-GEMM kernel in front of them is known
//     to have STARTED, not to have completed.
__device__ __forceinline__ void griddep_enter() {
  griddep_wait();
  griddep_launch();
}

// The designs' kernels release their consumer at entry and wait before anything else: the launches and prologues of a whole
// chain of small kernels then overlap, and a kernel that waits knows that everything before it in the stream is complete,
// because its predecessor waited too.  Ahead of the wait stand loads of weights, which no step writes, and of the step's uploaded inputs (positions,
// sequences, tables: copied before its first kernel), and prefetches into L2 of what may still be written (states: a prefetched line stays coherent);
// never a load of anything that a kernel of the step writes.  In a kernel launched this way nothing that an earlier kernel of the step wrote is read through the read-only path (__ldg; kernels launched plainly,
// such as the scans of prompt portions, may).  Decode steps, device time
// with plain launches and so: Soselix, 8 sequences, 35 kernels 338 us -> 300; Mulenex, 24 sequences 529 -> 480.

}  // namespace b200
