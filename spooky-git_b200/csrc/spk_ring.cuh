// spk_ring.cuh -- the order of the loads of a ring of stages (plain C++ too:
// the tests compile it for the host).
//
// Load j of a ring of nst stages, counted from 0 in the order of issue, goes
// to stage j % nst and completes that stage's phase j / nst, which a wait
// names by its parity.  A stage is loaded again only after its last load was
// waited for, so at most the last nst loads are in flight; each is the last
// one of its stage, and a wait for it returns at once where it has completed.
#pragma once

#ifdef __CUDACC__
#define SPK_RING_FN __host__ __device__ __forceinline__
#else
#define SPK_RING_FN inline
#endif

namespace spk {

SPK_RING_FN int ring_stage(int j, int nst) { return j % nst; }
SPK_RING_FN unsigned ring_parity(int j, int nst) { return (unsigned)(j / nst) & 1u; }
// the first load that can be in flight after `issued` loads
SPK_RING_FN int ring_first_pending(int issued, int nst) { return issued > nst ? issued - nst : 0; }

}  // namespace spk
