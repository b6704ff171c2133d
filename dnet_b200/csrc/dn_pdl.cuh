// dn_pdl.cuh -- programmatic dependent launch: a kernel's blocks may start while the one in front still runs, and wait for it before they touch
// anything that it writes or reads; weights, which no kernel writes, may be asked for before.  (Launched without the attribute both are no-ops.)
#pragma once

namespace dn {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace dn
