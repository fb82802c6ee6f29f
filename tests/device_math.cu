// Host entries to the __host__ __device__ functions of the kernels' headers, so
// that tests without a GPU run the code that the kernels run.
#include "pic_adjoint.cuh"

extern "C" {
int dm_max_slots() { return pic::kMaxSlots; }
int dm_max_slot(int it) { return pic::max_slot(it); }
int dm_max_cleared(int it) { return pic::max_cleared(it); }
}
