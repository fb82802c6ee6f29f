// Host entries to the __host__ __device__ functions of the kernels' headers, so
// that tests without a GPU run the code that the kernels run.
#include "pic_adjoint.cuh"

extern "C" {
int dm_out_mixed_align() { return (int)alignof(pic::OutMixed); }
int dm_out_mixed_size() { return (int)sizeof(pic::OutMixed); }
int dm_max_slots() { return pic::kMaxSlots; }
int dm_max_slot(int it) { return pic::max_slot(it); }
int dm_max_cleared(int it) { return pic::max_cleared(it); }
int dm_no_quantum() { return pic::kNoQuantum; }
int dm_quantum_plain(int E, unsigned hi) {
    return pic::quantum_for(E, pic::exponent_hi(hi), pic::kKeepPlain, pic::kLeastPlain);
}
int dm_quantum_mixed(int E, unsigned bits) {
    return pic::quantum_for(E, pic::exponent_f(bits), pic::kKeepMix, pic::kLeastMix);
}
}
