// smallsys.cu -- dispatch of the one-launch path for small Fock spaces
// (smallsys.h) over the orbital count.
#include "smallsys.h"

namespace mctdhb {

template <int M>
int small_prepare_tmpl();
template <int M>
int small_waves_tmpl(int (&at)[kClusterSizes]);
template <int M>
int small_launch_tmpl(const SmallSys& s, int part, int i, cudaStream_t st);
template <int M>
int small_batch_tmpl(const BatchSlot* slots, const int* list, const int* nlist, int nslots,
                     int part, int blocks, cudaStream_t st);

bool small_eligible(int N, int M, uint32_t D2, double macs) {
    const double P = 0.5 * M * (M + 1);
    return N >= 2 && M >= 2 && M <= kMaxTemplOrb && (double)D2 * P * P <= macs;
}

#define MCTDHB_BY_M(call)                                                       \
    switch (M) {                                                                \
        case 2: return call(2);                                                 \
        case 3: return call(3);                                                 \
        case 4: return call(4);                                                 \
        case 5: return call(5);                                                 \
        case 6: return call(6);                                                 \
        case 7: return call(7);                                                 \
        case 8: return call(8);                                                 \
    }                                                                           \
    set_error("small-space path: %d orbitals outside 2..8", M);                 \
    return -1

int small_prepare(int M) {
#define CALL(m) small_prepare_tmpl<m>()
    MCTDHB_BY_M(CALL);
#undef CALL
}

int small_waves(int M, int (&at)[kClusterSizes]) {
#define CALL(m) small_waves_tmpl<m>(at)
    MCTDHB_BY_M(CALL);
#undef CALL
}

int small_launch(const SmallSys& s, int part, int i, cudaStream_t st) {
    const int M = s.sp.M;
#define CALL(m) small_launch_tmpl<m>(s, part, i, st)
    MCTDHB_BY_M(CALL);
#undef CALL
}

int small_batch_launch(int M, const BatchSlot* slots, const int* list, const int* nlist,
                       int nslots, int part, int blocks, cudaStream_t st) {
#define CALL(m) small_batch_tmpl<m>(slots, list, nlist, nslots, part, blocks, st)
    MCTDHB_BY_M(CALL);
#undef CALL
}

}  // namespace mctdhb
