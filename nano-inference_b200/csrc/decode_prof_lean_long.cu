// The instrumented form of the long-context build (see decode_lean_long.cu and decode_prof.cu).
#define MI_PROF 1
#define MI_LEAN 2
#include "decode_kernel.cuh"

namespace mi {

const void* decode_kernel_prof_lean_long(int HD, int G) {
    #define MI_PICK(hd, g) if (HD == hd && G == g) return (const void*)decode_kernel<hd, g>;
    MI_PICK(128, 6) MI_PICK(128, 8) MI_PICK(64, 2)      // head shapes of models whose embedding width this build takes (1024 < E <= 2048)
    #undef MI_PICK
    return nullptr;
}

}  // namespace mi
