// The instrumented form of the short-context build for narrow models (see decode_lean_small.cu and decode_prof.cu).
#define MI_PROF 1
#define MI_LEAN 1
#define MI_SMALL 1
#include "decode_kernel.cuh"

namespace mi {

const void* decode_kernel_prof_lean_small(int HD, int G) {
    #define MI_PICK(hd, g) if (HD == hd && G == g) return (const void*)decode_kernel<hd, g>;
    MI_PICK(64, 7) MI_PICK(64, 2)      // head shapes that occur with the embedding widths this build takes
    #undef MI_PICK
    return nullptr;
}

}  // namespace mi
