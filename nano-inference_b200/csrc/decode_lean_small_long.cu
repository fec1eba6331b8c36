// The long-context build (decode_lean_long.cu) of the decode kernel for models of 513 to 1024 embedding values.
#define MI_LEAN 2
#define MI_SMALL 1
#include "decode_kernel.cuh"

namespace mi {

const void* decode_kernel_lean_small_long(int HD, int G) {
    #define MI_PICK(hd, g) if (HD == hd && G == g) return (const void*)decode_kernel<hd, g>;
    MI_PICK(64, 7) MI_PICK(64, 2)      // head shapes that occur with the embedding widths this build takes
    #undef MI_PICK
    return nullptr;
}

}  // namespace mi
