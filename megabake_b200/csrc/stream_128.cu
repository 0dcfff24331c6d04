// The streaming decode kernel for heads of 128 dimensions.
#include "stream_kernel.cuh"

namespace mk {
const void* stream_kernel_128(int token_class) {
  const void* kernels[] = {reinterpret_cast<const void*>(&decode_stream<1, 128>), reinterpret_cast<const void*>(&decode_stream<8, 128, true>),
                           reinterpret_cast<const void*>(&decode_stream<8, 128>), reinterpret_cast<const void*>(&decode_stream<16, 128>),
                           reinterpret_cast<const void*>(&decode_stream<32, 128>)};
  return kernels[token_class];
}
}  // namespace mk
