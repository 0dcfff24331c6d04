// The streaming decode kernel for heads of 64 dimensions.
#include "stream_kernel.cuh"

namespace mk {
const void* stream_kernel_64(int token_class) {
  const void* kernels[] = {reinterpret_cast<const void*>(&decode_stream<1, 64>), reinterpret_cast<const void*>(&decode_stream<8, 64, true>),
                           reinterpret_cast<const void*>(&decode_stream<8, 64>), reinterpret_cast<const void*>(&decode_stream<16, 64>),
                           reinterpret_cast<const void*>(&decode_stream<32, 64>)};
  return kernels[token_class];
}
}  // namespace mk
