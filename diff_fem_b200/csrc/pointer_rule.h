// pointer_rule.h — which of a caller's device buffers the kernels of a step
// use in place.
//
// Only memory of the scene's own GPU (the runtime's answer for the pointer,
// cudaPointerGetAttributes) is read and written by the kernels.  Anything else
// that a caller may pass as device memory (another GPU's tensor, managed or
// registered host memory, a pointer the runtime does not know) goes through a
// copy on the scene's stream, which serves it or refuses it with an error.
#pragma once

namespace dfem {

constexpr int kMemoryTypeDevice = 2;  // cudaMemoryTypeDevice
constexpr bool used_in_place(bool known, int type, int device, int scene_device) {
  return known && type == kMemoryTypeDevice && device == scene_device;
}

}  // namespace dfem
