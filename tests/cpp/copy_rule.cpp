// The rule that sends a copy to a kernel or to the copy engine, over pointers of
// either GPU with either one current (no GPU needed: the attributes are made up).
#include <cstdio>

#include "../../symphas_b200/csrc/sp_handle.h"

int main() {
  const auto rule = [](cudaMemoryType type, int of, int current, int device, uintptr_t ptr) {
    cudaPointerAttributes at{};
    at.type = type;
    at.device = of;
    return copy_by_kernel(at, reinterpret_cast<const void*>(ptr), 8, current, device);
  };
  const cudaMemoryType types[] = {cudaMemoryTypeDevice, cudaMemoryTypeManaged, cudaMemoryTypeHost,
                                  cudaMemoryTypeUnregistered};
  for (cudaMemoryType type : types)
    for (int of = 0; of < 2; ++of)
      for (int current = 0; current < 2; ++current)
        for (int device = 0; device < 2; ++device)
          for (uintptr_t ptr : {uintptr_t(4096), uintptr_t(4104), uintptr_t(4100)}) {
            const bool want =
                type == cudaMemoryTypeDevice && of == device && current == device && ptr != 4100;
            if (rule(type, of, current, device, ptr) != want) {
              std::printf("type %d of %d current %d handle %d ptr %d\n", int(type), of, current,
                          device, int(ptr));
              return 1;
            }
          }
  std::printf("ok\n");
  return 0;
}
