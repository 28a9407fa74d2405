// Generation with a model that has not been moved to the inference device.
#include "gradc/gradc.hpp"

#include <cstdio>

using namespace gradc;

int main() {
    NormalInit<float> init(0.0f, 0.02f);
    GPT<float> model(96, 16, 32, 4, 1, init, init, 1e-5f);
    const Device gpu(DeviceType::CUDA, 0);
    for (int moved = 0; moved < 2; ++moved) {
        if (moved) model.to(gpu);
        try {
            std::printf("%zu\n", generate_tokens_incremental(model, {1, 2, 3}, 8, 12, 1, gpu).size());
        } catch (const std::exception& e) {
            std::printf("%s\n", e.what());
        }
    }
    return 0;
}
