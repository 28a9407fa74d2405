// gradc::linear_group on an input of one device and parameters of another, without a GPU: nothing is realized, the addresses are made up.
#include "gradc/gradc.hpp"

#include <cstdio>

using namespace gradc;

static float memory[1 << 16];

static Tensor<float> on(Device d, std::vector<int64_t> shape, int64_t at, std::shared_ptr<ParamArena> arena) {
    auto owner = std::shared_ptr<void>((void*)memory, [](void*) {});
    Tensor<float> t(shape, dense_strides(shape), 0, std::make_shared<Storage<float>>(memory + at, shape_volume(shape), d, owner), false);
    if (arena) {
        t._get_state()->m_slot = {arena, 0};
        t.set_requires_grad(true);
    }
    return t;
}

int main() {
    for (int other = 0; other < 2; ++other) {
        auto arena = std::make_shared<ParamArena>();
        const Device x_at(DeviceType::CUDA, 0), w_at(DeviceType::CUDA, other);
        Tensor<float> x = on(x_at, {5, 8}, 0, nullptr);
        const char* said = "taken";
        try {
            linear_group(x, {{on(w_at, {8, 12}, 1024, arena), on(w_at, {12}, 2048, arena)}, {on(w_at, {8, 12}, 1024 + 128, arena), on(w_at, {12}, 2048 + 128, arena)}});
        } catch (const std::exception& e) {
            said = "refused";
        }
        std::printf("%s\n", said);
    }
    return 0;
}
