// Layers over one input taken together (gradc::linear_group) against the same layers one by one, for every subset of the outputs that
// a program may use.  Prints one line per subset: the outputs used, the parameters that received a gradient (bit per parameter) on
// either side, and the largest difference of a gradient over the largest gradient value.
#include "gradc/gradc.hpp"

#include <cstdio>

using namespace gradc;

struct Net : Module<float> {
    Linear<float> first, a, b, c;
    Net(const Initializer<float>& w, const Initializer<float>& z) : first(48, 160, w, z), a(160, 132, w, w), b(160, 132, w, w), c(160, 132, w, w) {
        register_module("first", &first);
        register_module("a", &a);
        register_module("b", &b);
        register_module("c", &c);
    }
    Tensor<float> forward(Tensor<float> in, int used, bool together) {
        Tensor<float> x = first.forward(in);
        std::vector<Tensor<float>> y = together ? linear_group(x, {{a.weight(), a.bias()}, {b.weight(), b.bias()}, {c.weight(), c.bias()}}) : std::vector<Tensor<float>>{a.forward(x), b.forward(x), c.forward(x)};
        Tensor<float> sum;
        for (int i = 0; i < 3; ++i)
            if (used >> i & 1) sum = sum._get_state() == nullptr ? y[(size_t)i].gelu() : sum + y[(size_t)i].gelu();
        return sum;
    }
};

int main() {
    const Device gpu(DeviceType::CUDA, 0);
    Net net(NormalInit<float>(0.0f, 0.1f), ZerosInit<float>());
    net.to(gpu);
    Tensor<float> in = Tensor<float>::normal({70, 48}, 0.0f, 1.0f, Device(DeviceType::CPU)).to(gpu);
    in.realize();
    std::vector<std::pair<std::string, Parameter<float>*>> params;
    net.ordered_parameters(params);
    for (int used = 1; used < 8; ++used) {
        std::vector<std::vector<float>> grads[2];
        int live[2] = {0, 0};
        for (int together = 0; together < 2; ++together)
            for (int pass = 0; pass < 2; ++pass) {  // the second one adds to the first
                if (pass == 0) net.zero_grad();
                Tensor<float> out = net.forward(in, used, together == 1);
                out.realize();
                out.backward();
                if (pass == 0) continue;
                for (size_t i = 0; i < params.size(); ++i) {
                    auto g = params[i].second->grad();
                    std::vector<float> h;
                    if (g.has_value()) {
                        live[together] |= 1 << i;
                        h.resize((size_t)g->volume());
                        gcb_check(gcb_copy_d2h(Backend::get().ctx(gpu), h.data(), g->data_ptr(), sizeof(float) * h.size()), "gradient");
                    }
                    grads[together].push_back(std::move(h));
                }
            }
        double worst = 0.0;
        for (size_t i = 0; i < params.size(); ++i) {
            double diff = 0.0, top = 0.0;
            for (size_t e = 0; e < std::min(grads[0][i].size(), grads[1][i].size()); ++e) {
                diff = std::max(diff, (double)std::abs(grads[0][i][e] - grads[1][i][e]));
                top = std::max(top, (double)std::abs(grads[0][i][e]));
            }
            if (top > 0.0) worst = std::max(worst, diff / top);
        }
        std::printf("%d %d %d %.3e\n", used, live[0], live[1], worst);
    }
    return 0;
}
