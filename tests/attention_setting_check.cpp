// A backward whose context no longer takes the fused attention kernels that its forward took.  Prints, per length, the largest 2-norm of
// a gradient's difference from the one without the change, over the gradient's.
#include "gradc/gradc.hpp"

#include <cstdio>

using namespace gradc;

int main() {
    const Device gpu(DeviceType::CUDA, 0);
    gcb_ctx* c = Backend::get().ctx(gpu);
    for (int64_t T : {64, 300}) {
        Tensor<float> in[3];
        for (auto& t : in) {
            t = Tensor<float>::normal({2, 3, T, 32}, 0.0f, 1.0f, Device(DeviceType::CPU)).to(gpu);
            t.realize();
            t = t.detach();
            t.set_requires_grad(true);
            t.realize();
        }
        std::vector<float> grads[2][3];
        for (int change = 0; change < 2; ++change) {
            for (auto& t : in) t.zero_grad();
            Tensor<float> out = sdpa(in[0], in[1], in[2], true);
            out.realize();
            Tensor<float> act = out.gelu();
            act.realize();
            if (gcb_ctx_launch_count_named(c, "attention_") == 0) { std::printf("not fused\n"); return 1; }
            if (change) gcb_check(gcb_ctx_set_gemm_split_mode(c, 1), "setting");  // which the tensor-core pair does not compute in
            act.backward();
            gcb_check(gcb_ctx_set_gemm_split_mode(c, 2), "setting");
            for (int i = 0; i < 3; ++i) {
                Tensor<float> g = make_contiguous(in[i].grad().value());
                grads[change][i].resize((size_t)g.volume());
                gcb_check(gcb_copy_d2h(c, grads[change][i].data(), g.data_ptr(), sizeof(float) * grads[change][i].size()), "gradient");
            }
        }
        double worst = 0.0;
        for (int i = 0; i < 3; ++i) {
            double diff = 0.0, top = 0.0;
            for (size_t e = 0; e < grads[0][i].size(); ++e) {
                const double d = (double)grads[0][i][e] - grads[1][i][e], v = grads[0][i][e];
                diff += d * d;
                top += v * v;
            }
            worst = std::max(worst, std::sqrt(diff / top));
        }
        std::printf("%lld %.3e\n", (long long)T, worst);
    }
    return 0;
}
