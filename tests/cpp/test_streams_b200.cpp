// The fp32 flash operator, forward and backward, from two threads with a stream each: a call's temporaries go back to the pool while its kernels
// are queued, so the other thread must not get them.  Every result has to have the bits of a call that ran alone.
#include <vesper/ops/flash_attention.h>

#include <atomic>
#include <cstdio>
#include <random>
#include <string>
#include <thread>
#include <vector>

using namespace vesper;

namespace {
constexpr int64_t B = 1, H = 8, D = 64;

struct Work {
    Tensor q, k, v, g;
    std::vector<std::vector<float>> alone;      // o, dq, dk, dv
};

Tensor random_tensor(int64_t N, unsigned seed) {
    std::mt19937 gen(seed);
    std::normal_distribution<float> d(0.f, 1.f);
    std::vector<float> h(static_cast<size_t>(B * H * N * D));
    for (auto& x : h) x = d(gen);
    Tensor t = empty({B, H, N, D}, DType::Float32, Device::CUDA);
    t.copy_from_host(h.data());
    return t;
}

// `calls` forward and backward passes queued one behind the other; the last one's results
std::vector<std::vector<float>> passes(const Work& w, int calls) {
    std::vector<Tensor> last;
    for (int i = 0; i < calls; ++i) {
        auto [o, lse] = ops::flash_attention_with_lse(w.q, w.k, w.v, 0.125f, true);
        auto [dq, dk, dv] = ops::flash_attention_backward(w.g, w.q, w.k, w.v, o, lse, 0.125f, true);
        last = {ops::flash_attention(w.q, w.k, w.v, 0.125f, true), dq, dk, dv};
    }
    std::vector<std::vector<float>> out;
    for (const Tensor& t : last) {
        out.emplace_back(t.numel());
        t.copy_to_host(out.back().data());
    }
    return out;
}
}  // namespace

int main(int argc, char** argv) {
    const int rounds = argc > 1 ? std::stoi(argv[1]) : 50;
    std::vector<Work> work(2);
    for (int i = 0; i < 2; ++i) {
        const int64_t N = 500;                  // one size: the two ask for the same blocks
        work[i].q = random_tensor(N, 10 * i + 1);
        work[i].k = random_tensor(N, 10 * i + 2);
        work[i].v = random_tensor(N, 10 * i + 3);
        work[i].g = random_tensor(N, 10 * i + 4);
        work[i].alone = passes(work[i], 1);
    }
    std::atomic<int> wrong{0};
    std::vector<std::thread> threads;
    for (int i = 0; i < 2; ++i)
        threads.emplace_back([&, i] {
            Stream s(Device::CUDA);
            Stream::set_current(s);
            for (int r = 0; r < rounds; ++r)
                if (passes(work[i], 1 + r % 4) != work[i].alone) ++wrong;
            s.synchronize();
        });
    for (auto& t : threads) t.join();
    std::printf("%d of %d results differ from a call alone\n", wrong.load(), 2 * rounds);
    return wrong == 0 ? 0 : 1;
}
