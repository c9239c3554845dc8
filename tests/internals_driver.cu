// States of a context that the C ABI cannot set, for test_internals_gpu.py: a driver that includes the library's
// internal headers and is linked with it. Prints "name value" lines.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "../include/nse2d.h"
#include "../nse2d-channel-gpu_b200/csrc/nse2d_internal.h"

using nse2d::Context;

#define OK(x)                                                                            \
    do {                                                                                 \
        if ((x) != 0) {                                                                  \
            std::fprintf(stderr, "%s: %s\n", #x, nse2d_last_error());                    \
            std::exit(1);                                                                \
        }                                                                                \
    } while (0)

static nse2d_ctx* channel(int Nx, int Ny, int precision) {
    nse2d_config c;
    nse2d_config_default(&c);
    c.Nx = Nx; c.Ny = Ny; c.stretch = 1; c.beta = 2.0; c.Reb = 2000.0; c.F0 = 0.05; c.nforce = 4; c.adapt = 1;
    c.precision = precision;
    nse2d_ctx* x = nullptr;
    OK(nse2d_create(&c, &x));
    return x;
}
static void start(nse2d_ctx* x) {
    const Context* c = x->c;
    std::vector<double> w((size_t)c->Nx * c->Ny), y(c->Ny);
    OK(nse2d_metrics(x, 0, y.data()));
    for (int j = 0; j < c->Ny; ++j)
        for (int i = 0; i < c->Nx; ++i) w[(size_t)j * c->Nx + i] = 3.0 * y[j] + 0.05 * std::sin(M_PI * (y[j] + 1.0)) * std::cos(2.0 * M_PI * i / c->Nx);
    OK(nse2d_set_omega(x, w.data(), 0, nullptr));
}
static long long steps_taken(nse2d_ctx* x) {
    long long n = 0;
    OK(nse2d_get_time(x, nullptr, nullptr, &n, nullptr, nullptr));
    return n;
}

// A wait that has timed out: the flag that the kernel would have left, then a run, steps, and a new state.
static void gave_up(int precision) {
    nse2d_ctx* x = channel(128, 65, precision);
    start(x);
    std::printf("one_launch %d\n", x->c->steps_R > 0);
    const int flag = 2;
    OK(cudaMemcpy(&x->c->ctl->nonfinite, &flag, sizeof(int), cudaMemcpyHostToDevice));
    int reason = -1;
    OK(nse2d_run(x, 1e300, 1e300, 0, 1e300, 5, &reason, nullptr));
    std::printf("reason %d\n", reason);
    OK(nse2d_step(x, 3, 1, nullptr));
    std::printf("steps_of_a_void_state %lld\n", steps_taken(x));
    start(x);
    OK(nse2d_run(x, 1e300, 1e300, 0, 1e300, 5, &reason, nullptr));
    std::printf("reason_of_a_new_state %d\nsteps_of_a_new_state %lld\n", reason, steps_taken(x));
    OK(nse2d_destroy(x));
}

// Two channels on two streams: the form of a step while the other one's steps are in flight, and alone.
static void shared(int precision) {
    cudaStream_t q[2];
    for (auto& s : q) OK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    nse2d_ctx *a = channel(1024, 513, precision), *b = channel(128, 129, precision), *c = channel(128, 129, precision);
    for (nse2d_ctx* x : {a, b, c}) start(x);
    std::printf("one_launch %d\n", a->c->steps_R > 0 && b->c->steps_R > 0);
    OK(nse2d_step(a, 2000, 1, q[0]));                        // 0.1 s
    OK(nse2d_step(b, 3, 1, q[1]));
    const bool busy = cudaStreamQuery(q[0]) == cudaErrorNotReady;
    std::printf("still_busy %d\nby_launches_beside_another %d\n", busy, b->c->graph_exec != nullptr);
    OK(cudaDeviceSynchronize());
    OK(nse2d_step(c, 3, 1, q[1]));
    std::printf("by_launches_alone %d\n", c->c->graph_exec != nullptr);
    OK(cudaDeviceSynchronize());
    // a was found in flight: its next call is by launches, and the one after that, with nobody beside it, is not
    for (int k = 0; k < 2; ++k) {
        if (a->c->graph_exec) { cudaGraphExecDestroy(a->c->graph_exec); a->c->graph_exec = nullptr; }
        OK(nse2d_step(a, 2, 1, q[0]));
        std::printf("first_channel_by_launches_%d %d\n", k, a->c->graph_exec != nullptr);
        OK(cudaDeviceSynchronize());
    }
    const size_t n = (size_t)128 * 129;
    std::vector<double> f[4];
    for (auto& v : f) v.resize(n);
    OK(nse2d_get_fields(b, f[0].data(), f[1].data(), 0, nullptr));
    OK(nse2d_get_fields(c, f[2].data(), f[3].data(), 0, nullptr));
    std::printf("same_bits %d\n", f[0] == f[2] && f[1] == f[3]);
    for (nse2d_ctx* x : {a, b, c}) OK(nse2d_destroy(x));
    for (auto& s : q) cudaStreamDestroy(s);
}

// Whether a grid's steps go in one launch: no graph was captured by a step that would replay one.
static void form(int Nx, int Ny, int precision) {
    nse2d_ctx* x = channel(Nx, Ny, precision);
    start(x);
    OK(nse2d_step(x, 2, 1, nullptr));
    OK(cudaDeviceSynchronize());
    std::printf("one_launch %d\nrows_a_cta %d\n", !x->c->graph_exec, x->c->steps_R);
    OK(nse2d_destroy(x));
}

// The tuner of the plans on a grid whose steps go in one launch: what it times is by launches, what follows is not.
static void autotune() {
    nse2d_ctx* x = channel(256, 129, 64);
    start(x);
    OK(nse2d_step(x, 2, 1, nullptr));
    std::printf("one_launch %d\n", x->c->steps_R > 0 && !x->c->cap_stream);
    nse2d_plan best;
    double ms = 0.0;
    OK(nse2d_autotune_plan(x, 2, &best, &ms, nullptr));
    std::printf("graphs_captured %d\n", x->c->cap_stream != nullptr);
    if (x->c->graph_exec) { cudaGraphExecDestroy(x->c->graph_exec); x->c->graph_exec = nullptr; }
    OK(nse2d_step(x, 2, 1, nullptr));
    std::printf("one_launch_after %d\n", !x->c->graph_exec);
    OK(nse2d_destroy(x));
}

// A wait of the model's kernels that has timed out: gradients and a training step, and the same once it is reported.
struct Model {
    static constexpr int Nx = 32, Ny = 17, H = 16;
    nse2d_cnn* n = nullptr;
    double* f = nullptr;                                     // five fields
    Model() {
        std::vector<double> y(Ny), h((size_t)5 * Nx * Ny);
        for (int j = 0; j < Ny; ++j) y[j] = -1.0 + 2.0 * j / (Ny - 1);
        for (size_t i = 0; i < h.size(); ++i) h[i] = std::sin(0.37 * (double)i);
        OK(nse2d_cnn_create(Nx, Ny, H, 1, y.data(), &n));
        for (int l = 0; l < 4; ++l) {
            int ci = 0, co = 0;
            OK(nse2d_cnn_layer_shape(n, l, &ci, &co));
            std::vector<float> w((size_t)co * 9 * ci), b(co, 0.1f);
            for (size_t i = 0; i < w.size(); ++i) w[i] = 0.1f * std::cos(0.71f * (float)i);
            OK(nse2d_cnn_set_params(n, l, w.data(), b.data()));
        }
        OK(cudaMalloc((void**)&f, h.size() * sizeof(double)));
        OK(cudaMemcpy(f, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
    ~Model() { nse2d_cnn_destroy(n); cudaFree(f); }
    const double* field(int k) const { return f + (size_t)k * Nx * Ny; }
    int gradients(float* loss) {
        const int idx = 0;
        return nse2d_cnn_gradients(n, field(0), field(1), field(2), field(3), field(4), &idx, 1, loss, nullptr);
    }
    int train() {
        const int idx = 0;
        return nse2d_cnn_train_step(n, field(0), field(1), field(2), field(3), field(4), &idx, 1, 1e-2f, 1e-4f, nullptr, nullptr);
    }
    void timed_out() {
        const int one = 1;
        OK(cudaMemcpy(nse2d::cnn_wait_flag(n->n), &one, sizeof(int), cudaMemcpyHostToDevice));
    }
    std::vector<float> weights() {
        std::vector<float> all;
        for (int l = 0; l < 4; ++l) {
            int ci = 0, co = 0;
            OK(nse2d_cnn_layer_shape(n, l, &ci, &co));
            std::vector<float> w((size_t)co * 9 * ci), b(co);
            OK(nse2d_cnn_get_params(n, l, w.data(), b.data()));
            all.insert(all.end(), w.begin(), w.end());
            all.insert(all.end(), b.begin(), b.end());
        }
        return all;
    }
};
static void model_wait() {
    Model a, b;
    float loss = 0.f, ref = 0.f;
    OK(b.gradients(&ref));
    a.timed_out();
    std::printf("gradients %d\n", a.gradients(&loss));
    std::printf("gradients_after %d\nloss_after_is_right %d\n", a.gradients(&loss), loss == ref);
    const std::vector<float> w0 = a.weights();
    a.timed_out();
    std::printf("train %d\n", a.train());
    std::printf("weights_kept %d\n", a.weights() == w0);
    std::printf("train_after %d\n", a.train());
    OK(b.train());
    std::printf("weights_after_are_the_first_steps %d\n", a.weights() == b.weights() && a.weights() != w0);
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "gave_up") gave_up(std::atoi(argv[2]));
    else if (what == "model_wait") model_wait();
    else if (what == "autotune") autotune();
    else if (what == "form") form(std::atoi(argv[2]), std::atoi(argv[3]), std::atoi(argv[4]));
    else if (what == "shared") shared(std::atoi(argv[2]));
    else return 2;
    return 0;
}
