// Host program of test_gpu_cnn_wait_flag.py: what the network's entry points do after a wait of the
// tensor-core training kernels has run out.  The flag that such a kernel sets is set from here, for which
// this unit has the library's own source of the network object.
#include "../optimizec_b200/csrc/dns2d_api.cu"

#include <cstdio>

static int fails = 0;
#define CHECK(x)                                             \
    do {                                                     \
        if (!(x)) {                                          \
            std::printf("line %d: %s\n", __LINE__, #x);      \
            ++fails;                                         \
        }                                                    \
    } while (0)

static void run(int H, int W)
{
    const int B = 2, n = 4;
    const size_t px = (size_t)H * W;
    std::vector<float> x(n * 3 * px), t(n * px), y(B * px);
    for (size_t i = 0; i < x.size(); ++i) x[i] = (float)std::sin(0.37 * (double)i);
    for (size_t i = 0; i < t.size(); ++i) t[i] = (float)std::cos(0.11 * (double)i);
    dns2d_cnn *net = nullptr;
    CHECK(dns2d_cnn_create(&net, 3, 16, 1, 0) == DNS2D_OK);
    CHECK(dns2d_cnn_set_train_tc(net, 1) == DNS2D_OK);
    CHECK(dns2d_cnn_set_dataset(net, x.data(), t.data(), n, H, W) == DNS2D_OK);
    CHECK(dns2d_cnn_train(net, 3, B, 1e-3f, 1, nullptr) == DNS2D_OK);
    CHECK(net->step == 3);
    int *flag = W % 16 == 0 ? net->planes.err : net->gw.err;
    CHECK(flag != nullptr);
    const size_t np = (size_t)net->nparams;
    std::vector<float> p0(np), p1(np), g(np);
    double loss = 0.0, losses[2];
    const int one = 1;
    auto set = [&] { CHECK(cudaMemcpy(flag, &one, 4, cudaMemcpyHostToDevice) == cudaSuccess); };
    CHECK(dns2d_cnn_get_params(net, p0.data()) == DNS2D_OK);
    // each entry point reports the flag once
    set();
    CHECK(dns2d_cnn_forward(net, x.data(), B, H, W, y.data()) == DNS2D_ERR_TIMEOUT);
    CHECK(dns2d_cnn_forward(net, x.data(), B, H, W, y.data()) == DNS2D_OK);
    set();
    CHECK(dns2d_cnn_loss_grad(net, x.data(), t.data(), B, H, W, &loss, g.data()) == DNS2D_ERR_TIMEOUT);
    CHECK(dns2d_cnn_loss_grad(net, x.data(), t.data(), B, H, W, &loss, g.data()) == DNS2D_OK);
    // training leaves the parameters and the step count as they were
    for (double *l : {(double *)nullptr, losses}) {
        set();
        CHECK(dns2d_cnn_train(net, 2, B, 1e-3f, 2, l) == DNS2D_ERR_TIMEOUT);
        CHECK(dns2d_cnn_get_params(net, p1.data()) == DNS2D_OK);
        CHECK(p0 == p1);
        CHECK(net->step == 3);
    }
    CHECK(dns2d_cnn_train(net, 2, B, 1e-3f, 2, losses) == DNS2D_OK);
    CHECK(dns2d_cnn_get_params(net, p1.data()) == DNS2D_OK);
    CHECK(p0 != p1 && net->step == 5);
    dns2d_cnn_destroy(net);
}

int main()
{
    run(8, 16);   // chunk planes
    run(12, 20);  // im2col GEMMs
    std::printf(fails ? "%d checks failed\n" : "ok\n", fails);
    return fails != 0;
}
