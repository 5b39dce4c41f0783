// Host logic of the corrector's entry points on a fake runtime (fake_cudart.h).
// Usage: corrector_host_check <scenario>; exit status 0 = as expected.
#include <cstdio>
#include <cstring>
#include <thread>

#include "fake_cudart.h"
#include "tsuner_b200.h"

#define EXPECT(c)                                                             \
    do {                                                                      \
        if (!(c)) {                                                           \
            std::printf("line %d: %s [%s]\n", __LINE__, #c, tsu_corr_last_error()); \
            return 1;                                                         \
        }                                                                     \
    } while (0)

alignas(128) static char X[1 << 16], Z[1 << 16], Wk[32 * 9 * 32 * 2], Y[1 << 17];
static float dW[32 * 9 * 32], db[32];

static int both_convolutions(int device) {
    cudaSetDevice(device);
    EXPECT(tsu_corr_conv3x3(X, 1, 16, 16, Wk, nullptr, 0, nullptr, Y, nullptr, nullptr) == TSU_OK);
    EXPECT(tsu_corr_conv3x3_wgrad(X, Z, 1, 16, 16, dW, db, nullptr) == TSU_OK);
    return 0;
}

// the raw entry points on one device after the other: each has its own
// shared-memory attribute and SM count
static int two_devices() {
    if (both_convolutions(0) || both_convolutions(1) || both_convolutions(0)) return 1;
    // 4000 rows of nine column groups: the launch fills the device it is for
    for (int d = 0; d < 2; d++) {
        cudaSetDevice(d);
        fake::launches.clear();
        EXPECT(tsu_corr_conv3x3(X, 1, 4000, 72, Wk, nullptr, 0, nullptr, Y, nullptr, nullptr) == TSU_OK);
        EXPECT(fake::launches.size() == 1 && fake::launches[0].grid == 2u * fake::sms[d]);
        fake::launches.clear();
        EXPECT(tsu_corr_conv3x3_wgrad(X, Z, 1, 16 * 300, 8, dW, db, nullptr) == TSU_OK);
        EXPECT(fake::launches.size() == 2 && fake::launches[0].grid == (unsigned)fake::sms[d]);
    }
    TsuCorrector *c[2] = {};
    for (int d = 0; d < 2; d++) EXPECT(tsu_corr_create(&c[d], 32, 32, 4, 1, 7, d) == TSU_OK);
    for (int d = 0; d < 2; d++) tsu_corr_destroy(c[d]);
    return 0;
}

// first calls from several threads at once, on both devices
static int threads() {
    int bad[8] = {};
    std::thread t[8];
    for (int k = 0; k < 8; k++) t[k] = std::thread([&, k] { bad[k] = both_convolutions(k & 1); });
    for (auto &x : t) x.join();
    for (int b : bad) EXPECT(!b);
    EXPECT(fake::blocks.empty());
    return 0;
}

// a prediction's device memory: one map (16 B per fine cell) for one sample,
// two for several, one again where there is no room for two
static int predict_memory() {
    const int n = 64;
    const size_t np = (size_t)n * n, map = 16 * np;
    std::vector<float> H(np, 1.f), coarse(3 * 3 * np / 16, 1.f), out(6 * np);
    for (int room = 1; room <= 2; room++) {
        TsuCorrector *c = nullptr;
        EXPECT(tsu_corr_create(&c, n, n, 4, 1, 7, 0) == TSU_OK);
        EXPECT(tsu_corr_set_site(c, H.data()) == TSU_OK);
        EXPECT(tsu_corr_add_samples(c, 3, coarse.data(), nullptr) == TSU_OK);
        const size_t before = fake::in_use;
        fake::memory = before + room * map;
        EXPECT(tsu_corr_predict(c, 0, 1, out.data(), out.data() + 3 * np, nullptr, nullptr) == TSU_OK);
        EXPECT(fake::in_use == before + map);
        fake::launches.clear();
        EXPECT(tsu_corr_predict(c, 0, 3, out.data(), out.data() + 3 * np, nullptr, nullptr) == TSU_OK);
        EXPECT(fake::in_use == before + room * map);
        EXPECT(fake::launches.size() == 3 * 8);  // features, six layers, the map
        EXPECT(tsu_corr_destroy(c) == TSU_OK);
        EXPECT(fake::blocks.empty());
        fake::memory = ~(size_t)0;
    }
    return 0;
}

int main(int argc, char **argv) {
    const char *s = argc > 1 ? argv[1] : "";
    if (!std::strcmp(s, "two_devices")) return two_devices();
    if (!std::strcmp(s, "threads")) return threads();
    if (!std::strcmp(s, "predict_memory")) return predict_memory();
    return 2;
}
