// Runs the control flow of the tensor-core GEMM's TMA-store epilogue (csrc/kernels/gemm_tc.cu, cut out of the source by the test into epilogue_body.inc) on the CPU: a warp
// is an OS thread, named barriers count warps and give up after a while, tensor memory and stores are stubs that take notes.  Every warp's wait for the accumulator
// succeeds or gives up on its own; whatever the four answers, no warp may be left waiting for another, and columns are stored where both warps that hold
// them have the accumulator.  Build: g++ -O1 -std=c++20 -pthread -I <folder of epilogue_body.inc> gemm_epilogue_emu.cpp
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>
using std::min;

static const int BM = 128;
struct Params { const float* bias; int splits, M, N, tma_out; int* err; };
struct Map {};
static std::mutex g_mu;
static std::condition_variable g_cv;
struct Bar { int arrived = 0, round = 0; bool all = true, answer = true; };
static Bar g_bar[16];
static bool g_stuck;
static std::vector<int> g_stored;                        // first column of every store
static bool g_wait_ok[4];                                // by quarter
static thread_local int t_quarter;

static bool meet(int id, int threads, bool ok) {
    std::unique_lock<std::mutex> l(g_mu);
    Bar& b = g_bar[id];
    b.all = b.all && ok;
    if (++b.arrived == threads / 32) {
        b.answer = b.all; b.all = true; b.arrived = 0; ++b.round;
        g_cv.notify_all();
        return b.answer;
    }
    const int r = b.round;
    if (!g_cv.wait_for(l, std::chrono::milliseconds(300), [&] { return b.round != r; })) { g_stuck = true; return false; }
    return b.answer;
}
static void bar_sync(int id, int threads) { meet(id, threads, true); }
[[maybe_unused]] static bool bar_all(int id, int threads, bool ok) { return meet(id, threads, ok); }
static bool mbar_wait(void*, int, int*, int) { return g_wait_ok[t_quarter]; }
static bool __all_sync(unsigned, bool v) { return v; }
static void __syncwarp() {}
static void tc_fence_after() {}
static void fence_proxy_async() {}
static void bulk_commit_wait() {}
static bool elect_one() { return true; }
static uint32_t smem_u32(const void*) { return 0; }
template <int C> static void tmem_ld_pieces(uint32_t, uint32_t* r) { for (int i = 0; i < C / 2; ++i) r[i] = 0; }
static float __uint_as_float(uint32_t) { return 0.f; }
static uint32_t pack_bf16x2(float, float) { return 0; }
static void stmatrix_x4_trans(uint32_t, const uint32_t*) {}
static void tma_store_2d(const void*, const Map*, int x, int) { std::lock_guard<std::mutex> l(g_mu); g_stored.push_back(x); }
static void tma_store_3d(const void*, const Map*, int x, int, int) { std::lock_guard<std::mutex> l(g_mu); g_stored.push_back(x); }

template <int BN, bool BATCHED> static void epilogue(int warp, Params p, int n0, int m0) {
    const int lane = 0, nkb = 1, batch = 0;
    [[maybe_unused]] const int split = 0;
    const uint32_t tmem_d = 0;
    static uint8_t smem[256 * 1024];
    int acc = 0;
    int* acc_full = &acc;
    Map map_o;
#include "epilogue_body.inc"
}

template <int BN> static int run(int N, int M) {
    int bad = 0;
    for (int answers = 0; answers < 16; ++answers) {
        for (int q = 0; q < 4; ++q) g_wait_ok[q] = answers >> q & 1;
        for (auto& b : g_bar) b = Bar();
        g_stuck = false;
        g_stored.clear();
        const Params p{nullptr, 1, M, N, 1, nullptr};
        std::vector<std::thread> th;
        for (int w = 2; w < 6; ++w) th.emplace_back([=] { t_quarter = w & 3; epilogue<BN, false>(w, p, 0, 0); });
        for (auto& t : th) t.join();
        const int ch = BN < 64 ? BN : 64, pieces = (min(BN, M) + ch - 1) / ch;
        for (int half = 0; half < 2; ++half) {
            const int want = g_wait_ok[2 * half] && g_wait_ok[2 * half + 1] && half * 64 < N ? pieces : 0;
            if (std::count(g_stored.begin(), g_stored.end(), half * 64) != want) ++bad;
        }
        if (g_stuck) ++bad;
    }
    return bad;
}

int main() {
    const int bad = run<16>(128, 5) + run<64>(64, 64) + run<256>(128, 200) + run<256>(100, 256);
    printf("bad=%d\n", bad);
    return bad ? 1 : 0;
}
