// smem_opt_in (honei_b200/csrc/smem_opt_in.hh) against a stand-in for the two CUDA calls it
// makes: two devices with a limit per kernel each, one of which can be made to refuse.
#include "../../honei_b200/csrc/smem_opt_in.hh"

#include <cstdio>
#include <thread>
#include <vector>

static thread_local int t_device = 0;
static std::mutex g_mu;
static std::map<std::pair<const void *, int>, int> g_limit;
static int g_calls = 0;
static bool g_refuse = false;

extern "C" cudaError_t CUDARTAPI cudaGetDevice(int * device)
{
    *device = t_device;
    return cudaSuccess;
}

extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void * f, cudaFuncAttribute, int value)
{
    std::lock_guard<std::mutex> lock(g_mu);
    ++g_calls;
    if (g_refuse) return cudaErrorInvalidValue;
    g_limit[std::make_pair(f, t_device)] = value;
    return cudaSuccess;
}

static int failures = 0;
static void check(bool ok, const char * what)
{
    if (ok) return;
    ++failures;
    std::printf("FAILED: %s\n", what);
}

static int limit(const void * f, int device)
{
    std::lock_guard<std::mutex> lock(g_mu);
    return g_limit[std::make_pair(f, device)];
}

int main()
{
    static const char kernel[3] = {};
    const void * a = kernel, * b = kernel + 1, * c = kernel + 2;

    check(hb2::smem_opt_in(a, 60000) == cudaSuccess && limit(a, 0) == 60000, "the first launch opts in");
    check(hb2::smem_opt_in(a, 60000) == cudaSuccess && g_calls == 1, "a second one makes no call");
    check(hb2::smem_opt_in(a, 50000) == cudaSuccess && limit(a, 0) == 60000, "never lowered");
    check(hb2::smem_opt_in(a, 90000) == cudaSuccess && limit(a, 0) == 90000, "raised where needed");
    t_device = 1;
    check(hb2::smem_opt_in(a, 60000) == cudaSuccess && limit(a, 1) == 60000, "the second device on its own");
    g_refuse = true;
    check(hb2::smem_opt_in(b, 70000) == cudaErrorInvalidValue, "a refusal is returned");
    g_refuse = false;
    check(hb2::smem_opt_in(b, 70000) == cudaSuccess && limit(b, 1) == 70000, "and not remembered");
    t_device = 0;

    // every thread finds its own size allowed after its call, whatever the others ask for
    std::vector<std::thread> threads;
    bool ok[8];
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            ok[t] = true;
            for (int i = 0; i < 2000; ++i)
            {
                const int bytes = 50000 + 1000 * ((i * 7 + t * 13) % 40);
                ok[t] = hb2::smem_opt_in(c, bytes) == cudaSuccess && limit(c, 0) >= bytes && ok[t];
            }
        });
    for (auto & t : threads) t.join();
    for (int t = 0; t < 8; ++t) check(ok[t], "concurrent sizes");
    if (! failures) std::printf("ok\n");
    return failures != 0;
}
