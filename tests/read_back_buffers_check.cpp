// ReadBackBuffers (2dradiation_b200/csrc/read_back_buffers.hpp) over a
// counted fake allocator.  Prints the first expectation that fails; exits 0
// when none does.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>

#include "read_back_buffers.hpp"

static std::mutex g_m;
static std::set<char *> g_live;
static bool g_refuse = false;
static int g_bad = 0;
static char *fake_alloc()
{
    std::lock_guard<std::mutex> lock(g_m);
    if (g_refuse)
        return nullptr;
    char *p = static_cast<char *>(std::malloc(8));
    g_live.insert(p);
    return p;
}
static void fake_release(char *p)
{
    std::lock_guard<std::mutex> lock(g_m);
    if (!g_live.erase(p))
        g_bad++;
    std::free(p);
}
// a device's reset frees what its CUDA context had allocated
static void reset(std::set<char *> gone)
{
    for (char *p : gone)
        g_live.erase(p);
}
#define EXPECT(x)                                              \
    do                                                         \
        if (!(x))                                              \
        {                                                      \
            std::printf("line %d: %s\n", __LINE__, #x);        \
            return 1;                                          \
        }                                                      \
    while (0)

int main()
{
    using grlbm::ReadBackBuffers;
    ReadBackBuffers b(fake_alloc, fake_release);
    const ReadBackBuffers::Place zero{0, 11}, two{2, 12}, again{0, 13};
    // a buffer waits for the next read-back
    char *p = b.take(zero);
    b.give(zero, p);
    EXPECT(g_live.size() == 1 && b.take(zero) == p);
    b.give(zero, p);
    // another device has its own
    char *q = b.take(two);
    EXPECT(q != p && g_live.size() == 2);
    b.give(two, q);
    // bounded, per device
    char *many[9];
    for (char *&m : many)
        m = b.take(zero);
    for (char *m : many)
        b.give(zero, m);
    EXPECT(g_live.size() == 1 + ReadBackBuffers::kKept);
    // after a reset of the device none of its old buffers is handed out, or released
    std::set<char *> old = g_live;
    old.erase(q);
    reset(old);
    char *fresh[6];
    for (char *&m : fresh)
    {
        m = b.take(again);
        EXPECT(m && !old.count(m));
    }
    for (char *m : fresh)
        b.give(again, m);
    EXPECT(g_live.size() == 1 + ReadBackBuffers::kKept && g_bad == 0);
    // the other device's is still there
    EXPECT(b.take(two) == q);
    b.give(two, q);
    // none to be had
    g_refuse = true;
    EXPECT(b.take(ReadBackBuffers::Place{1, 14}) == nullptr);
    g_refuse = false;
    // several threads
    std::thread t[8];
    for (std::thread &x : t)
        x = std::thread([&b] {
            for (int k = 0; k < 2000; k++)
            {
                const ReadBackBuffers::Place at{k % 3, (unsigned long long)(20 + k % 3)};
                char *a = b.take(at), *c = b.take(at);
                if (!a || !c || a == c)
                    std::abort();
                b.give(at, a);
                b.give(at, c);
            }
        });
    for (std::thread &x : t)
        x.join();
    EXPECT(g_bad == 0);
    return 0;
}
