// The sweep planner with its k-th allocation failing, for every k: it has to throw, and end its threads.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

extern "C" int sweep_plan_throws(int n, const int *pntr, const int *indx, const int *diag);

static std::atomic<long> g_left{-1};   // allocations until one fails; negative: none does
void *operator new(size_t bytes) {
    if (g_left.load() >= 0 && g_left.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void *p = std::malloc(bytes ? bytes : 1)) return p;
    throw std::bad_alloc();
}
void *operator new[](size_t bytes) { return operator new(bytes); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
void operator delete[](void *p, size_t) noexcept { std::free(p); }

int main() {
    const int n = 80000, stride = 200;   // a grid of 200 x 400: up to five planning threads
    std::vector<int> pntr(1, 0), indx, diag;
    for (int i = 0; i < n; i++) {
        if (i >= stride) indx.push_back(i - stride);
        if (i % stride) indx.push_back(i - 1);
        diag.push_back((int)indx.size());
        indx.push_back(i);
        pntr.push_back((int)indx.size());
    }
    int thrown = 0;
    for (long k = 0;; k = std::max(k + 1, k * 11 / 10)) {
        g_left = k;
        const int st = sweep_plan_throws(n, pntr.data(), indx.data(), diag.data());
        const bool failed = g_left.exchange(-1) < 0;
        if (!failed) {   // fewer allocations than k
            if (st != 0) return 1;
            break;
        }
        thrown += st == -1;
    }
    std::printf("%d\n", thrown);
    return thrown > 20 ? 0 : 2;
}
