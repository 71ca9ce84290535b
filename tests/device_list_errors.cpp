// Errors of DeviceList::replace (lbm_device_list.h) on the host, with memory whose first, second or no call fails:
// after an error data and count are the former list's, and nothing leaks.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "lbm_device_list.h"

static int calls_left = 1 << 30, live = 0;
struct FakeMem {
    static constexpr int OK = 0;
    static int alloc(void** p, size_t bytes) {
        if (calls_left-- <= 0) return 2;
        *p = malloc(bytes);
        ++live;
        return OK;
    }
    static int upload(void* dst, const void* src, size_t bytes) {
        if (calls_left-- <= 0) return 1;
        memcpy(dst, src, bytes);
        return OK;
    }
    static void release(void* p) {
        free(p);
        --live;
    }
};

#define CHECK(c) \
    if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }

int main() {
    lbm::DeviceList<int, FakeMem> l;
    for (int ok = 0; ok < 2; ++ok) {  // nothing to keep yet: an empty list
        calls_left = ok;
        CHECK(l.replace({7, 8}) == (ok ? 1 : 2) && l.data == nullptr && l.count == 0 && live == 0);
    }
    calls_left = 1 << 30;
    CHECK(l.replace({1, 2, 3}) == 0 && l.count == 3 && live == 1);
    for (int ok = 0; ok < 2; ++ok) {
        calls_left = ok;
        CHECK(l.replace({4, 5, 6, 7, 8}) == (ok ? 1 : 2));
        CHECK(l.data && l.count == 3 && l.data[0] == 1 && l.data[2] == 3 && live == 1);
    }
    calls_left = 1 << 30;
    CHECK(l.replace({4, 5}) == 0 && l.count == 2 && l.data[1] == 5 && live == 1);
    l.clear();
    CHECK(l.data == nullptr && l.count == 0 && live == 0);
    printf("list errors: ok\n");
    return 0;
}
