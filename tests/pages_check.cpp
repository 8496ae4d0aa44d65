// populate_pages (csrc/lbm_pages.h) with the linker's stand-ins for madvise and getcpu, for
// test_cpu_pages.py.  argv[1] "far": every thread but the caller is on another memory node; "near": all
// on one.  Checks that the whole pages of the array, and nothing else, are asked for once each, and that
// no page is touched from another node than the caller's.
#include <sys/mman.h>

#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

#include "lbm_pages.h"

static std::thread::id caller;
static bool far_helpers = false;
static std::mutex lock;
static std::map<uintptr_t, size_t> asked;
static int bad = 0, from_helpers = 0;

extern "C" int __wrap_getcpu(unsigned* cpu, unsigned* node) {
    *cpu = 0;
    *node = far_helpers && std::this_thread::get_id() != caller ? 1 : 0;
    return 0;
}
extern "C" int __wrap_madvise(void* p, size_t n, int advice) {
    std::lock_guard<std::mutex> g(lock);
    bad += advice != MADV_POPULATE_WRITE || asked.count((uintptr_t)p) || (far_helpers && std::this_thread::get_id() != caller);
    from_helpers += std::this_thread::get_id() != caller;
    asked[(uintptr_t)p] = n;
    return 0;
}

int main(int, char** argv) {
    caller = std::this_thread::get_id();
    far_helpers = std::strcmp(argv[1], "far") == 0;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    for (size_t bytes : {size_t(1) << 20, size_t(4) << 20, (size_t(4) << 20) + 5 * page + 24, size_t(100) << 20}) {
        for (size_t off : {size_t(0), size_t(24)}) {
            char* m = (char*)mmap(nullptr, bytes + 2 * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            asked.clear();
            lbm::populate_pages(m + off, bytes);
            const uintptr_t b = ((uintptr_t)m + off + page - 1) / page * page, e = ((uintptr_t)m + off + bytes) / page * page;
            uintptr_t at = b;
            for (auto& [p, n] : asked) {
                bad += p != at;
                at = p + n;
            }
            bad += e - b < (size_t(4) << 20) ? !asked.empty() : at != e;
            munmap(m, bytes + 2 * page);
        }
    }
    if (bad) std::printf("FAIL %d\n", bad);
    else std::printf("ok %d\n", from_helpers);
    return bad != 0;
}
