// host_copy where the process cannot have the threads it would like: the copy is made by those there are.
#include <sys/resource.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "host_convert.cpp"

int main() {
    using glasssix::excalibur::host_copy;
    std::vector<char> src(8 << 20), dst(src.size());
    for (size_t i = 0; i < src.size(); ++i) src[i] = (char)(i * 7 + i / 4096);
    // room for one or two thread stacks
    long pages = 0;
    if (FILE* f = std::fopen("/proc/self/statm", "r")) {
        if (std::fscanf(f, "%ld", &pages) != 1) pages = 0;
        std::fclose(f);
    }
    const rlim_t room = (rlim_t)pages * sysconf(_SC_PAGESIZE) + (20 << 20);
    const rlimit limit = {room, room};
    if (setrlimit(RLIMIT_AS, &limit) != 0) return 1;
    size_t ready = 0;
    host_copy(dst.data(), src.data(), src.size(), [&](size_t n) { ready = n; });
    if (ready != src.size() || std::memcmp(dst.data(), src.data(), src.size())) return 2;
    std::memset(dst.data(), 0, dst.size());
    host_copy(dst.data(), src.data(), src.size());
    if (std::memcmp(dst.data(), src.data(), src.size())) return 3;
    std::printf("ok\n");
    return 0;
}
