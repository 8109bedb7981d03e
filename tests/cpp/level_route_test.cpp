// csrc/level_route.h over every kind of output; prints "ok".
#include <cstdio>

#include "level_route.h"

using gbfs::LevelRoute;

static const int32_t *at(uintptr_t p) { return reinterpret_cast<const int32_t *>(p); }

static LevelRoute route(int type, int ptr_device, int device, uintptr_t p = 1024)
{
    return gbfs::level_route(at(p), type, ptr_device, device);
}

static bool overlap(std::vector<uintptr_t> ptr, std::vector<int32_t> count, std::vector<LevelRoute> r = {})
{
    std::vector<const int32_t *> out;
    for (uintptr_t p : ptr) out.push_back(at(p));
    r.resize(ptr.size(), LevelRoute::KERNEL);
    std::vector<std::pair<uintptr_t, uintptr_t>> scratch;
    return gbfs::outputs_overlap(out.data(), count.data(), r.data(), ptr.size(), scratch);
}

int main()
{
    const bool routes = route(0, 0, 0) == LevelRoute::HOST && route(1, 0, 0) == LevelRoute::HOST &&
                        route(1, 3, 0) == LevelRoute::HOST && route(2, 0, 0) == LevelRoute::KERNEL &&
                        route(2, 5, 5) == LevelRoute::KERNEL && route(2, 1, 0) == LevelRoute::COPY &&
                        route(2, 0, 1) == LevelRoute::COPY && route(3, 1, 0) == LevelRoute::KERNEL &&
                        route(3, 0, 0) == LevelRoute::KERNEL;
    const bool aligned = route(2, 0, 0, 1025) == LevelRoute::COPY && route(3, 0, 0, 1026) == LevelRoute::COPY &&
                         route(2, 0, 0, 1028) == LevelRoute::KERNEL && route(1, 0, 0, 1027) == LevelRoute::HOST;
    const bool apart = !overlap({}, {}) && !overlap({64}, {5}) && !overlap({64, 84}, {5, 5}) && !overlap({84, 64}, {5, 5}) &&
                       !overlap({200, 100, 300}, {25, 25, 25}) && !overlap({100, 100}, {0, 25});
    const bool over = overlap({64, 64}, {5, 5}) && overlap({64, 80}, {5, 5}) && overlap({80, 64}, {5, 5}) &&
                      overlap({300, 100, 200, 180}, {5, 5, 5, 6}) && overlap({100, 500, 104}, {50, 1, 1});
    const LevelRoute K = LevelRoute::KERNEL, C = LevelRoute::COPY, H = LevelRoute::HOST;
    const bool mixed = !overlap({64, 64, 64}, {5, 5, 5}, {K, H, H}) && overlap({64, 66}, {5, 5}, {K, C}) && overlap({64, 64, 64}, {5, 5, 5}, {K, H, K});
    std::printf(routes && aligned && apart && over && mixed ? "ok\n" : "wrong: %d %d %d %d %d\n", routes, aligned, apart, over, mixed);
    return routes && aligned && apart && over && mixed ? 0 : 1;
}
