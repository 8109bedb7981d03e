// csrc/level_route.h over every kind of output; prints "ok".
#include <cstdio>

#include "level_route.h"

using gbfs::LevelRoute;

static const int32_t *at(uintptr_t p) { return reinterpret_cast<const int32_t *>(p); }

static LevelRoute route(int type, int ptr_device, int device, uintptr_t p = 1024)
{
    return gbfs::level_route(at(p), type, ptr_device, device);
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
    std::printf(routes && aligned ? "ok\n" : "wrong: %d %d\n", routes, aligned);
    return routes && aligned ? 0 : 1;
}
