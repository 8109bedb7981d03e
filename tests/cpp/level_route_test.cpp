// csrc/level_route.h over every kind of output; prints "ok".
#include <cstdio>

#include "level_route.h"

using gbfs::LevelRoute;
using gbfs::level_route;

int main()
{
    const bool ok = level_route(0, 0, 0) == LevelRoute::HOST && level_route(1, 0, 0) == LevelRoute::HOST &&
                    level_route(1, 3, 0) == LevelRoute::HOST && level_route(2, 0, 0) == LevelRoute::KERNEL &&
                    level_route(2, 5, 5) == LevelRoute::KERNEL && level_route(2, 1, 0) == LevelRoute::COPY &&
                    level_route(2, 0, 1) == LevelRoute::COPY && level_route(3, 1, 0) == LevelRoute::KERNEL &&
                    level_route(3, 0, 0) == LevelRoute::KERNEL;
    std::printf(ok ? "ok\n" : "wrong route\n");
    return ok ? 0 : 1;
}
