// Co-resident blocks of the cooperative kernels, the same for every context of a device: asked
// for once per device (the occupancy queries are a good part of a small world's creation). Plain
// C++, so that the failure paths run without a device.
#pragma once

#include <map>
#include <mutex>

namespace avbd
{

struct LaunchShape
{
    int colourBlocks = 1, colourFlowBlocks = 1, iterBlocks = 0, wideBlocks = 0;
};

class LaunchShapes
{
public:
    // `iterations`: this context could set the iteration kernels' attributes. query(iterations,
    // shape) fills the shape and returns whether every answer came; only a whole answer is kept,
    // so that one failed call costs that context its single-launch iterations and no later one.
    template <class Query>
    LaunchShape of(int device, bool iterations, Query query)
    {
        std::lock_guard<std::mutex> hold(lock);
        auto it = known.find(device);
        LaunchShape shape;
        if (it != known.end())
            shape = it->second;
        else if (query(iterations, shape) && iterations)
            known.emplace(device, shape);
        if (!iterations)
            shape.iterBlocks = shape.wideBlocks = 0;
        return shape;
    }

private:
    std::mutex lock;
    std::map<int, LaunchShape> known;
};

} // namespace avbd
