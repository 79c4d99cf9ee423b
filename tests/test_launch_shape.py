"""What contexts of a device share of their launch shape, where an attribute or an occupancy query
fails: made to fail on the host, without a device."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avbd_demo3d_b200", "csrc")

PROGRAM = r"""
#include "avbd_launch_shape.h"
#include <cstdio>
#include <cstdlib>
using namespace avbd;
static int queries = 0;
static void expect(bool ok, int line)
{
    if (!ok)
    {
        std::printf("line %d\n", line);
        std::exit(1);
    }
}
int main()
{
    LaunchShapes shapes;
    auto good = [](bool iterations, LaunchShape &s) {
        ++queries;
        s.colourBlocks = 296;
        s.colourFlowBlocks = 444;
        s.iterBlocks = s.wideBlocks = iterations ? 148 : 0;
        return true;
    };
    auto failing = [](bool, LaunchShape &s) {
        ++queries;
        s = LaunchShape();
        return false;
    };
    // a failed query leaves that context without the iteration kernels and the next one with them
    LaunchShape s = shapes.of(0, true, failing);
    expect(s.iterBlocks == 0 && s.wideBlocks == 0, __LINE__);
    s = shapes.of(0, true, good);
    expect(s.iterBlocks == 148 && s.wideBlocks == 148, __LINE__);
    // failed attributes likewise, on a device seen first so
    s = shapes.of(1, false, good);
    expect(s.iterBlocks == 0 && s.wideBlocks == 0 && s.colourBlocks == 296, __LINE__);
    s = shapes.of(1, true, good);
    expect(s.iterBlocks == 148 && s.wideBlocks == 148, __LINE__);
    // and on a device known whole, whose shape stays known
    const int before = queries;
    s = shapes.of(0, false, good);
    expect(s.iterBlocks == 0 && s.wideBlocks == 0 && s.colourFlowBlocks == 444, __LINE__);
    s = shapes.of(0, true, failing);
    expect(s.iterBlocks == 148 && s.wideBlocks == 148 && queries == before, __LINE__);
    return 0;
}
"""


def test_a_failed_call_costs_only_its_context(tmp_path):
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
