"""The outlet columns that the drop-in interface hands out, when the sync mode changes between a collision and its
stream: every stream's own columns, with the host arrays pinned and not."""
import os
import subprocess

import pytest

import lbgpu

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "lb.h"
#include "boundaries.h"
#include "lbgpu.h"
#define LX 60
#define LY 24
static double omega = 1.4;
static Dynamics bulk, wall;
static size_t col = (LY + 2);

static void build(Simulation *sim)
{
    bulk.dynamicsFun = &bgk; bulk.selfData = &omega;
    wall.dynamicsFun = &bounceBack; wall.selfData = 0;
    constructSim(sim, LX, LY);
    for (int x = 1; x <= LX; ++x)
        for (int y = 1; y <= LY; ++y) {
            iniEquilibrium(&sim->lattice[x][y], 1. + 0.01 * ((x * 7 + y * 3) % 11), 0.01 * ((x + y) % 5), 0.01 * ((x * y) % 3));
            setDynamics(sim, x, y, (y == 1 || y == LY) ? &wall : &bulk);
        }
}

/* the two columns as the last call left them on the host, against the whole state */
static int columns_hold(Simulation *sim)
{
    Node *got = (Node *)malloc(2 * col * sizeof(Node));
    int ok = 1;
    memcpy(got, &sim->lattice[LX - 2][0], 2 * col * sizeof(Node));
    lbSyncToHost(sim);
    for (size_t k = 0; k < 2 * col; ++k)
        if (memcmp(got[k].fPop, sim->lattice[LX - 2][k].fPop, sizeof got[k].fPop)) ok = 0;
    free(got);
    return ok;
}

int main(int argc, char **argv)
{
    const int pinned = atoi(argv[1]), between = atoi(argv[2]), form = atoi(argv[3]);
    Simulation sim;
    build(&sim);
    if (pinned) {   /* whole copies pin the arrays */
        lbSetSyncMode(&sim, LB_SYNC_FULL);
        collide(&sim); propagate(&sim);
    }
    lbSetSyncMode(&sim, LB_SYNC_OUTLET);
    for (int round = 0; round < 3; ++round) {
        if (form) collide_with_stream(&sim); else collide(&sim);
        if (!columns_hold(&sim)) { printf("after collide\n"); return 1; }
        lbSetSyncMode(&sim, between);
        if (form) finalize_stream(&sim); else propagate(&sim);
        lbSetSyncMode(&sim, LB_SYNC_OUTLET);
        propagate(&sim);
        if (!columns_hold(&sim)) { printf("stale columns in round %d\n", round); return 1; }
        collide(&sim);
        propagate(&sim);
        if (!columns_hold(&sim)) { printf("own columns in round %d\n", round); return 1; }
    }
    if (lbGetLastError()) { printf("%s\n", lbGetLastErrorString()); return 1; }
    destructSim(&sim);
    printf("ok\n");
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("dropin") / "columns")
    with open(exe + ".c", "w") as f:
        f.write(SOURCE)
    libdir = os.path.dirname(lbgpu.LIB_PATH)
    subprocess.run(["gcc", "-O1", "-I", os.path.join(ROOT, "include"), "-o", exe, exe + ".c", "-L", libdir, "-llbgpu",
                    "-Wl,-rpath," + libdir], check=True)
    return exe


@pytest.mark.parametrize("pinned", [0, 1])
@pytest.mark.parametrize("between", ["none", "full"])
@pytest.mark.parametrize("form", [0, 1])
def test_each_stream_hands_out_its_own_columns(program, pinned, between, form):
    mode = {"none": 0, "outlet": 1, "full": 2}[between]
    r = subprocess.run([program, str(pinned), str(mode), str(form)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
