"""How launches share the GPU, asked of the library's own host code (no GPU):
plan_check.cu is built against the library and answers queries."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cfd-simulator_b200")
# six SST solves whose plan needs other CTAs, and other shared memory, once the
# first, fifth and sixth are laminar
SIX = [(502, 55), (324, 55), (708, 132), (318, 60), (302, 185), (162, 152)]


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan_check")
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "plan_check.cu"), os.path.join(PKG, "libcfd_b200.so"),
                    "-Xlinker", "-rpath", "-Xlinker", PKG], check=True)

    def run(queries):
        out = subprocess.run([exe], input="\n".join(queries) + "\n", text=True, capture_output=True, check=True).stdout
        return [[int(v) for v in row.split()] for row in out.splitlines()]
    return run


def plan(jobs, threads=512, capacity=148):
    return f"plan {capacity} {threads} " + " ".join(f"{ni} {nj} {sst}" for ni, nj, sst in jobs)


def test_a_plan_changes_with_a_members_model(ask):
    before, after = ask([plan([(i, j, 1) for i, j in SIX]),
                         plan([(i, j, 0 if k in (0, 4, 5) else 1) for k, (i, j) in enumerate(SIX)])])
    assert before[3] == after[3] == 1
    assert before[:2] != after[:2]  # so a graph of the one must not replay against the other


def test_plans_of_any_batch_are_sound(ask):
    rng = random.Random(4)
    queries = []
    for _ in range(300):
        jobs = [(2 * rng.randint(10, 400), rng.randint(5, 200), rng.randint(0, 1)) for _ in range(rng.randint(1, 40))]
        queries.append(plan(jobs, threads=rng.choice([64, 128, 256, 512])))
    for query, (ctas, smem, teams, ok) in zip(queries, ask(queries)):
        assert ok == 1 and 1 <= ctas <= 148 and teams >= 1 and 0 < smem <= 222032, query


def test_a_wait_behind_other_solves_stays_within_its_limit(ask):
    # a CTA that has no part in a solve waits for it in the next one
    cases = [(32, 200, [(1500, 700, 1)] * 8 + [(1600, 400, 1)] * 8),
             (32, 200, [(1400, 380, 1)] * 12 + [(2400, 600, 1)] * 12),
             (256, 200, [(768, 192, 1)] * 21 + [(192, 48, 1), (384, 96, 1), (768, 192, 1)]),
             (256, 2000, [(768, 192, 1)] * 21 + [(192, 48, 1), (384, 96, 1), (768, 192, 1)]),
             (8, 100000, [(768, 192, 1)] * 4 + [(384, 96, 0)] * 9)]
    rng = random.Random(7)
    for _ in range(100):
        jobs = [(2 * rng.randint(10, 1500), rng.randint(5, 900), rng.randint(0, 1)) for _ in range(rng.randint(2, 30))]
        cases.append((rng.choice([1, 32, 256]), rng.choice([50, 200, 2000, 50000]), jobs))
    queries = [plan(jobs).replace("plan 148 512", f"waits 148 512 {n} {cap}") for n, cap, jobs in cases]
    for query, (permille,) in zip(queries, ask(queries)):
        assert permille <= 500, query


def test_every_column_tile_holds_columns(ask):
    # the plain CG's tiling, for every block size up to 5,000 columns and any threads
    queries = [f"tiles {threads} {nj} 1 5000" for threads in range(32, 513, 32) for nj in (1, 6, 48, 192, 400, 3000)]
    for query, (bad, where) in zip(queries, ask(queries)):
        assert bad == 0, (query, bad, where)


def test_a_sweep_of_any_width_fits_on_chip(ask):
    widths = list(range(1, 4000, 37)) + [104448, 104449, 104450, 130000, 355000, 10 ** 6, 10 ** 8]
    for ni, (size,) in zip(widths, ask([f"sweeps {ni}" for ni in widths])):
        assert 0 <= size <= 222032, (ni, size)


def test_planning_many_solves_is_quick(ask):
    # a plan is made between launches, with the GPU idle: 20 ms each with every number
    # of teams tried and every solve priced for it, 0.5 ms now
    import time
    queries = [plan([(192, 48, 1)] * 512)] * 100
    start = time.perf_counter()
    assert all(ok == 1 for _, _, _, ok in ask(queries))
    assert time.perf_counter() - start < 1.0


def test_a_lone_launch_leaves_room_for_others(ask):
    grids = [(192, 48), (384, 96), (768, 192), (234, 61), (1500, 60)]
    queries = [f"share 148 512 {n} {ni} {nj} 1" for ni, nj in grids for n in (1, 2, 3, 7, 200)]
    answers = ask(queries)
    for query, (share, least, used) in zip(queries, answers):
        assert least <= used <= share <= 148, query
    for k, _ in enumerate(grids):
        alone, two = answers[5 * k], answers[5 * k + 1]
        assert alone[2] > 74 or two[2] == alone[2]  # narrower only if two do not fit
        assert 2 * two[2] <= 148 or two[2] == alone[2]


def test_every_team_is_whole_rows_of_ctas(ask):
    rng = random.Random(11)
    queries = [f"whole {rng.randint(1, 148)} {rng.choice([32, 64, 128, 256, 512])} {rng.randint(1, 3000)} "
               f"{rng.randint(1, 1500)}" for _ in range(3000)]
    for query, (ok,) in zip(queries, ask(queries)):
        assert ok == 1, query
