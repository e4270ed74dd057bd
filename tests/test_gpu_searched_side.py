"""The comparisons with "the searched step" once more, with a handle that does search.

A handle whose configuration has neighbor_skin 0 steps on lists of the library's own where a run
of steps pays for them, so tests that take one for the searched side compare lists with lists.
Here such handles are told to search (set_neighbor_skin(0)) and are seen to do so after every
call, and the same test bodies run on them: lists against searching, and the searched step
against the oracle, five steps of 2^20 grains among them."""
from __future__ import annotations

import pytest

import test_gpu_lists
import test_gpu_scale
from test_gpu_scale import c1_settled                          # noqa: F401 (a fixture)
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


class Searched(ParticleDynamics):
    def __init__(self, config, **kw):
        super().__init__(config, **kw)
        if config.neighbor_skin == 0.0:
            self.set_neighbor_skin(0.0)

    def _seen(self):
        if self.tuning()["neighbor_skin_m"] == 0.0:
            assert self.kernels_per_step() >= 5                # on lists: 1 or 2

    def advance(self, steps):
        super().advance(steps)
        self._seen()

    def take_step(self):
        super().take_step()
        self._seen()


def _cases(module, *names):
    return [pytest.param(getattr(module, name), args, id=f"{name}-{'-'.join(map(str, args))}".rstrip("-"))
            for name, *rows in names for args in (rows or [()])]


@pytest.mark.parametrize("body,args", _cases(
    test_gpu_lists,
    ("test_lists_equal_search_every_step_packed_springs", (False,), (True,)),
    ("test_lists_equal_search_every_step_reference_cube",),
    ("test_lists_equal_search_in_a_collapsing_column",),
    ("test_lists_hold_pairs_two_cells_apart", (0, 1.5e-3), (1, 2.5e-3), (2, 2.5e-3)),
    ("test_builds_follow_the_displacement_bound",),
    ("test_tiny_skin_and_overflowing_lists_stay_exact",),
    ("test_set_state_mid_run_rebuilds",),
    ("test_skin_switch_mid_run_stays_exact",),
    ("test_every_contact_kernel_variant_is_exact", (0, 256), (64, 128), (48, 64), (1, 256), (2, 256)),
    ("test_contact_kernel_switches_mid_run",),
    ("test_bulk_staged_kernel_over_many_tiles",),
    ("test_contact_parallel_kernel_equals_search", (31, True, False), (33, False, False),
     (16383, True, False), (16385, True, False), (40000, False, False)),
    ("test_contact_parallel_kernel_many_contacts_on_one_grain", (30,), (33,), (60,)),
    ("test_chains_launched_early_equal_search", (16383,), (16384,), (75776,), (75777,))))
def test_lists_against_searching(body, args, monkeypatch):
    monkeypatch.setattr(test_gpu_lists, "ParticleDynamics", Searched)
    body(*args)


@pytest.mark.parametrize("body,args", _cases(
    test_gpu_scale,
    ("test_c0_column_from_rest_bit_exact",),
    ("test_c0_collapsing_column_bit_exact", (0.0,)),
    ("test_c1_bench_workload_from_rest_bit_exact", ("searched",))))
def test_searching_against_the_oracle(body, args, monkeypatch, oracle_for):
    monkeypatch.setattr(test_gpu_scale, "ParticleDynamics", Searched)
    body(oracle_for, *args)


def test_searching_a_settled_column_against_the_oracle(monkeypatch, oracle_for, c1_settled):  # noqa: F811
    monkeypatch.setattr(test_gpu_scale, "ParticleDynamics", Searched)
    test_gpu_scale.test_c1_settled_column_bit_exact(oracle_for, c1_settled, "searched")
