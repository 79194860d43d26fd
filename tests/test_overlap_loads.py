"""Kernels of a solve are launched to overlap: the next one's blocks are
resident while the previous one still writes what they will read.  So the
sources give the read-only path (const __restrict__, __ldg) only to data that
the previous kernel cannot be writing: the caller's right-hand side and
metrics, the plan's twiddles and eigenvalues, and the iterate a sweep's x
forward reads, which the gate separates from the x inverse that wrote it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pascal_poisson_fft_b200", "csrc")
CONSTANT = {"f", "tw", "tw_half", "tw_n", "tw_ny", "tw_dct", "dmx", "dx3", "dmx3"}
FILES = ["ppf_x.cu", "ppf_x_dev.cuh", "ppf_y.cu", "ppf_y_dev.cuh", "ppf_ghost.cu", "ppf_misc_dev.cuh", "ppf_tdma.cu"]


@pytest.mark.parametrize("name", FILES)
def test_written_data_takes_ordinary_loads(name):
    text = open(os.path.join(CSRC, name)).read()
    if name == "ppf_tdma.cu":   # other kernels there are launched in ordinary order
        text = text.split("// Coefficient-array solves")[0]
        text = "".join(k for k in re.split(r"(?=__global__)", text) if "pdl_enter();" in k)
    names = set(re.findall(r"const [\w<>:]+\s*\*\s*__restrict__\s+(\w+)", text))
    assert names <= CONSTANT, names - CONSTANT
    # loads through __ldg or ldg: of pairs of the right-hand side (fl) and of
    # the iterate (p of ld_pair_al), and of tables
    loads = set(re.findall(r"\b(?:__ldg|ldg)\(\s*(?:reinterpret_cast<[^>]*>\()?\s*([\w.]+)", text))
    assert loads <= CONSTANT | {"fl", "p"}, loads


def test_the_iterate_is_not_a_restricted_pointer():
    # the FP32 first iterate is only read by the pass that adds to it, which
    # without a const would be found read-only all the same
    for name in ("ppf_x.cu", "ppf_x_dev.cuh"):
        assert not re.search(r"float\s*\*\s*__restrict__\s+U\b", open(os.path.join(CSRC, name)).read())


def test_the_z_solves_read_through_plain_pointers():
    # in place: read after the wait, so not restricted (a restricted pointer's
    # loads may be moved above the wait)
    text = open(os.path.join(CSRC, "ppf_tdma.cu")).read()
    kernels = re.findall(r"__global__[^{;]*?(k_\w+)\(([^{;]*?)\)\s*\{\s*pdl_enter\(\);", text)
    assert {k for k, _ in kernels} >= {"k_thomas_z", "k_thomas_exact", "k_thomas_tab", "k_thomas_tab_cyc"}
    for kernel, params in kernels:
        assert not re.search(r"__restrict__\s+data_", params), kernel


def test_the_gate_separates_the_iterate_from_its_readers():
    # every pass of a mixed solve is followed by the gate, on the same stream
    text = open(os.path.join(CSRC, "ppf_api.cu")).read()
    body = text[text.index("int solve_impl("):]
    body = body[:body.index("launch_ghosts(")]
    steps = re.findall(r"run_pass<float>|launch_sweep_gate", body)
    assert steps == ["run_pass<float>", "launch_sweep_gate"] * 2
