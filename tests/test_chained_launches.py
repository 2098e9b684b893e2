"""Kernels that are set up while their predecessors still run (launch.cuh).

On the CPU, the rule that makes it safe, from the sources: a waiting kernel is
resident while the kernels before it write, so it must not read their output
through the read-only path (const __restrict__ parameters, __ldg) nor through any
pointer whose loads the compiler may move above the wait.  On the GPU: many steps
of a context without markers, which run as one graph of chained kernels, equal
the same steps one by one, bit for bit, from even and odd step numbers and with
the concentration set in between."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "softflow_b200", "csrc")

# the __restrict__ parameters of each chained kernel, all of them constant over the
# chain, the kernel's own caller's data, or only written by the kernel
CONSTANT = {"items", "chans", "links", "rows", "cfield", "caps", "off", "pos", "frc", "x", "t"}
KERNELS = {
    "k_lattice_step": CONSTANT | {"dst", "gdst"},
    "k_lattice_step_bc": CONSTANT | {"dst"},
    "k_lattice_step4": CONSTANT | {"dst", "gdst"},
    "k_lattice_step8h": CONSTANT | {"dst", "status"},
    "k_ibb": CONSTANT,
    "k_zou_he": CONSTANT,
    "k_marker_prep": CONSTANT | {"phi_tbl"},
    "k_tile_slots": CONSTANT,
    "k_tile_fill": CONSTANT | {"list"},
    "k_sa_init": CONSTANT,
    "k_sa_prep": CONSTANT,
    "k_sa_alloc": CONSTANT,
    "k_sa_fill": CONSTANT,
    "k_sa_gather": CONSTANT | {"Fx", "Fy"},
    "k_mlp_train_tile": CONSTANT | {"part", "part_loss", "status"},
    "k_mlp_adam": CONSTANT | {"g_out", "loss_out", "md"},
}
# functions that chained kernels pass other kernels' output to
FUNCTIONS = {"lattice_run4f": {"dst", "gdst", "cfield"}, "lattice_run4": {"dst", "gdst", "cfield"},
             "lattice_run8h": {"dst", "status"}, "contact_cells": {"chans"},
             "warp_tile_add": set(), "band_spread": set(), "group_sort": set(),
             "tile_list_sort": set(), "phi_lut": set(), "load_model": set()}


def _sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                out[f] = re.sub(r"//[^\n]*", "", h.read())
    return out


def _functions(text):
    """(name, parameter list, body) of every function with a body."""
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        i, depth = m.end(), 1
        while depth and i < len(text):
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        head = re.match(r"\s*(const\s*)?\{", text[i:])
        if not head:
            continue
        j = k = i + head.end()
        depth = 1
        while depth and k < len(text):
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), text[m.end():i - 1], text[j:k]


def _restricted(params):
    return set(re.findall(r"__restrict__\s+(\w+)", params))


def test_chained_kernels_read_other_kernels_output_with_ordinary_loads():
    seen, helpers = set(), set()
    for text in _sources().values():
        for name, params, body in _functions(text):
            if "chain_begin(" in body and name.startswith("k_"):
                seen.add(name)
                assert name in KERNELS, name
                assert _restricted(params) <= KERNELS[name], name
                for local in re.findall(r"const \w+\* __restrict__ (\w+) =", body):
                    raise AssertionError(f"{name}: {local}")
            if name in FUNCTIONS:
                helpers.add(name)
                assert _restricted(params) <= FUNCTIONS[name], name
    assert seen == set(KERNELS) and helpers == set(FUNCTIONS)


def test_no_load_names_the_read_only_path():
    """The qualifiers of a kernel's parameters alone decide which path its loads take."""
    for f, text in _sources().items():
        assert "__ldg" not in text and "ld.global.nc" not in text, f


# ------------------------------------------------------------------ on the GPU

def _build(name, precision):
    from cases import CASES, build_gpu, gaussian_conc
    import oracle as O
    extra = {
        # FP16-shifted storage: eight, four and one cell a lane by the row length
        "wide": dict(spec=dict(nx=520, ny=21, collision=O.MRT, tau=0.8, body_fx=2e-5),
                     capsules=[], conc=None),
        "four": dict(spec=dict(nx=132, ny=20, collision=O.BGK, tau=0.8, body_fx=2e-5),
                     capsules=[], conc=None),
        "odd": dict(spec=dict(nx=67, ny=19, collision=O.REGULARIZED, tau=0.8, body_fx=2e-5),
                    capsules=[], conc=None),
        "large": dict(spec=dict(nx=1028, ny=600, collision=O.BGK, tau=0.8, body_fx=1e-6),
                      capsules=[], conc=None),
        "scalar": dict(spec=dict(nx=96, ny=24, collision=O.BGK, tau=0.8, body_fx=2e-5,
                                 scalar_enabled=1, scalar_D=0.05),
                       capsules=[], conc=gaussian_conc(48.0, 11.5, 6.0)),
        "scalar_odd": dict(spec=dict(nx=67, ny=24, collision=O.MRT, tau=0.8, body_fx=2e-5,
                                     scalar_enabled=1, scalar_D=0.05),
                           capsules=[], conc=gaussian_conc(30.0, 11.5, 6.0)),
    }
    return build_gpu(extra.get(name) or CASES[name], precision)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16s"])
@pytest.mark.parametrize("name", ["wide", "four", "odd", "large", "scalar", "scalar_odd",
                                  "zouhe_reg", "cavity", "pillars_ibb", "pillars_zouhe"])
@pytest.mark.parametrize("start", [2, 3])
def test_chained_steps_equal_single_steps(sfg, oracle_mod, name, precision, start):
    """35 steps are two graphs of 16 and three single steps; then the concentration
    is set anew, and 17 more follow."""
    out = []
    for chained in (True, False):
        sim = _build(name, precision)
        ctx, ad = sim.context(), sim.advectionDiffusion()
        for _ in range(start):
            ctx.step(1)
        for n in (35, 17):
            if chained:
                ctx.step(n)
            else:
                for _ in range(n):
                    ctx.step(1)
                    ctx.synchronize()
            if ad is not None and n == 35:
                ad.setConcentration(ad.concentration()[::-1].copy())
        out.append([sim.field().distributions(), *sim.field().macroscopic()])
        if ad is not None:
            out[-1] += [ad.populations(), ad.concentration()]
        sim.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    assert np.abs(out[0][2]).max() > 0
