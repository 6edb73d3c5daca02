"""The C-ABI library loads and exports every symbol include/*.h declares;
host-side argument validation works without a GPU."""
import ctypes as C
import glob
import os
import re

import pytest

import picgpu as P
from conftest import ROOT


def header_functions():
    names = set()
    for h in glob.glob(os.path.join(ROOT, "include", "*.h")):
        src = open(h).read()
        src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
        names |= set(re.findall(r"\b(pic_[a-z0-9_]+)\s*\(", src))
    return sorted(names)


def test_header_declares_functions():
    assert "pic_create" in header_functions()
    assert "pic_compat_run" in header_functions()


@pytest.mark.parametrize("name", header_functions())
def test_library_exports(name):
    lib = C.CDLL(P.LIB_PATH)
    assert hasattr(lib, name), name


def test_binding_covers_header():
    assert set(header_functions()) <= set(P.SIGNATURES)


def test_status_strings():
    L = P.load()
    assert L.pic_status_string(0) == b"ok"
    assert L.pic_status_string(7) == b"device wait timed out"


def test_config_validation_is_host_side():
    bad = P.config(1, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, -1)])
    with pytest.raises(P.PicError) as e:
        P.Handle(bad)
    assert e.value.status == 1
    bad = P.config(64, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, 0)])  # q without q_int
    with pytest.raises(P.PicError) as e:
        P.Handle(bad)
    assert e.value.status == 1
    bad = P.config(64, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, -1),
                                           P.species(100, 1.5, 1.0, 1)])  # not integer multiples
    with pytest.raises(P.PicError) as e:
        P.Handle(bad)
    assert e.value.status == 1
    # push chunks above 32768 particles could overflow the window's 32-bit cell moments
    bad = P.config(64, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, -1)], chunk=32772)
    with pytest.raises(P.PicError) as e:
        P.Handle(bad)
    assert e.value.status == 1
    # the bulk-copy push pipelines (variants 2 and 4) were removed
    for variant in (2, 4, -1):
        bad = P.config(64, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, -1)],
                       push_variant=variant)
        with pytest.raises(P.PicError) as e:
            P.Handle(bad)
        assert e.value.status == 1


def test_compat_params_validation_is_host_side():
    import numpy as np
    p = P.ref_params(nx=1)
    with pytest.raises(P.PicError) as e:
        P.compat_run(p, *(np.zeros(100) for _ in range(4)))
    assert e.value.status == 1


def test_no_device_is_reported(monkeypatch):
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    c = P.config(64, 64, 1.0, 1.0, 0.1, [P.species(100, -1.0, 1.0, -1)])
    with pytest.raises(P.PicError) as e:
        P.Handle(c)
    assert e.value.status == 9


@pytest.mark.parametrize("struct,ctype", [
    ("pic_ref_params", P.RefParams), ("pic_species_desc", P.SpeciesDesc), ("pic_config", P.Config),
    ("pic_init_spec", P.InitSpec), ("pic_diag", P.Diag), ("pic_mcc_params", P.MccParams),
    ("pic_dsmc_params", P.DsmcParams), ("pic_tune_result", P.TuneResult),
    ("pic_adjoint_result", P.AdjointResult), ("pic_particles_view", P.ParticlesView)])
def test_binding_structures_are_laid_out_as_the_header_s(struct, ctype, tmp_path):
    """Every field of the C structure, in order, at the offset the binding gives it."""
    import subprocess

    src = re.sub(r"/\*.*?\*/", "", open(os.path.join(ROOT, "include", "pic.h")).read(), flags=re.S)
    body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (struct, struct), src, re.S)[1]
    fields = [re.sub(r"\[.*", "", f.strip().lstrip("*").strip()) for d in body.split(";") if d.strip()
              for f in re.sub(r"^\s*(const\s+)?(unsigned\s+)?(long\s+long|\w+)\s", "", d.strip()).split(",")]
    assert fields == [f[0] for f in ctype._fields_]
    c = tmp_path / "layout.c"
    c.write_text('#include <stddef.h>\n#include <stdio.h>\n#include "pic.h"\nint main(void) {\n' +
                 "".join(f'printf("%zu ", offsetof({struct}, {f}));\n' for f in fields) +
                 f'printf("%zu", sizeof({struct}));\nreturn 0;\n}}\n')
    subprocess.run(["gcc", "-I" + os.path.join(ROOT, "include"), str(c), "-o", str(tmp_path / "layout")], check=True)
    got = [int(x) for x in subprocess.run([str(tmp_path / "layout")], capture_output=True, check=True).stdout.split()]
    assert got == [getattr(ctype, f).offset for f in fields] + [C.sizeof(ctype)]
