"""The C-ABI library loads and exports every symbol the header declares (no GPU, no compute)."""

import ctypes
import re

from conftest import ROOT


def declared_entry_points():
    names = []
    for header in sorted((ROOT / "include").glob("*.h")):
        text = re.sub(r"/\*.*?\*/", "", header.read_text(), flags=re.S)
        names += re.findall(r"^\s*(?:const\s+char\s*\*|int64_t|int)\s+(keepvq_\w+)\s*\(", text, flags=re.M)
    return names


def test_header_declares_entry_points():
    names = declared_entry_points()
    assert "keepvq_routed_matvec" in names and "keepvq_decode_weights" in names


def test_library_exports_every_declared_symbol():
    from keep_b200 import _lib

    lib = _lib.load()
    for name in declared_entry_points():
        assert hasattr(lib, name), f"libkeepvq.so lacks {name}"
    assert sorted(declared_entry_points()) == _lib.exported_names(), "ctypes table and header disagree"
    assert lib.keepvq_abi_version() == 3
    assert lib.keepvq_status_string(-2).decode() == "inconsistent sizes"


def test_no_source_of_randomness_that_may_throw():
    """The entry points are C: an exception that leaves one ends the process.  ``std::random_device`` throws
    where the host has no entropy to give (no /dev/urandom in a sandbox, no descriptor left)."""
    import subprocess

    from keep_b200 import _lib

    names = subprocess.run(["nm", "-D", "--undefined-only", str(_lib.LIBRARY_PATH)], capture_output=True, text=True, check=True).stdout
    assert "random_device" not in names


def test_struct_sizes_match_the_compiler():
    """ctypes mirrors of the argument structs have the layout gcc gives the header."""
    import subprocess
    import tempfile

    from keep_b200 import _lib

    structs = {"keepvq_decode_args": _lib.DecodeArgs, "keepvq_matvec_args": _lib.MatvecArgs}
    structs.update(getattr(_lib, "EXTRA_STRUCTS", {}))
    body = "".join(f'printf("{n} %zu\\n", sizeof({n}));' for n in structs)
    src = f'#include <stdio.h>\n#include "keepvq.h"\nint main(void){{{body}return 0;}}'
    with tempfile.TemporaryDirectory() as tmp:
        (c := __import__("pathlib").Path(tmp) / "s.c").write_text(src)
        exe = c.with_suffix("")
        subprocess.run(["gcc", "-I", str(ROOT / "include"), str(c), "-o", str(exe)], check=True)
        out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    for line in out.splitlines():
        name, size = line.split()
        assert ctypes.sizeof(structs[name]) == int(size), name


def test_packed_arguments_take_what_ctypes_takes():
    """The structs packed in one step equal those set field by field, also for a float beyond fp32's range
    (which becomes an infinity) and an integer beyond its field's."""
    from keep_b200 import _lib

    def flat(cls):
        for name, kind in cls._fields_:
            yield from flat(kind) if hasattr(kind, "_fields_") else [(name, kind)]

    def by_field(args, values):
        for name, kind in args._fields_:
            if hasattr(kind, "_fields_"):
                by_field(getattr(args, name), values)
            else:
                setattr(args, name, next(values))
        return args

    for cls, pack in ((_lib.MoELayerArgs, _lib.pack_layer_args), (_lib.GroupedProjectionArgs, _lib.pack_grouped_args), (_lib.MatvecArgs, _lib.pack_matvec_args)):
        fields = list(flat(cls))
        plain = [1.5 if kind is ctypes.c_float else 7 for _, kind in fields]
        for i in range(-1, len(fields)):
            values = list(plain)
            if i >= 0:
                values[i] = {ctypes.c_float: -1e40, ctypes.c_int32: 2 ** 32 + 3, ctypes.c_int64: 2 ** 64 + 3}.get(fields[i][1], 2 ** 63)
            want = by_field(cls(), iter(values))
            got = pack(*values)
            assert bytes(got) == bytes(want), (cls, i)


def test_padding_of_the_grouped_arguments_means_nothing():
    """A C caller that fills in the fields and leaves the struct's padding as it finds it is served like
    one that clears it.  (Calls that the library refuses for a misaligned row, before any CUDA call.)"""
    from keep_b200 import _lib

    lib, args = _lib.load(), _lib.GroupedProjectionArgs
    pointers = "x rhs codes scales codebook out workspace res_codes res_scales res_table hot_of_slot".split()
    numbers = "x_dtype routes scales_dtype slots out_dim in_dim groups codebook_all_odd out_dtype workspace_bytes x_div res_rows res_groups".split()
    for filler in (0x00, 0x08, 0xFF):
        a = args.from_buffer(bytearray([filler]) * ctypes.sizeof(args))
        for name in pointers + numbers:  # the fields of this version of the header
            setattr(a, name, None if name in pointers else 0)
        for name in ("x", "rhs", "codes", "scales", "codebook", "out", "workspace"):
            setattr(a, name, 256)
        a.x = 264  # fp16 rows that start between two 16-byte boundaries
        a.x_dtype = a.scales_dtype = a.out_dtype = _lib.dtype_tag(__import__("torch").float16)
        a.routes = a.slots = a.out_dim = a.groups = a.codebook_all_odd = a.x_div = 1
        a.in_dim, a.workspace_bytes = 256, 1 << 20
        assert lib.keepvq_grouped_projection(a, None) == -4, filler  # KEEPVQ_ERR_ALIGN


def test_operators_refuse_cpu_tensors():
    import pytest
    import torch

    from keep_b200 import _lib, kernels

    x = torch.zeros(64)
    with pytest.raises(_lib.KeepVQError):
        kernels.vq_qmv(x, torch.zeros(8, 8, dtype=torch.uint16), torch.ones(8, 1), None, in_dim=64, out_dim=8,
                       group_size=64, code_bits=16)


def test_custom_ops_register_without_a_gpu():
    """Importing ``keep_b200.torch_ops`` defines every operator under ``torch.ops.keepvq`` with a
    schema (no compute happens without a device)."""
    import torch

    from keep_b200 import torch_ops

    for name in torch_ops.OPS:
        schema = getattr(torch.ops.keepvq, name).default._schema
        assert schema.name == f"keepvq::{name}" and len(schema.returns) >= 1
