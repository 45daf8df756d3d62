"""CPU: the C-ABI library builds for sm_100a, loads, and exports every declared symbol."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def built_lib():
    from flashqla_b200 import build
    return build.build()


def test_library_builds_and_loads(built_lib):
    from flashqla_b200 import _cabi
    lib = _cabi.lib()
    assert lib.qla_abi_version() == 2
    assert lib.qla_status_string(0) == b"ok"
    assert lib.qla_status_string(-1) == b"invalid argument"


def test_every_declared_symbol_is_exported(built_lib):
    from flashqla_b200 import _cabi
    header = (ROOT / "include" / "flashqla_b200.h").read_text()
    declared = set(re.findall(r"QLA_API\s+[\w\s\*]+?\b(qla_\w+)\s*\(", header))
    assert declared, "no declarations found"
    assert declared == set(_cabi.EXPORTS), (declared, set(_cabi.EXPORTS))
    handle = ctypes.CDLL(str(built_lib))
    for name in declared:
        assert hasattr(handle, name), name


def test_struct_layouts_match_header(built_lib):
    """Field order of the ctypes mirrors follows the header (names in order)."""
    from flashqla_b200 import _cabi
    header = (ROOT / "include" / "flashqla_b200.h").read_text()
    for cls in (_cabi.QlaRecurrentArgs, _cabi.QlaChunkFwdArgs):
        body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (cls.__name__, cls.__name__), header, re.S).group(1)
        body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
        names = re.findall(r"(\w+)\s*;", body)
        assert names == [f[0] for f in cls._fields_], cls.__name__


def test_every_launch_can_report(built_lib):
    """Each argument structure whose kernel waits or checks indices has a status word; the chain's is read only from callers that say
    that they have it, because its structure ended in front of it before."""
    from flashqla_b200 import _cabi
    for cls in (_cabi.QlaRecurrentArgs, _cabi.QlaChunkFwdArgs, _cabi.QlaChunkBwdArgs, _cabi.QlaStateCommitArgs, _cabi.QlaCpChainArgs):
        assert "status" in {f[0] for f in cls._fields_}, cls.__name__
    assert [f[0] for f in _cabi.QlaCpChainArgs._fields_][-2:] == ["has_status", "status"]


def test_argument_validation_without_gpu(built_lib):
    """Host-side checks of the entry point run before any launch, so they work without a GPU."""
    from flashqla_b200 import _cabi
    lib = _cabi.lib()
    assert lib.qla_recurrent_update(None, None) == -1
    a = _cabi.QlaRecurrentArgs(num_seqs=1, total_tokens=1, tokens_per_seq=1, num_k_heads=3, num_v_heads=4)
    assert lib.qla_recurrent_update(a, None) == -1
    assert b"divisible" in lib.qla_last_error()


def test_python_api_rejects_bad_inputs():
    import flashqla_b200 as fq
    q = torch.zeros(2, 4, 1, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="flattened"):
        fq.fused_sigmoid_gating_delta_rule_update(None, None, None, q, q, q, None, None)
    q = torch.zeros(1, 4, 1, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="CUDA"):
        fq.fused_sigmoid_gating_delta_rule_update(None, None, None, q, q, q, None, None)


def test_manifest_describes_the_header(built_lib):
    """The JSON manifest written beside the library lists every exported function and every argument
    structure with the header's field order, and its offsets are those of the ctypes mirrors."""
    import json
    from flashqla_b200 import _cabi, manifest
    path = built_lib.parent / manifest.MANIFEST_NAME
    assert path.exists(), "the build writes the manifest"
    m = json.loads(path.read_text())
    header = (ROOT / "include" / "flashqla_b200.h").read_text()
    assert m["abi_version"] == int(re.search(r"#define QLA_ABI_VERSION (\d+)", header).group(1))
    assert set(m["exports"]) == set(_cabi.EXPORTS)
    for name, desc in m["structs"].items():
        body = re.search(r"typedef struct %s \{(.*?)\} %s;" % (name, name), header, re.S).group(1)
        body = re.sub(r"/\*.*?\*/", "", body, flags=re.S)
        assert [f["name"] for f in desc["fields"]] == re.findall(r"(\w+)\s*;", body), name
        cls = getattr(_cabi, name)
        assert desc["size"] == ctypes.sizeof(cls)
        assert all(f["offset"] == getattr(cls, f["name"]).offset for f in desc["fields"])
    for flag, value in m["flags"].items():
        c_name = "QLA_" + flag
        assert re.search(r"%s\s*=\s*%d\b|#define %s\s+%d\b" % (c_name, value, c_name, value), header), c_name


def test_manifest_lists_every_kernel_with_its_cubin(built_lib):
    """The build leaves one cubin per translation unit with kernels; the manifest's kernel entries point at
    them and carry launch constants that agree with the library's own (qla_kernel_launch_info)."""
    import json
    from flashqla_b200 import _cabi, manifest
    m = json.loads((built_lib.parent / manifest.MANIFEST_NAME).read_text())
    kernels = m["kernels"]
    assert kernels, "the build records its kernels"
    names = {k["kernel_name"] for k in kernels}
    assert set(manifest.KERNEL_RULES) <= names
    lib = _cabi.lib()
    for k in kernels:
        assert (built_lib.parent / k["cubin"]).exists(), k["cubin"]
        assert k["registers"] and k["export_name"].startswith("_Z")
        if k["kernel_name"] in manifest.KERNEL_RULES:
            block, smem = ctypes.c_int32(), ctypes.c_size_t()
            assert lib.qla_kernel_launch_info(k["kernel_name"].encode(), ctypes.byref(block), ctypes.byref(smem)) == 0
            assert block.value == 32 * k["num_warps"] and smem.value == k["shared"], k["kernel_name"]
    assert lib.qla_kernel_launch_info(b"no_such_kernel", ctypes.byref(block), ctypes.byref(smem)) == -1


def test_manifest_has_a_rule_for_every_kernel_that_asks_for_shared_memory(built_lib):
    """A launcher that loads a cubin cannot read a kernel's dynamic shared memory from the compiler's report: every kernel whose limit
    the library raises (the recurrent ones by a template parameter) has its bytes in the manifest."""
    import json
    from flashqla_b200 import build, manifest
    names = {n for src in build.sources() for n in re.findall(r"ensure_dynamic_smem<(\w+)", src.read_text())}
    assert {"chunk_fwd_kernel", "cp_chain_kernel"} <= names
    names = {n for n in names if n.endswith("_kernel")} | {"recurrent_kernel", "recurrent_chain_kernel", "recurrent_step_kernel"}
    m = json.loads((built_lib.parent / manifest.MANIFEST_NAME).read_text())
    for name in names:
        entries = [k for k in m["kernels"] if re.search(r"\d%s(I|E)" % name, k["export_name"])]
        assert entries and all(k["shared"] and k["shared"] + k["static_shared"] <= 227 * 1024 for k in entries), name


def test_manifest_gives_every_form_of_the_scan_its_shared_memory(built_lib):
    """chunk_fwd_kernel<T, kStateOnly, kAux, kTrace, kNorm, kState16, kWIn>: the forms with kAux and kWIn use more than the plain one."""
    import json
    from flashqla_b200 import _cabi, manifest
    m = json.loads((built_lib.parent / manifest.MANIFEST_NAME).read_text())
    lib, seen, shared = _cabi.lib(), set(), {}
    for k in m["kernels"]:
        form = re.search(r"chunk_fwd_kernelI\w+?Lb[01]ELb([01])ELb[01]ELb[01]ELb[01]ELb([01])E", k["export_name"])
        if form is None:
            continue
        name = "chunk_fwd_kernel" + {("0", "0"): "", ("1", "0"): ":aux", ("0", "1"): ":w_in_scan"}[form.groups()]
        block, smem = ctypes.c_int32(), ctypes.c_size_t()
        assert lib.qla_kernel_launch_info(name.encode(), ctypes.byref(block), ctypes.byref(smem)) == 0
        assert k["kernel_name"] == name and k["shared"] == smem.value and len(k["param_names"]) == 9
        assert k["shared"] + k["static_shared"] <= 227 * 1024
        seen.add(name)
        shared[name] = smem.value
    assert len(seen) == 3 and shared["chunk_fwd_kernel"] < min(shared["chunk_fwd_kernel:aux"], shared["chunk_fwd_kernel:w_in_scan"])


def test_another_torch_means_another_build(built_lib, tmp_path, monkeypatch):
    """The host module is compiled against torch and Python: a build for others is neither current nor accepted."""
    from types import SimpleNamespace
    from flashqla_b200 import _cabi, build
    assert build.is_current()
    (tmp_path / "version.py").write_text("__version__ = '0.0'\n")
    monkeypatch.setattr(build, "_torch_dir", lambda: tmp_path)
    assert not build.is_current()
    monkeypatch.undo()
    monkeypatch.setattr("sys.implementation.cache_tag", "cpython-00")
    assert not build.is_current()
    monkeypatch.undo()
    _cabi._check_built_for_this_torch(_cabi.host())
    with pytest.raises(_cabi.QlaError, match="rebuild"):
        _cabi._check_built_for_this_torch(SimpleNamespace(torch_version="0.0.0"))


@pytest.mark.parametrize("field,offset", [("q", 2), ("k", 4), ("state", 4), ("inter", 8)])
def test_pointers_the_recurrent_kernels_cannot_read_are_refused(built_lib, field, offset):
    """Tensors move in pieces of 8 or 16 bytes: a pointer between two pieces is an error before any launch."""
    from flashqla_b200 import _cabi
    ptrs = dict(q=4096, k=4096, v=4096, a=4096, b=4096, o=4096, state=4096, inter=4096, status=4096)
    ptrs[field] += offset
    a = _cabi.QlaRecurrentArgs(num_seqs=1, total_tokens=1, tokens_per_seq=1, num_k_heads=2, num_v_heads=2, qkv_dtype=1,
                               flags=_cabi.REC_A_IS_LOG_DECAY | _cabi.REC_B_IS_BETA, state_slots=1, inter_slots=1, inter_steps=1, **ptrs)
    assert _cabi.lib().qla_recurrent_update(a, None) == -1
    assert b"start on" in _cabi.lib().qla_last_error()
    if field in ("state", "inter"):
        c = _cabi.QlaStateCommitArgs(num_seqs=1, num_v_heads=1, inter_steps=1, inter_slots=1, state_slots=1, accepted=4096,
                                     inter=ptrs["inter"], state=ptrs["state"])
        assert _cabi.lib().qla_state_commit(c, None) == -1
        assert b"start on" in _cabi.lib().qla_last_error()
