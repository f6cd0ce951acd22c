"""The entries of a decode or prefill step through ctypes, with the arguments of the extension (csrc/py_entries.cpp): what serves
where the extension was not built (no Python headers, or a library named by Q4K_B200_LIBRARY that has none beside it).  The same
calls of the C ABI with the same structures, 1 to 3 us slower each."""
from __future__ import annotations

import ctypes as C

import torch


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def _len(t) -> int:
    return 0 if t is None else t.numel()


def _stream(stream) -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()) if stream is None else stream.cuda_stream


class CtypesEntries:
    def __init__(self, lib, desc_type):
        self._lib, self._desc = lib, desc_type

    def _one(self, entry, desc, workspace, failure, stream) -> int:
        return entry(C.byref(desc.c_struct()), _ptr(workspace), workspace.numel(), _ptr(failure), _stream(stream))

    def decode_mmv(self, desc, workspace, failure, stream) -> int:
        return self._one(self._lib.q4k_decode_mmv, desc, workspace, failure, stream)

    def prefill_project(self, desc, workspace, failure, stream) -> int:
        return self._one(self._lib.q4k_prefill_project, desc, workspace, failure, stream)

    def decode_mmv_paired(self, a, b, workspace, failure, stream) -> int:
        return self._lib.q4k_decode_mmv_paired(C.byref(a.c_struct()), C.byref(b.c_struct()), _ptr(workspace), workspace.numel(), _ptr(failure),
                                               _stream(stream))

    def decode_mmv_ranges(self, ranges, workspace, failure, stream) -> int:
        descs = [r.c_struct() for r in tuple(ranges)]
        return self._lib.q4k_decode_mmv_ranges((self._desc * len(descs))(*descs), len(descs), _ptr(workspace), workspace.numel(), _ptr(failure),
                                               _stream(stream))

    def prefill_paired_swiglu(self, gate, up, normalized, swiglu, m, workspace, failure, stream) -> int:
        return self._lib.q4k_prefill_paired_swiglu(C.byref(gate.c_struct()), C.byref(up.c_struct()), _ptr(normalized), _ptr(swiglu), m,
                                                   _ptr(workspace), workspace.numel(), _ptr(failure), _stream(stream))

    def pack_q8(self, rows, fp32, out, failure, stream) -> int:
        entry = self._lib.q4k_pack_q8_f32 if fp32 else self._lib.q4k_pack_q8_bf16
        return entry(_ptr(rows), rows.numel(), out.c_struct(), _ptr(failure), _stream(stream))

    def q8_project(self, weight, x, out, residual, stream) -> int:
        return self._lib.q4k_q8_project(C.byref(weight.c_struct()), x.c_struct(), _ptr(out), out.numel(), _ptr(residual), _len(residual),
                                        _stream(stream))

    def q8_mlp(self, gate, up, down, residual, gamma, eps, out, m, workspace, pending, stream):
        submitted = C.c_int(0)
        st = self._lib.q4k_q8_mlp(C.byref(gate.c_struct()), C.byref(up.c_struct()), C.byref(down.c_struct()), _ptr(residual), _ptr(gamma), eps,
                                  _ptr(out), m, _ptr(workspace), workspace.numel() * workspace.element_size(), _stream(stream),
                                  C.byref(submitted), _ptr(pending))
        return st, submitted.value
