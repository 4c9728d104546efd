"""The error sinogram, and the subset's records, are written by the kernel that
a VCD gradient is launched behind (programmatic dependent launch: the gradient's CTAs may be resident
while it is).  The read-only path is for memory that no one writes while the
kernel lives, so no reader of e may use it, in any storage type or width."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    'mbirtorch_b200', 'csrc')


def _source(name):
    return re.sub(r'//[^\n]*', '', open(os.path.join(CSRC, name)).read())


def _body(src, start):
    """The brace-delimited block that opens at or after `start`."""
    a = src.index('{', start)
    depth = 0
    for i in range(a, len(src)):
        depth += {'{': 1, '}': -1}.get(src[i], 0)
        if depth == 0:
            return src[a:i + 1]
    raise AssertionError('unbalanced braces')


def test_error_sinogram_readers_use_no_read_only_loads():
    proj, common = _source('projectors.cuh'), _source('mbir_common.cuh')
    found = 0
    for reader in ('ReadScaled', 'ReadWeighted'):
        body = _body(proj, proj.index(f'struct {reader} {{'))
        for m in re.finditer(r'void (get\w+)\(|float (get)\(', body):
            get = _body(body, m.end())
            assert '__ldg' not in get, (reader, get)
            for helper in set(re.findall(r'(\w+)\(\s*[ew]\s*\+', get)):
                defs = [d.end() for d in re.finditer(rf'void {helper}\(', common)]
                assert defs, helper
                for d in defs:
                    code = _body(common, d)
                    assert '__ldg' not in code and '.nc' not in code, (reader, helper)
                    found += 1
    assert found >= 4   # both readers' four-value loads were looked at


def test_gradient_reads_its_records_by_coherent_loads():
    """The tail of one step forms the next subset's records, which the gradient
    behind it reads: through load_rec, whose loads are coherent, and not as an
    element of the (restrict) parameter, which the compiler may load through
    the read-only path."""
    proj, back4, common = (_source(f) for f in ('projectors.cuh', 'back_cone4.cuh',
                                                'mbir_common.cuh'))
    for src, kernel in ((proj, 'back_cone_kernel_body('), (back4, 'back_cone4_kernel_body(')):
        body = _body(src, src.index(kernel))
        assert 'load_rec(recs' in body and not re.search(r'(?<!load_rec\()\brecs\[', body)
    assert 'ldg_f32x4' in _body(proj, proj.index('ConeFwdRec load_rec('))
    asm = _body(common, common.index('float4 ldg_f32x4('))
    assert 'volatile' in asm and 'ld.global.v4' in asm and '.nc' not in asm
