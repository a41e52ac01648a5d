"""Several host threads on one device, each with its own system and stream:
the launches of one must not change what another's may take. The rules' and
meshes' kernels take different amounts of dynamic shared memory (stresses 70
KB and 57 KB a block, tiles 27 KB to 217 KB), all beyond the 48 KB that need
no leave."""
from __future__ import annotations

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["stress", "evaluate", "standard"])
@pytest.mark.parametrize("name", ["j2_steel", "hill_chaboche_sheet"])
def test_threads_with_different_rules(pkg, cuda, call, name):
    mat = getattr(pkg.material, name)()
    jobs = []
    for nx, rule in ((4, (2, 0)), (40, (3, 0)), (400, (2, 0)), (90, (2, 5))):
        mesh = pkg.structured_hex_mesh(nx, 12, 1, nx * 1.0e-3, 12.0e-3, 1.0e-3)
        s = pkg.NonlinearSystem(mesh, mat, "logarithmic", rule[0], rule[1], 2,
                                element="standard" if call == "standard" else "incompatible_modes")
        gen = torch.Generator(device=cuda).manual_seed(nx)
        u = 1.0e-6 * torch.randn(mesh.num_dofs, generator=gen, device=cuda, dtype=torch.float64)
        jobs.append((s, u, torch.cuda.Stream()))

    def once(s, u):
        if call == "stress":
            return s.stress(u).cauchy
        ev = s.evaluate(u, 0.0, True)
        return torch.cat([ev.internal, ev.tangent])

    torch.cuda.synchronize()
    errors, results = [], [None] * len(jobs)
    start = threading.Barrier(len(jobs))

    def work(k):
        s, u, stream = jobs[k]
        try:
            s.set_stream(stream)
            with torch.cuda.stream(stream):
                start.wait()
                for _ in range(1000 if call == "stress" else 60):
                    got = once(s, u)
                results[k] = got.clone()
                stream.synchronize()
        except Exception as e:  # a worker's failure is the test's
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k, (s, u, _) in enumerate(jobs):
        s.set_stream(None)
        assert torch.equal(results[k], once(s, u))
