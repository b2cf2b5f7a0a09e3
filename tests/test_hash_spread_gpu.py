"""Keys whose bits are anything but random: power-of-two strides in every column, planes, lines, bits of floats.  All are
found and nothing else is, in the full table of the smallest capacity."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _lattice(side, strides, dim):
    r = torch.arange(side, device=DEV) - side // 2
    axes = torch.meshgrid(*[r * s for s in strides], indexing="ij")
    return torch.stack(axes, -1).reshape(-1, len(strides))[:, :dim].to(torch.int32)


def _keys(kind, dim):
    if kind == "floats":
        g = torch.Generator(device=DEV).manual_seed(dim)
        return torch.unique(torch.randint(-60, 60, (400_000, dim), generator=g, device=DEV).float().view(torch.int32), dim=0)
    if kind == "plane":
        return _lattice(700, (1, 1), 2)[:, [0, 1] + [0] * (dim - 2)].contiguous() if dim > 2 else _lattice(700, (1, 1), 2)
    shift = int(kind)
    side = min(80 if dim > 2 else 700, 2 ** (31 - shift))
    return torch.unique(_lattice(side, (2**shift,) * min(dim, 3), dim), dim=0)


@pytest.mark.parametrize("kind", ["0", "10", "17", "22", "plane", "floats"])
@pytest.mark.parametrize("dim", [2, 3])
def test_structured_keys(kind, dim):
    import ash

    keys = _keys(kind, dim)
    n = len(keys)
    index = torch.arange(n, device=DEV).float().view(-1, 1)
    m = ash.HashMap(dim, {"i": 1}, n, DEV)
    order = torch.randperm(n, device=DEV)
    m.insert(keys[order].contiguous(), {"i": index[order].contiguous()})
    masks, values = m.find(keys, return_indices=False, return_values=True)
    assert m.size() == n and masks.all() and torch.equal(values["i"], index)
    other = keys.clone()
    other[:, 0] += 1 if kind in ("10", "17", "22", "floats") else 100_000
    assert not m.find(other)[0].any()
    assert m.engine.backend.status() == 0
