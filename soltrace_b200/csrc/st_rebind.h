// A context's workspace on the device of its next run, free of CUDA so that it can be checked without
// a second device.
#pragma once
#include <new>

namespace stb {

// Selects `device` (select: 0 on success) and gives the workspace to it: a workspace serves one device
// and starts afresh on another.  Its destructor selects the old device to free what lies there, so
// the new one is selected again before anything is made for it.
template <typename Workspace, typename Select>
auto rebind(Workspace &ws, int device, Select select) {
    auto e = select(device);
    if (e || ws.device == device) return e;
    ws.~Workspace();
    new (&ws) Workspace();
    ws.device = device;
    return select(device);
}

}  // namespace stb
