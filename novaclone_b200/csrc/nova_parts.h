// Sources whose kernels no one run needs together are compiled in parts
// (build.py: -DNOVA_PART=p), each an object and so a module of its own: the first
// launch from a module unpacks and loads all of it.  Parts 0 .. n - 1 hold kernels,
// part n the dispatch.  First pass of a process, one module per source -> in
// parts: 20 steps at 64^3 37 -> 10 ms, 120 x 75 x 100 37 -> 9.8, 256^3 41 -> 14, MHD at
// 128^3 57 -> 13, FP32-split jet 192 x 192 x 384 57 -> 18, shear layer 39 -> 12.
#pragma once

#ifndef NOVA_PART
#error "compiled in parts: -DNOVA_PART=p (build.py)"
#endif
