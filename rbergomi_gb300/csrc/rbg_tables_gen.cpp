// rbg_tables_gen.cpp -- run by the build on the host: prints the fixed-point
// tables (FixedTables, rbg_fixed.cuh) as the initialiser of the library's device
// copy, which is loaded with the module.  A copy filled at run time would make
// some call wait for the device, or fail while another thread captures a graph.
#include <cinttypes>
#include <cstdio>

#include "rbg_fixed.cuh"

int main()
{
    static rbg::FixedTables F;
    rbg::fill_fixed_tables(F);
    // one plain list in member order (the braces of the nested arrays may be left out)
    auto u64 = [](uint64_t v) { std::printf("0x%016" PRIx64 "ull,\n", v); };
    for (const rbg::FixedPair& p : F.normals.ln) { u64(p.x); u64(p.y); }
    for (const rbg::FixedPair& p : F.normals.trig) { u64(p.x); u64(p.y); }
    for (uint64_t v : F.normals.ln2) u64(v);
    for (uint64_t v : F.exp2) u64(v);
    for (const rbg::MillsRow& r : F.mills.r) {
        u64(r.b0); u64(r.b1); u64(r.b2); u64(r.b3); u64(r.b4);
        std::printf("0x%08" PRIx32 "u,\n0x%08" PRIx32 "u,\n", r.b5, r.b6);
    }
    return 0;
}
