// How many threads of this process can run at the same time: the cores it may run on, and what a control group's CPU
// quota leaves of them (threads beyond the quota only use it up early; the process then stands still until the next
// period).  Reads files only; `root` is put in front of their paths.
#pragma once
#include <sched.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <thread>

namespace mascot {

// The first line of a file, or nothing.
inline std::string first_line(const std::string& path) {
    char buf[256] = "";
    if (FILE* f = std::fopen(path.c_str(), "r")) {
        if (!std::fgets(buf, sizeof buf, f)) buf[0] = 0;
        std::fclose(f);
    }
    return buf;
}

// Cores' worth of time that the quotas of the process's control groups allow; 0: no limit is known.  A quota of any group
// on the way up from the process's own counts (version 2: cpu.max; version 1: cpu.cfs_quota_us and cpu.cfs_period_us).
// In a container the path of /proc/self/cgroup may be the host's: the walk then only finds the container's root.
inline double quota_cores(const std::string& root) {
    double least = 0;
    auto limit = [&](double quota, double period) {
        if (quota > 0 && period > 0 && (least == 0 || quota / period < least)) least = quota / period;
    };
    FILE* f = std::fopen((root + "/proc/self/cgroup").c_str(), "r");
    if (!f) return 0;
    char line[4096];
    while (std::fgets(line, sizeof line, f)) {
        line[std::strcspn(line, "\n")] = 0;
        const char* controllers = std::strchr(line, ':');
        const char* path = controllers ? std::strchr(controllers + 1, ':') : nullptr;
        if (!path) continue;
        const std::string names(controllers + 1, path), list = "," + names + ",";
        const bool v2 = names.empty();
        if (!v2 && list.find(",cpu,") == std::string::npos) continue;
        for (std::string group = path + 1;; group.resize(group.find_last_of('/'))) {
            if (!group.empty() && group.back() == '/') group.pop_back();
            if (v2) {
                double quota = 0, period = 0;
                if (std::sscanf(first_line(root + "/sys/fs/cgroup" + group + "/cpu.max").c_str(), "%lf %lf", &quota, &period) == 2) limit(quota, period);
            } else {
                const std::string dir = root + "/sys/fs/cgroup/cpu" + group;
                limit(std::atof(first_line(dir + "/cpu.cfs_quota_us").c_str()), std::atof(first_line(dir + "/cpu.cfs_period_us").c_str()));
            }
            if (group.find('/') == std::string::npos) break;
        }
    }
    std::fclose(f);
    return least;
}

inline int usable_cores(const std::string& root = "") {
    cpu_set_t set;
    CPU_ZERO(&set);
    int n = sched_getaffinity(0, sizeof set, &set) == 0 ? CPU_COUNT(&set) : (int)std::thread::hardware_concurrency();
    const double quota = quota_cores(root);
    if (quota > 0) n = std::min(n, (int)quota);
    return std::max(1, n);
}

}  // namespace mascot
